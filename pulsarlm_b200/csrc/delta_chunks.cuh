// Delta rules over prompt portions in chunks of 16 tokens, bfloat16 engine: what the two recurrent mixers
// (gated_delta.cu, delta_rule.cu) share.
//
// A token's update of a head's state S [dim, vdim] is S <- diag(g) S + k z^T with a row z that itself reads the old
// state. Over a chunk that starts from S0 the rows solve a unit lower triangular system whose right-hand side
// is linear in S0 (the WY form of Householder products: Bischof and Van Loan 1987; for delta rules Yang et al.
// 2024), so with matrices that do not know S0
//
//   Z = Zi + Wm S0        [16, vdim]      O = Oi + Qg S0 + M Z      S <- diag(gC) S0 + Kd^T Z (+ Kv^T V)
//
// A first kernel makes Zi, Wm, Qg, M, Kd, gC (Oi, Kv) of all chunks side by side, all in fp32, decays between two tokens
// as running products (never as quotients, nor as differences of long sums of logarithms). The kernels below walk the
// chunks: one chain step per 16 tokens instead of one per token. A CTA has a head's 16 value columns; warp w of
// dim / 16 has their 16 state rows from 16 w on, transposed, in the accumulators of m16n8k16 products: that layout is
// also the A operand's, so the state goes from one product into the next without leaving registers. Every product
// multiplies fp32 numbers as three bfloat16 terms each (six of the nine products of terms; the rest is below
// fp32's last bit). The warps' shares of S0's products meet in shared memory, one barrier a chunk; all else
// lies in the scratch in the order the lanes read it.
#pragma once

#include <climits>

#include "cluster_helpers.cuh"
#include "mma_helpers.cuh"

namespace {

constexpr int kDeltaChunk = 16;
constexpr int kDeltaWindow = 128;  // chunks of an entry in one pass of the two kernels, at most
// The chunks' scratch in a call is held to this by fewer chunks of an entry a pass (four at least): 2,048 tokens of 32 heads of 64 x 64
// in one pass are 100 MB (157 MB the general rule), four such entries 400 MB without a bound.
constexpr int64_t kDeltaScratchBytes = 256 << 20;
constexpr int kDeltaCols = 16;     // value columns of a CTA of the walk

// Where a chunk's matrices lie in its scratch, in floats. All of it in fragment order. A matrix that is an operand (wm, qg,
// kd, kv by 16 state rows, m) is three bfloat16 terms: 384 floats, per term the 16 bytes that a lane reads of two 16 x 8 tiles.
// Of the results' starts (zi, oi) and the packed values (vv) a lane reads 16 bytes per tile of 16 columns.
struct DeltaChunkLayout {
    int wm, qg, kd, kv, m, zi, oi, vv, g, floats;
    __host__ __device__ constexpr DeltaChunkLayout(int dim, int vdim, bool general)
    : wm(0), qg(24 * dim), kd(48 * dim), kv(72 * dim), m(general ? 96 * dim : 72 * dim), zi(m + 384), oi(zi + 16 * vdim),
      vv(oi + (general ? 16 * vdim : 0)), g(vv + (general ? 8 * vdim : 0)), floats(g + dim) {}
};

// While a chunk is put together in shared memory the operands are fp32: 256 floats per 16 state rows, and 256 for m. Every tile
// of 128 floats takes kStagedTile there, so that a column's places meet fewer banks twice (all starts are whole tiles).
constexpr int kStagedTile = 136;
struct DeltaStageLayout {
    int wm, qg, kd, kv, m, zi, oi, vv, g, floats;
    __host__ __device__ constexpr DeltaStageLayout(int dim, int vdim, bool general)
    : wm(0), qg(tiles(16 * dim)), kd(tiles(32 * dim)), kv(tiles(48 * dim)), m(general ? tiles(64 * dim) : kv), zi(m + tiles(256)),
      oi(zi + tiles(16 * vdim)), vv(oi + (general ? tiles(16 * vdim) : 0)), g(vv + (general ? tiles(8 * vdim) : 0)),
      floats(g + dim) {}
    __host__ __device__ static constexpr int tiles(int n) { return n / 128 * kStagedTile; }
};

// Places in shared memory, each a base of one index and a fixed distance for the other. Element (token t, channel d) of a
// [16, dim] operand whose k axis is the channel (Wm, Qg) ...
__device__ __forceinline__ int place_of_channel(int d) {
    return (d >> 4) * 2 * kStagedTile + (((d & 7) >> 1) << 2) + ((d >> 3 & 1) << 1) + (d & 1);
}
__host__ __device__ constexpr int at_token(int t) { return (t >> 3) * kStagedTile + (t & 7) * 16; }
// ... or the token (Kd, Kv); (for channel 4 l + 32 h + r with r < 4: place_of_quad(l) + at_quad(h, r) more)
__device__ __forceinline__ int place_of_source(int s) { return (((s & 7) >> 1) << 2) + ((s >> 3) << 1) + (s & 1); }
__device__ __forceinline__ int place_of_quad(int l) { return (l >> 1) * kStagedTile + (l & 1) * 64; }
__host__ __device__ constexpr int at_quad(int h, int r) { return h * 4 * kStagedTile + r * 16; }
// Element (t, s) of M: place_of_source(s) + at_token(t). Element (t, column c) of a result, and the packed values' 32 bits of
// tokens t, t + 1.
__device__ __forceinline__ int place_of_column(int c) { return (c >> 4) * 2 * kStagedTile + (c & 7) * 16 + ((c >> 3 & 1) << 1); }
__host__ __device__ constexpr int at_result(int t) { return (t >> 3) * kStagedTile + ((t & 7) >> 1) * 4 + (t & 1); }
__device__ __forceinline__ int place_of_value(int c) { return (c >> 4) * kStagedTile + (c & 7) * 16 + (c >> 3 & 1); }
__host__ __device__ constexpr int at_value(int t) { return ((t & 7) >> 1) * 4 + 2 * (t >> 3); }
// A channel of gC: 16 floats per 16 state rows, four per lane & 3.
__device__ __forceinline__ int place_of_decay(int d) {
    return (d >> 4) * 16 + ((d & 7) >> 1) * 4 + (d >> 3 & 1) * 2 + (d & 1);
}

// Two fp32 numbers as three pairs of bfloat16.
__device__ __forceinline__ void three_pairs(float x, float y, uint32_t& hi, uint32_t& mid, uint32_t& lo) {
    hi = pack_bf16(x, y);
    const float rx = x - __uint_as_float(hi << 16), ry = y - __uint_as_float(hi & 0xffff0000u);
    mid = pack_bf16(rx, ry);
    lo = pack_bf16(rx - __uint_as_float(mid << 16), ry - __uint_as_float(mid & 0xffff0000u));
}

// What was put together leaves for the scratch: the operands (all that comes before zi) as three terms, the others as
// they are.
__device__ __forceinline__ void send_chunk(const float* out, float* scratch, const DeltaStageLayout& at, int dim) {
    const float4* src = reinterpret_cast<const float4*>(out);
    uint4* dst = reinterpret_cast<uint4*>(scratch);
    const int groups = at.zi / (2 * kStagedTile);    // (16 state rows of an operand, or m: two tiles)
    for (int idx = threadIdx.x; idx < groups * 32; idx += blockDim.x) {
        const int group = idx >> 5, lane = idx & 31;
        const float4 a = src[group * (kStagedTile / 2) + lane], b = src[group * (kStagedTile / 2) + kStagedTile / 4 + lane];
        uint4 hi, mid, lo;
        three_pairs(a.x, a.y, hi.x, mid.x, lo.x);
        three_pairs(a.z, a.w, hi.y, mid.y, lo.y);
        three_pairs(b.x, b.y, hi.z, mid.z, lo.z);
        three_pairs(b.z, b.w, hi.w, mid.w, lo.w);
        uint4* to = dst + group * 96 + lane;
        to[0] = hi;
        to[32] = mid;
        to[64] = lo;
    }
    float4* tail = reinterpret_cast<float4*>(scratch) + groups * 96;
    const int tiles = (at.g - at.zi) / kStagedTile;
    for (int idx = threadIdx.x; idx < tiles * 32 + dim / 4; idx += blockDim.x) {
        tail[idx] = src[at.zi / 4 + idx + min(idx >> 5, tiles) * ((kStagedTile - 128) / 4)];
    }
}

// values[i], i < 16, of a whole warp's lanes, summed: the lanes 2 i and 2 i + 1 get sum i.
__device__ __forceinline__ float sum_over_warp(float (&values)[16]) {
    const int lane = threadIdx.x & 31;
    float v[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const bool upper = lane & 16;
        const float give = upper ? values[i] : values[i + 8], keep = upper ? values[i + 8] : values[i];
        v[i] = keep + __shfl_xor_sync(0xffffffffu, give, 16);
    }
#pragma unroll
    for (int n = 4; n >= 1; n >>= 1) {
        const bool upper = lane & (2 * n);
#pragma unroll
        for (int i = 0; i < n; ++i) {
            const float give = upper ? v[i] : v[i + n], keep = upper ? v[i + n] : v[i];
            v[i] = keep + __shfl_xor_sync(0xffffffffu, give, 2 * n);
        }
    }
    return v[0] + __shfl_xor_sync(0xffffffffu, v[0], 1);
}

// values[i], i < 16, of the eight lanes that share lane >> 3, summed: lane l of them gets sums 2 (l & 7) and the next.
__device__ __forceinline__ void sum_over_eight(float (&values)[16], float& even, float& odd) {
    const int l = threadIdx.x & 7;
    float a[8], b[4];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const bool upper = l & 4;
        const float give = upper ? values[i] : values[i + 8], keep = upper ? values[i + 8] : values[i];
        a[i] = keep + __shfl_xor_sync(0xffffffffu, give, 4);
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const bool upper = l & 2;
        const float give = upper ? a[i] : a[i + 4], keep = upper ? a[i + 4] : a[i];
        b[i] = keep + __shfl_xor_sync(0xffffffffu, give, 2);
    }
    const bool upper = l & 1;
    const float give0 = upper ? b[0] : b[2], give1 = upper ? b[1] : b[3];
    even = (upper ? b[2] : b[0]) + __shfl_xor_sync(0xffffffffu, give0, 1);
    odd = (upper ? b[3] : b[1]) + __shfl_xor_sync(0xffffffffu, give1, 1);
}

// One pass over the entries that go in chunks: those of `least` rows and more, `window` chunks of each.
struct DeltaPass {
    int n_entries, least, window, pass;
};

// Chunks of an entry of `count` rows in this pass.
__device__ __forceinline__ int delta_chunks_of(int count, const DeltaPass& p) {
    return count < p.least ? 0 : max(0, min((count + kDeltaChunk - 1) / kDeltaChunk - p.pass * p.window, p.window));
}

// The entry and its chunk that scratch slot `slot` of this pass belongs to; false past the last. (By a whole warp.)
__device__ __forceinline__ bool delta_find_chunk(const int32_t* counts, const DeltaPass& p, int slot, int& entry, int& chunk) {
    const int lane = threadIdx.x & 31;
    int before = 0;
    for (int base = 0; base < p.n_entries; base += 32) {
        const int mine = base + lane < p.n_entries ? delta_chunks_of(counts[base + lane], p) : 0;
        int upto = mine;
#pragma unroll
        for (int offset = 1; offset < 32; offset <<= 1) {
            const int other = __shfl_up_sync(0xffffffffu, upto, offset);
            upto += lane >= offset ? other : 0;
        }
        const uint32_t past = __ballot_sync(0xffffffffu, before + upto > slot);
        if (past != 0) {
            const int who = __ffs(past) - 1;
            entry = base + who;
            chunk = slot - before - __shfl_sync(0xffffffffu, upto - mine, who);
            return true;
        }
        before += __shfl_sync(0xffffffffu, upto, 31);
    }
    return false;
}

// Up to 32 entries: the place in the entries' order of the `nth` longest of those that go in chunks. (By a whole warp.) Chains
// of several lengths then start with the longest.
__device__ __forceinline__ int delta_nth_longest(const int32_t* counts, const DeltaPass& p, int nth) {
    if (p.n_entries > 32) {
        return nth;
    }
    const int lane = threadIdx.x & 31;
    const int count = lane < p.n_entries ? counts[lane] : 0;
    const uint32_t longer = __ballot_sync(0xffffffffu, count >= p.least);
    int rank = 0;
    for (int other = 0; other < p.n_entries; ++other) {
        const int theirs = __shfl_sync(0xffffffffu, count, other);
        rank += theirs > count || (theirs == count && other < lane);
    }
    const uint32_t found = __ballot_sync(0xffffffffu, count >= p.least && rank == nth);
    return found == 0 ? nth : __popc(longer & ((1u << (__ffs(found) - 1)) - 1u));
}

// The `nth` entry that goes in chunks, and how many chunks of this pass come before its own; false past the last. (By a whole
// warp.)
__device__ __forceinline__ bool delta_find_entry(const int32_t* counts, const DeltaPass& p, int nth, int& entry, int& before) {
    const int lane = threadIdx.x & 31;
    before = 0;
    for (int base = 0; base < p.n_entries; base += 32) {
        const int count = base + lane < p.n_entries ? counts[base + lane] : 0;
        const uint32_t longer = __ballot_sync(0xffffffffu, count >= p.least);
        const int rank = __popc(longer & ((1u << lane) - 1u));
        const uint32_t found = __ballot_sync(0xffffffffu, count >= p.least && rank == nth);
        int sum = found == 0 || lane < __ffs(found) - 1 ? delta_chunks_of(count, p) : 0;
#pragma unroll
        for (int offset = 16; offset > 0; offset >>= 1) {
            sum += __shfl_xor_sync(0xffffffffu, sum, offset);
        }
        before += sum;
        if (found != 0) {
            entry = base + __ffs(found) - 1;
            return true;
        }
        nth -= __popc(longer);
    }
    return false;
}

struct DeltaChainParams {
    const float* scratch;
    float* state;
    const int32_t* first_rows;
    const int32_t* counts;
    const int32_t* slots;
    float* o_raw;
    int n_heads, vdim;
    DeltaPass pass;
    int32_t* status;  // (bit 8 where a chunk did not come; may be nullptr)
};

struct TermsA {
    uint32_t t[3][4];  // hi, mid, lo
};
struct TermsB {
    uint4 t[3];        // two tiles' registers of each term
};
__device__ __forceinline__ void terms_of(TermsA& a, const float (&lo8)[4], const float (&hi8)[4]) {
    three_pairs(lo8[0], lo8[1], a.t[0][0], a.t[1][0], a.t[2][0]);
    three_pairs(lo8[2], lo8[3], a.t[0][1], a.t[1][1], a.t[2][1]);
    three_pairs(hi8[0], hi8[1], a.t[0][2], a.t[1][2], a.t[2][2]);
    three_pairs(hi8[2], hi8[3], a.t[0][3], a.t[1][3], a.t[2][3]);
}
// d0, d1 = a b's two tiles: the largest terms' product in an accumulator of its own, the small products before their sum meets
// it. (An accumulator that already holds something rounds at its size with every product that joins.)
__device__ __forceinline__ void mma_terms(float (&d0)[4], float (&d1)[4], const TermsA& a, const TermsB& b) {
    constexpr int kA[5] = {2, 0, 1, 1, 0}, kB[5] = {0, 2, 1, 0, 1};
    float small0[4] = {}, small1[4] = {};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        d0[i] = d1[i] = 0.0f;
    }
    mma_bf16(d0, a.t[0], b.t[0].x, b.t[0].y);
    mma_bf16(d1, a.t[0], b.t[0].z, b.t[0].w);
#pragma unroll
    for (int i = 0; i < 5; ++i) {
        mma_bf16(small0, a.t[kA[i]], b.t[kB[i]].x, b.t[kB[i]].y);
        mma_bf16(small1, a.t[kA[i]], b.t[kB[i]].z, b.t[kB[i]].w);
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        d0[i] += small0[i];
        d1[i] += small1[i];
    }
}

// The sum of the warps' shares of Z and its start: every warp makes it whole.
template <int N, int NW>
__device__ __forceinline__ void sum_of_shares(float (&z)[2][4], const float4 (&zi)[2], const float4 (&shares)[N][NW][32], int lane) {
#pragma unroll
    for (int j = 0; j < 2; ++j) {
        float4 sum = shares[j][0][lane];
#pragma unroll
        for (int other = 1; other < NW; ++other) {
            const float4 part = shares[j][other][lane];
            sum = make_float4(sum.x + part.x, sum.y + part.y, sum.z + part.z, sum.w + part.w);
        }
        z[j][0] = zi[j].x + sum.x;
        z[j][1] = zi[j].y + sum.y;
        z[j][2] = zi[j].z + sum.z;
        z[j][3] = zi[j].w + sum.w;
    }
}

// Less than infinity while all of Z is.
__device__ __forceinline__ float size_of(const float (&z)[2][4]) {
    float size = 0.0f;
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        size += fabsf(z[0][r]) + fabsf(z[1][r]);
    }
    return size;
}

// A chunk's outputs o = Oi + M Z of warp w's eight tokens (S0's part joins later), from Z's terms. `size`: size_of(Z).
__device__ __forceinline__ void chunk_outputs(float (&o)[4], float size, TermsA& az, const TermsB& m, const float4& oi, int w,
                                              int lane) {
    float half[4] = {0.0f, 0.0f, 0.0f, 0.0f};
    o[0] = oi.x;
    o[1] = oi.y;
    o[2] = oi.z;
    o[3] = oi.w;
    // A row of Z that is not finite would reach the chunk's earlier tokens through the zeros above M's diagonal: it is
    // left out of the product, and the tokens from its own on are not a number. (What this needs of Z is in its terms.)
    if (!__all_sync(0xffffffffu, size < INFINITY)) {
        uint32_t bad[2] = {0u, 0u};  // bit t: token t's row, at this lane's column and the one 8 on
#pragma unroll
        for (int q = 0; q < 4; ++q) {
#pragma unroll
            for (int r = 0; r < 2; ++r) {
                const uint32_t exponent = 0x7f80u << (16 * r);
                if ((az.t[0][q] & exponent) == exponent) {
                    bad[q & 1] |= 1u << (8 * (q >> 1) + (lane & 3) * 2 + r);
#pragma unroll
                    for (int term = 0; term < 3; ++term) {
                        az.t[term][q] &= 0xffffu << (16 * (1 - r));
                    }
                }
            }
        }
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            bad[h] |= __shfl_xor_sync(0xffffffffu, bad[h], 1);
            bad[h] |= __shfl_xor_sync(0xffffffffu, bad[h], 2);
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {  // (tokens 8 w + (lane % 4) * 2 and the next: bits 0 to its own)
            if (bad[i >> 1] & ((2u << (w * 8 + (lane & 3) * 2 + (i & 1))) - 1u)) {
                o[i] = NAN;
            }
        }
    }
    constexpr int kA[6] = {2, 0, 1, 1, 0, 0}, kB[6] = {0, 2, 1, 0, 1, 0};
#pragma unroll
    for (int i = 0; i < 6; ++i) {
        const uint4 b = m.t[kB[i]];
        mma_bf16(i % 2 ? o : half, az.t[kA[i]], w == 0 ? b.x : b.z, w == 0 ? b.y : b.w);
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        o[i] += half[i];
    }
}

// What a lane of the joint form needs of a chunk, a chunk ahead of its use in registers.
template <bool GENERAL>
struct DeltaLane {
    TermsB wm, qg, kd, m, kv;
    float4 zi[2], g;
    uint4 vv;
};

// Outputs by the chain's warps. grid (entries that go in chunks, heads, vdim / 16), NW = dim / 16 warps. On the path from a chunk to the
// next are only Z's products, their sum over the warps, and the state's update; O's products fill the waits between and are added up a
// chunk later. Bound by
// that path where an SM has one CTA (0.85 us a chunk); many CTAs fill the waits of one another, and a step of their short chains begins
// with plain loads and no set-up. The walks took 681 us for one prompt of 2,048 tokens, 32 heads of 64 x 64. Slower: 32 columns a CTA.
template <int NW, bool GENERAL>
__global__ void __launch_bounds__(NW * 32) delta_chain_joint_kernel(const DeltaChainParams p) {
    pl_grid_trigger();
    pl_grid_wait();
    constexpr int kDim = NW * 16;
    __shared__ float4 shares[2][4][NW][32];  // by chunk parity: two tiles of Z, two of O
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    const int head = blockIdx.y, ct = blockIdx.z;
    int e, before;
    if (!delta_find_entry(p.counts, p.pass, blockIdx.x, e, before)) {
        return;
    }
    const int count = p.counts[e];
    const int n_chunks = delta_chunks_of(count, p.pass);
    if (n_chunks == 0) {
        return;
    }
    const DeltaChunkLayout at(kDim, p.vdim, GENERAL);
    constexpr DeltaChunkLayout kAt(kDim, 0, GENERAL);  // (the places up to zi hold for any vdim)
    const int64_t step = static_cast<int64_t>(p.n_heads) * at.floats;
    const float* chunk0 = p.scratch + (static_cast<int64_t>(before) * p.n_heads + head) * at.floats;
    const float* src = chunk0 + w * 384 + lane * 4;
    const float* src_m = chunk0 + kAt.m + lane * 4;
    const float* src_zi = chunk0 + kAt.zi + (ct * 2 * 32 + lane) * 4;
    const float* src_oi = chunk0 + at.oi + ((ct * 2 + w) * 32 + lane) * 4;
    const float* src_vv = chunk0 + at.vv + (ct * 32 + lane) * 4;
    const float* src_g = chunk0 + at.g + w * 16 + (lane & 3) * 4;
    auto terms = [](TermsB& b, const float* from) {
#pragma unroll
        for (int term = 0; term < 3; ++term) {
            b.t[term] = *reinterpret_cast<const uint4*>(from + term * 128);
        }
    };
    auto fetch_m = [&](TermsB& m) {
        terms(m, src_m);
        src_m += step;
    };
    auto fetch = [&](DeltaLane<GENERAL>& in) {
        terms(in.wm, src);
        terms(in.qg, src + kAt.qg);
        if constexpr (!GENERAL) {
            terms(in.kd, src + kAt.kd);
        }
        in.zi[0] = *reinterpret_cast<const float4*>(src_zi);
        in.zi[1] = *reinterpret_cast<const float4*>(src_zi + 128);
        in.g = *reinterpret_cast<const float4*>(src_g);
        if constexpr (GENERAL) {
            terms(in.kv, src + kAt.kv);
            in.vv = *reinterpret_cast<const uint4*>(src_vv);
            src_vv += step;
        } else if (w < 2) {
            fetch_m(in.m);
        }
        src += step;
        src_zi += step;
        src_g += step;
    };
    DeltaLane<GENERAL> even = {}, odd = {};
    fetch(even);

    // S transposed: s[j][r] is column ct * 16 + lane / 4 (+ 8 for r >= 2), row w * 16 + 8 j + (lane % 4) * 2 + r % 2.
    float s[2][4];
    float* corner = p.state + ((static_cast<int64_t>(p.slots[e]) * p.n_heads + head) * kDim + w * 16 + (lane & 3) * 2) * p.vdim +
        ct * kDeltaCols + (lane >> 2);
#pragma unroll
    for (int j = 0; j < 2; ++j) {
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            s[j][r] = corner[static_cast<int64_t>(8 * j + (r & 1)) * p.vdim + (r >> 1) * 8];
        }
    }
    // This lane's outputs: columns lane / 4 and 8 on, tokens 8 w + (lane % 4) * 2 and the next (of the first two warps).
    const int done = p.pass.pass * p.pass.window * kDeltaChunk;
    const int rows = count - done;
    const int64_t o_stride = static_cast<int64_t>(p.n_heads) * p.vdim;
    int token = w * 8 + (lane & 3) * 2;
    float* dst = p.o_raw + (p.first_rows[e] + done + token) * o_stride +
        static_cast<int64_t>(head) * p.vdim + ct * kDeltaCols + (lane >> 2);
    float o[4] = {0.0f, 0.0f, 0.0f, 0.0f};
    auto finish = [&](int parity) {
#pragma unroll
        for (int other = 0; other < NW; ++other) {
            const float4 part = shares[parity][2 + w][other][lane];
            o[0] += part.x;
            o[1] += part.y;
            o[2] += part.z;
            o[3] += part.w;
        }
        if (token < rows) {
            dst[0] = o[0];
            dst[8] = o[2];
        }
        if (token + 1 < rows) {
            dst[o_stride] = o[1];
            dst[o_stride + 8] = o[3];
        }
        token += kDeltaChunk;
        dst += kDeltaChunk * o_stride;
    };

    auto advance = [&](const DeltaLane<GENERAL>& in, DeltaLane<GENERAL>& ahead, int c, const int parity) {
        // (M, Oi and Kd, which the chunk's end reads: a chunk ahead too the general rule's registers would not hold them)
        TermsB m = in.m;
        TermsB kd_now = in.kd;
        float4 oi = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if constexpr (GENERAL) {
            terms(kd_now, src - step + kAt.kd);
            if (w < 2) {
                fetch_m(m);
                oi = *reinterpret_cast<const float4*>(src_oi);
                src_oi += step;
            }
        }
        if (c + 1 < n_chunks) {
            fetch(ahead);
        }
        TermsA a, az;
        terms_of(a, s[0], s[1]);
        float d[2][4];
        mma_terms(d[0], d[1], a, in.wm);  // this warp's rows' share of S0's part of Z
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            shares[parity][j][w][lane] = make_float4(d[j][0], d[j][1], d[j][2], d[j][3]);
        }
        const float decay[2][2] = {{in.g.x, in.g.y}, {in.g.z, in.g.w}};
        float written[2][4] = {};
        if constexpr (GENERAL) {  // + Kv^T V: the values are bfloat16 as they are
            const uint32_t v[4] = {in.vv.x, in.vv.y, in.vv.z, in.vv.w};
#pragma unroll
            for (int term = 2; term >= 0; --term) {
                mma_bf16(written[0], v, in.kv.t[term].x, in.kv.t[term].y);
                mma_bf16(written[1], v, in.kv.t[term].z, in.kv.t[term].w);
            }
        }
#pragma unroll
        for (int j = 0; j < 2; ++j) {
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                s[j][r] = fmaf(s[j][r], decay[j][r & 1], written[j][r]);
            }
        }
        __syncthreads();
        float z[2][4];
        sum_of_shares(z, in.zi, shares[parity], lane);
        const float size = size_of(z);
        float q[2][4];
        mma_terms(q[0], q[1], a, in.qg);  // (and of O: made while the sums of Z come in, read after the next barrier)
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            shares[parity][2 + j][w][lane] = make_float4(q[j][0], q[j][1], q[j][2], q[j][3]);
        }
        terms_of(az, z[0], z[1]);
        float moved[2][4];
        mma_terms(moved[0], moved[1], az, kd_now);
#pragma unroll
        for (int j = 0; j < 2; ++j) {
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                s[j][r] += moved[j][r];
            }
        }
        if (w < 2) {
            if (c > 0) {
                finish(parity ^ 1);  // the chunk before: its shares were written before this chunk's barrier
            }
            chunk_outputs(o, size, az, m, oi, w, lane);
        }
    };
    for (int c = 0; c < n_chunks; c += 2) {
        advance(even, odd, c, 0);
        if (c + 1 < n_chunks) {
            advance(odd, even, c + 1, 1);
        }
    }
    __syncthreads();
    if (w < 2) {
        finish((n_chunks - 1) & 1);
    }
#pragma unroll
    for (int j = 0; j < 2; ++j) {
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            corner[static_cast<int64_t>(8 * j + (r & 1)) * p.vdim + (r >> 1) * 8] = s[j][r];
        }
    }
}

// A CTA's chunk in shared memory, in floats: the operands and M as they lie in the scratch, and of the rest the CTA's columns.
template <int DIM, bool GENERAL>
struct DeltaRing {
    static constexpr DeltaChunkLayout kAt{DIM, 0, GENERAL};  // (the places up to zi hold for any vdim)
    static constexpr int kZi = kAt.zi, kOi = kZi + 256, kVv = kOi + (GENERAL ? 256 : 0), kG = kVv + (GENERAL ? 128 : 0);
    static constexpr int kFloats = kG + DIM;
    static constexpr int kSlots = DIM == 128 || GENERAL ? 3 : 4;  // (two CTAs of 64 rows an SM)
    static constexpr int kBytes = kSlots * kFloats * 4 + 2 * 2 * DIM / 16 * 32 * 16;
};

// Outputs by warps of their own. grid (entries that go in chunks x heads, vdim / 16), 2 NW warps, NW = dim / 16. On the path from a
// chunk to the next are only Z's products, their sum over the warps, and the state's update: the first NW warps do nothing else. They leave the state that
// a chunk starts from in shared memory, where the other NW take it up for O's products, a barrier behind, and add those up a
// chunk later. The chunks' matrices come into shared memory by bulk copies, three or four chunks in flight. Bound by the path's
// instructions, each of which waits for the one before it (0.74 us a chunk; 0.85 where NW warps made the outputs too, with what
// a lane needs of a chunk in registers, up to 250 a thread). In the part, beside the kernels around it, us, before and now: one
// prompt of 2,048 tokens, 32 heads of 64 x 64: 128 and 95 a decay per channel, 175 and 101 the general rule; 16 heads of 128 x
// 128 206 and 177 the general rule; twelve portions of 1,500 tokens in all 100 and 70. Slower: 32 columns a CTA (140); lines
// asked into L1 or L2 chunks ahead change nothing.
template <int NW, bool GENERAL>
__global__ void __launch_bounds__(NW * 64, NW >= 8 ? 1 : 8 / NW) delta_chain_kernel(const DeltaChainParams p) {
    pl_grid_trigger();
    pl_grid_wait();
    constexpr int kDim = NW * 16;
    __shared__ float4 shares[2][2][NW][32];     // by chunk parity: two tiles of Z,
    __shared__ float4 o_shares[2][2][NW][32];   // two of O,
    const int tid = threadIdx.x, lane = tid & 31, w = (tid >> 5) % NW;
    const bool outputs = tid >= NW * 32;
    const int head = blockIdx.x % p.n_heads, ct = blockIdx.y;
    int e, before;
    if (!delta_find_entry(p.counts, p.pass, delta_nth_longest(p.counts, p.pass, blockIdx.x / p.n_heads), e, before)) {
        return;
    }
    const int count = p.counts[e];
    const int n_chunks = delta_chunks_of(count, p.pass);
    if (n_chunks == 0) {
        return;
    }
    using Ring = DeltaRing<kDim, GENERAL>;
    const DeltaChunkLayout at(kDim, p.vdim, GENERAL);
    const int64_t step = static_cast<int64_t>(p.n_heads) * at.floats;
    const float* chunk0 = p.scratch + (static_cast<int64_t>(before) * p.n_heads + head) * at.floats;
    extern __shared__ __align__(128) float ring[];   // [slots][Ring::kFloats], and the state before the chunk, by its parity
    auto states = reinterpret_cast<float4(*)[2][NW][32]>(ring + Ring::kSlots * Ring::kFloats);
    __shared__ __align__(8) uint64_t landed[Ring::kSlots];
    __shared__ volatile int lost;
    // One thread of the outputs' warps brings a chunk in, kSlots of them in flight.
    const bool brings = tid == blockDim.x - 32;
    auto bring = [&](int c) {
        const float* from = chunk0 + c * step;
        float* to = ring + c % Ring::kSlots * Ring::kFloats;
        uint64_t* bar = &landed[c % Ring::kSlots];
        auto copy = [&](int dst, int src, int floats) {
            asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                             smem_u32(to + dst)),
                         "l"(from + src), "r"(floats * 4), "r"(smem_u32(bar))
                         : "memory");
        };
        mbar_expect_tx(bar, Ring::kFloats * 4);
        copy(0, 0, Ring::kZi);
        copy(Ring::kZi, at.zi + ct * 256, 256);
        if constexpr (GENERAL) {
            copy(Ring::kOi, at.oi + ct * 256, 256);
            copy(Ring::kVv, at.vv + ct * 128, 128);
        }
        copy(Ring::kG, at.g, kDim);
    };
    if (brings) {
        lost = 0;
        for (int i = 0; i < Ring::kSlots; ++i) {
            mbar_init(&landed[i], 1);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    if (brings) {
        for (int c = 0; c < min(Ring::kSlots, n_chunks); ++c) {
            bring(c);
        }
    }
    // A chunk's place once it is there. (Where one never comes the wait gives up: the state's end, this chunk's outputs and all later
    // ones are not a number, and the status word says so. Whoever gave up said it before the next meeting, and what was made
    // of the chunk is stored behind that.)
    int slot = 0;
    uint32_t phase = 0;
    const float* cur = ring;
    auto wait_for_chunk = [&] { mbar_wait(&landed[slot], phase, &lost); };
    auto next_chunk = [&] {
        cur += Ring::kFloats;
        if (++slot == Ring::kSlots) {
            slot = 0;
            phase ^= 1u;
            cur = ring;
        }
    };
    auto terms = [](TermsB& b, const float* from) {
#pragma unroll
        for (int term = 0; term < 3; ++term) {
            b.t[term] = *reinterpret_cast<const uint4*>(from + term * 128);
        }
    };
    const int own = w * 384 + lane * 4;
    // Both halves of the CTA meet once a chunk and once after the last, each from a branch of its own: __syncthreads() is only for
    // places that every thread comes by, a named barrier counts threads wherever they are.
    auto meet = [] { asm volatile("bar.sync 1, %0;" ::"n"(NW * 64) : "memory"); };

    if (!outputs) {
        // S transposed: s[j][r] is column ct * 16 + lane / 4 (+ 8 for r >= 2), row w * 16 + 8 j + (lane % 4) * 2 + r % 2.
        float s[2][4];
        float* corner = p.state + ((static_cast<int64_t>(p.slots[e]) * p.n_heads + head) * kDim + w * 16 + (lane & 3) * 2) * p.vdim +
            ct * kDeltaCols + (lane >> 2);
#pragma unroll
        for (int j = 0; j < 2; ++j) {
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                s[j][r] = corner[static_cast<int64_t>(8 * j + (r & 1)) * p.vdim + (r >> 1) * 8];
            }
        }
        TermsB wm, kd, kv = {};
        float4 zi[2], g;
        uint4 vv = {};
        auto read_chunk = [&] {
            wait_for_chunk();
            terms(wm, cur + own);
            terms(kd, cur + Ring::kAt.kd + own);
            zi[0] = *reinterpret_cast<const float4*>(cur + Ring::kZi + lane * 4);
            zi[1] = *reinterpret_cast<const float4*>(cur + Ring::kZi + 128 + lane * 4);
            g = *reinterpret_cast<const float4*>(cur + Ring::kG + w * 16 + (lane & 3) * 4);
            if constexpr (GENERAL) {
                terms(kv, cur + Ring::kAt.kv + own);
                vv = *reinterpret_cast<const uint4*>(cur + Ring::kVv + lane * 4);
            }
            next_chunk();
        };
        read_chunk();
        for (int c = 0; c < n_chunks; ++c) {
            const int parity = c & 1;
            TermsA a, az;
            terms_of(a, s[0], s[1]);
            float d[2][4];
            mma_terms(d[0], d[1], a, wm);  // this warp's rows' share of S0's part of Z
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                states[parity][j][w][lane] = make_float4(s[j][0], s[j][1], s[j][2], s[j][3]);
                shares[parity][j][w][lane] = make_float4(d[j][0], d[j][1], d[j][2], d[j][3]);
            }
            meet();
            const float decay[2][2] = {{g.x, g.y}, {g.z, g.w}};
            float written[2][4] = {};
            if constexpr (GENERAL) {  // + Kv^T V: the values are bfloat16 as they are
                const uint32_t v[4] = {vv.x, vv.y, vv.z, vv.w};
#pragma unroll
                for (int term = 2; term >= 0; --term) {
                    mma_bf16(written[0], v, kv.t[term].x, kv.t[term].y);
                    mma_bf16(written[1], v, kv.t[term].z, kv.t[term].w);
                }
            }
#pragma unroll
            for (int j = 0; j < 2; ++j) {
#pragma unroll
                for (int r = 0; r < 4; ++r) {
                    s[j][r] = fmaf(s[j][r], decay[j][r & 1], written[j][r]);
                }
            }
            float z[2][4], moved[2][4];
            sum_of_shares(z, zi, shares[parity], lane);
            terms_of(az, z[0], z[1]);
            mma_terms(moved[0], moved[1], az, kd);
            if (c + 1 < n_chunks) {
                read_chunk();  // (under the products' latency)
            }
#pragma unroll
            for (int j = 0; j < 2; ++j) {
#pragma unroll
                for (int r = 0; r < 4; ++r) {
                    s[j][r] += moved[j][r];
                }
            }
        }
        meet();
#pragma unroll
        for (int j = 0; j < 2; ++j) {
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                corner[static_cast<int64_t>(8 * j + (r & 1)) * p.vdim + (r >> 1) * 8] = lost ? NAN : s[j][r];
            }
        }
        return;
    }

    // This lane's outputs: columns lane / 4 and 8 on, tokens 8 w + (lane % 4) * 2 and the next (of the first two warps).
    const int done = p.pass.pass * p.pass.window * kDeltaChunk;
    const int rows = count - done;
    const int64_t o_stride = static_cast<int64_t>(p.n_heads) * p.vdim;
    int token = w * 8 + (lane & 3) * 2;
    float* dst = p.o_raw + (p.first_rows[e] + done + token) * o_stride +
        static_cast<int64_t>(head) * p.vdim + ct * kDeltaCols + (lane >> 2);
    float o[4] = {0.0f, 0.0f, 0.0f, 0.0f};
    auto finish = [&](int parity) {
#pragma unroll
        for (int other = 0; other < NW; ++other) {
            const float4 part = o_shares[parity][w][other][lane];
            o[0] += part.x;
            o[1] += part.y;
            o[2] += part.z;
            o[3] += part.w;
        }
        if (lost) {
            o[0] = o[1] = o[2] = o[3] = NAN;
        }
        if (token < rows) {
            dst[0] = o[0];
            dst[8] = o[2];
        }
        if (token + 1 < rows) {
            dst[o_stride] = o[1];
            dst[o_stride + 8] = o[3];
        }
        token += kDeltaChunk;
        dst += kDeltaChunk * o_stride;
    };
    for (int c = 0; c < n_chunks; ++c) {
        const int parity = c & 1;
        meet();  // the chunk's state and shares of Z are there, and the chunk before it was read by everyone
        if (brings && c > 0 && c - 1 + Ring::kSlots < n_chunks) {
            bring(c - 1 + Ring::kSlots);
        }
        wait_for_chunk();
        TermsB qg, m = {};
        terms(qg, cur + Ring::kAt.qg + own);
        float4 zi[2] = {}, oi = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (w < 2) {
            terms(m, cur + Ring::kAt.m + lane * 4);
            zi[0] = *reinterpret_cast<const float4*>(cur + Ring::kZi + lane * 4);
            zi[1] = *reinterpret_cast<const float4*>(cur + Ring::kZi + 128 + lane * 4);
            if constexpr (GENERAL) {
                oi = *reinterpret_cast<const float4*>(cur + Ring::kOi + (w * 32 + lane) * 4);
            }
        }
        next_chunk();
        float s[2][4], q[2][4];
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            const float4 part = states[parity][j][w][lane];
            s[j][0] = part.x;
            s[j][1] = part.y;
            s[j][2] = part.z;
            s[j][3] = part.w;
        }
        TermsA a;
        terms_of(a, s[0], s[1]);
        mma_terms(q[0], q[1], a, qg);  // this warp's rows' share of S0's part of O, read after the next barrier
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            o_shares[parity][j][w][lane] = make_float4(q[j][0], q[j][1], q[j][2], q[j][3]);
        }
        if (w < 2) {
            if (c > 0) {
                finish(parity ^ 1);  // the chunk before: its shares were written before this chunk's barrier
            }
            float z[2][4];
            TermsA az;
            sum_of_shares(z, zi, shares[parity], lane);
            terms_of(az, z[0], z[1]);
            chunk_outputs(o, size_of(z), az, m, oi, w, lane);
        }
    }
    meet();
    if (w < 2) {
        finish((n_chunks - 1) & 1);
    }
    if (brings && lost) {
        if (p.status != nullptr) {
            atomicOr(p.status, 8);
        }
        for (int spin = 0; spin < (1 << 16); ++spin) {
            __nanosleep(64);  // copies in flight land meanwhile
        }
    }
}

// Whether the outputs go to warps of their own (delta_chain_kernel) or the chain's warps make them too (delta_chain_joint_kernel).
// The former shortens the path from chunk to chunk, for chains that have an SM each, and keeps more copies in flight, for scratch
// that does not stay in L2; it needs twice the warps and a ring of shared memory, which many short chains wait for. Both give the same
// bits. Whole calls, 32 heads of 64 x 64, us, joint and apart: one entry of 1, 4, 12, 32, 64 chunks 15.4 and 16.8, 19.0 and 19.8, 28.4 and
// 24.7, 58.5 and 50.3, 107.5 and 88.2 (the general rule 16.4 and 13.3, 21.8 and 20.1, 33.5 and 28.8, 65.6 and 55.1, 120 and 104; 12
// heads 0.76 to 1.15 times as long up to 4 chunks); 12 entries of 1, 3, 8 (75 MB of scratch), 12 (112 MB) chunks 33 and 37, 55 and 60,
// 124 and 123, 192 and 171; the general rule, 5 entries of 4, 12 (70 MB), 16 (94 MB), 32 chunks 42 and 45, 99 and 100, 138 and 128, 277 and 238.
// Never ahead with more CTAs than SMs: 64 heads of 32 x 128 with a decay per channel (two entries of 32 chunks 144 and 167),
// and at most even where values are wider than keys.
template <int NW, bool GENERAL>
inline bool delta_chain_apart(int n_heads, int vdim, int64_t slots, int n_long, int64_t longest) {
    const int64_t ctas = static_cast<int64_t>(n_long) * n_heads * (vdim / kDeltaCols), chunks = slots / n_long;
    if (ctas <= 148) {
        return chunks >= (NW == 8 ? 6 : GENERAL ? 4 : 10);
    }
    const int64_t bytes = slots * n_heads * DeltaChunkLayout(NW * 16, vdim, GENERAL).floats * 4;
    const int64_t kept = (chunks >= 8 && vdim >= 64 ? 54 : 92) << 20;  // about what of L2 the matrices keep
    // (a chain much longer than the others, in all its passes, is a path again, on an SM that it shares: 1,500 tokens beside eight
    // portions of 20, 16 heads of 128 x 128, the general rule 344 and 367)
    return bytes >= kept && vdim <= NW * 16 && (NW > 2 ? longest < 4 * chunks : GENERAL);
}

template <int NW, bool GENERAL>
cudaError_t launch_delta_chain(const DeltaChainParams& p, int n_long, bool apart, cudaStream_t stream) {
    using Ring = DeltaRing<NW * 16, GENERAL>;
    if (!apart) {
        return pl_launch_overlapped(delta_chain_joint_kernel<NW, GENERAL>, dim3(n_long, p.n_heads, p.vdim / kDeltaCols),
                                    dim3(NW * 32), 0, stream, p);
    }
    // Where every CTA can have an SM to itself, more than half of one's shared memory sees to it: CTAs that come in while the
    // chunks' matrices still hold some SMs would otherwise share the others (one prompt: 135 us so, 95 alone).
    constexpr int kAlone = 120 * 1024, kMost = Ring::kBytes > kAlone ? Ring::kBytes : kAlone;
    if (const cudaError_t set = pl_allow_smem<delta_chain_kernel<NW, GENERAL>>(kMost); set != cudaSuccess) {
        return set;
    }
    const dim3 grid(n_long * p.n_heads, p.vdim / kDeltaCols);
    const bool alone = static_cast<int64_t>(grid.x) * grid.y <= 148;
    return pl_launch_overlapped(delta_chain_kernel<NW, GENERAL>, grid, dim3(NW * 64), alone ? kMost : Ring::kBytes, stream, p);
}

// The heads' norm over vdim, its weight and the gate: out = o * rsqrt(mean(o^2) + eps) * norm * sigmoid(gate), four values a
// lane, LANES lanes a (token, head). 2,048 tokens of 32 heads of 64: a warp a head took 23.4 us, this 11.6 (34 MB, 0.45 of the copy
// rate: short CTAs that load, wait once and store). norm_stride: distance between heads' norm weights (0: all heads have the same).
template <int LANES>
__global__ void __launch_bounds__(256) delta_finish_kernel(const float* __restrict__ o_raw, const float* __restrict__ norm,
                                                           int norm_stride, const __nv_bfloat16* __restrict__ gate_pre,
                                                           int64_t gate_stride, __nv_bfloat16* __restrict__ out,
                                                           int64_t out_stride, int n_tokens, int n_heads, int vdim, float eps) {
    pl_grid_trigger();
    const int64_t pair = (static_cast<int64_t>(blockIdx.x) * 256 + threadIdx.x) / LANES;
    const int d = threadIdx.x % LANES * 4;
    const int t = static_cast<int>(pair / n_heads), h = static_cast<int>(pair % n_heads);
    const bool there = t < n_tokens && d < vdim;
    float4 weight = make_float4(0.0f, 0.0f, 0.0f, 0.0f), o = weight, g = weight;
    if (there) {
        weight = *reinterpret_cast<const float4*>(norm + h * norm_stride + d);
    }
    pl_grid_wait();
    if (there) {
        o = *reinterpret_cast<const float4*>(o_raw + pair * vdim + d);
        g = pl_load4(gate_pre + t * gate_stride + h * vdim + d);
    }
    float square = fmaf(o.x, o.x, fmaf(o.y, o.y, fmaf(o.z, o.z, o.w * o.w)));
#pragma unroll
    for (int offset = LANES / 2; offset > 0; offset >>= 1) {
        square += __shfl_xor_sync(0xffffffffu, square, offset);
    }
    if (there) {
        const float factor = 1.0f / sqrtf(square / static_cast<float>(vdim) + eps);
        const float4 r = make_float4(o.x * factor * weight.x * (1.0f / (1.0f + expf(-g.x))),
                                     o.y * factor * weight.y * (1.0f / (1.0f + expf(-g.y))),
                                     o.z * factor * weight.z * (1.0f / (1.0f + expf(-g.z))),
                                     o.w * factor * weight.w * (1.0f / (1.0f + expf(-g.w))));
        pl_store4(out + t * out_stride + h * vdim + d, r);
    }
}

// Whether its loads of four values start where they have to.
inline bool delta_finish_supports(const float* norm, const void* gate_pre, int64_t gate_stride, const void* out,
                                  int64_t out_stride, int vdim) {
    return vdim % 4 == 0 && vdim <= 128 && gate_stride % 4 == 0 && out_stride % 4 == 0 &&
        (reinterpret_cast<uintptr_t>(norm) & 15) == 0 &&
        ((reinterpret_cast<uintptr_t>(gate_pre) | reinterpret_cast<uintptr_t>(out)) & 7) == 0;
}
inline void launch_delta_finish(const float* o_raw, const float* norm, int norm_stride, const void* gate_pre, int64_t gate_stride,
                                void* out, int64_t out_stride, int n_tokens, int n_heads, int vdim, float eps,
                                cudaStream_t stream) {
    const int lanes = vdim <= 16 ? 4 : vdim <= 32 ? 8 : vdim <= 64 ? 16 : 32;
    const int64_t threads = static_cast<int64_t>(n_tokens) * n_heads * lanes;
    auto kernel = lanes == 4 ? delta_finish_kernel<4> : lanes == 8 ? delta_finish_kernel<8>
                : lanes == 16 ? delta_finish_kernel<16> : delta_finish_kernel<32>;
    pl_launch_overlapped(kernel, dim3(static_cast<unsigned>((threads + 255) / 256)), dim3(256), 0, stream, o_raw, norm, norm_stride,
                         static_cast<const __nv_bfloat16*>(gate_pre), gate_stride, static_cast<__nv_bfloat16*>(out), out_stride,
                         n_tokens, n_heads, vdim, eps);
}

// Which form an entry's portion takes: up to step_most tokens the one of delta_step.cuh, from chunk_least on chunks, the walk
// between. By its own length alone, so that nothing else in the step moves a request's sums. The lines were drawn where neither side
// loses much from one entry to 64 of a length (us of a call with cold caches, one and 64 entries):
//   32 heads of 64 x 64, decay per channel: 2 tokens step 12 and 41, walk 12 and 59; 12 tokens walk 18 and 291, chunks 18 and 117
//   the general rule: 2 tokens 14 and 43, 12 and 74; 8 tokens walk 16 and 158, chunks 18 and 156; 12 tokens 21 and 217, 18 and 158
//   16 heads of 128 x 128: channel 12 tokens walk 25 and 684, chunks 20 and 213; general 29 and 520, 27 and 276
//   16 heads of 64 x 128: 12 tokens walk 18 and 287, chunks 23 and 107; 16 tokens 21 and 351, 23 and 110
//   64 heads of 32 x 32: 1 token step 10 and 31, walk 12 and 27; channel 12 tokens walk 16 and 123, chunks 16 and 94 (16 entries 41
//   and 33, four 18 and 21); general 24 tokens walk 18 and 150, chunks 18 and 191, 32 tokens 18 and 192, 18 and 197
struct DeltaForms {
    int step_most, chunk_least;
};
inline DeltaForms delta_forms(bool general, int dim, int vdim, int dtype, const void* state) {
    const bool sizes = dtype == PL_BF16 && (dim == 32 || dim == 64 || dim == 128);
    const bool small = dim * vdim <= 1024;
    const bool step = sizes && (vdim == 32 || vdim == 64 || vdim == 128) && (reinterpret_cast<uintptr_t>(state) & 15) == 0;
    const bool chunks = sizes && vdim % kDeltaCols == 0 && vdim <= 256;
    return {step && !small ? 2 : 0, !chunks ? INT_MAX : small ? (general ? 32 : 16) : vdim > dim ? 16 : 12};
}

// What a step's entries need: whether any takes the step form, the longest walk, how many go in chunks, their chunks in all and
// those of the longest.
struct DeltaStep {
    int singles, walk_longest, n_long, n_chunks, longest_chunks;
};
// Chunks of an entry in a pass, slots for chunks in one, and passes, where a chunk of a head takes `floats` of scratch.
inline int delta_window(const DeltaStep& step, int n_heads, int floats) {
    const int64_t each = static_cast<int64_t>(max(step.n_long, 1)) * n_heads * floats * 4;
    return static_cast<int>(min(static_cast<int64_t>(kDeltaWindow), max(static_cast<int64_t>(4), kDeltaScratchBytes / each)));
}
inline int64_t delta_chunk_slots(const DeltaStep& step, int window) {
    const int64_t most = static_cast<int64_t>(step.n_long) * window;
    return step.n_chunks < most ? step.n_chunks : most;
}
inline int delta_passes(const DeltaStep& step, int window) { return (step.longest_chunks + window - 1) / window; }

}  // namespace
