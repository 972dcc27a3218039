// bfloat16 matrix product for prompts on pairs of SMs:
//   Y[T, N] = X[T, K] * W[N, K]^T,  fp32 accumulation, T in the hundreds and up.
//
// Two CTAs of a cluster work on one 256-feature x 256-token tile with
// `tcgen05.mma.cta_group::2` (M = 256 over the pair, N = 256, K = 16 per instruction).
// The weights sit on the MMA's M axis and the tokens on its N axis, as in the other
// products of this library. Each CTA loads its own 128 features of W and its own 128
// of the tile's 256 tokens of X per 64-deep k block (32 KB where a lone CTA with a
// 128 x 256 tile of its own would need 48 KB for the same number of MMA cycles: one SM
// takes in about 64 bytes a clock, which held a single-CTA kernel of that tile to 0.6 -
// 0.7 of the GEMM peak); the instruction reads both CTAs' shared memory and writes each CTA's 128 rows of the accumulator into that
// CTA's tensor memory.
//
// Roles per CTA (192 threads): warp 0 loads with TMA (`.cta_group::2` loads, whose
// bytes are counted on the barrier of the pair's first CTA); warp 1 of the first CTA
// issues the MMAs for the pair and commits them to both CTAs' barriers
// (`tcgen05.commit ... multicast::cluster`), and owns (in both CTAs) the tensor
// memory allocation; warps 2-5 read their CTA's accumulator rows and store them.
// A chunk of 32 tokens leaves through shared memory in rows of 128 features, 16 bytes a store (a store of two bytes a lane
// and token was what bound tiles of few k blocks: 2,048 tokens by 32,000 rows of 2,048 took 271.6 us, now 159.7; gated,
// 16,384 rows, 131.1 and now 96.2; 28,672 rows of 4,096, bound by the MMAs, 307 and now 306).
// Tiles are 256 tokens high, or 192 where that leaves less of a round idle (tile_tokens below).
// Two accumulators let the epilogue of one tile overlap the MMAs of the next; the
// second CTA's epilogue releases an accumulator by arriving on the first CTA's barrier.
// A pair is persistent and takes every P-th whole tile (P pairs), token tiles fastest:
// the P tiles in work at one time are then neighbours that share a few weight tiles, so
// each weight tile comes from HBM once and is served to the other pairs from L2 (with a
// contiguous run of tiles per pair the pairs' weight tiles together overflow the L2 and
// every token tile re-reads its weights from HBM: 2.07 GB instead of 0.25 GB for the
// 2048 x 28672 x 4096 product).
//
// Gated mode: W holds two stacked matrices, gate over up ([2N, K]), and the kernel
// writes silu(gate x) * (up x) ([T, N]). A CTA's 128 rows are then 64 gate rows over
// the 64 up rows of the same features (two TMA boxes per stage); in the epilogue the
// warps that hold gate and up rows hand each other half of a chunk through shared memory,
// round both to bfloat16 (as a product that stored them would)
// and apply the activation (or the clamped unit of gate_units.cuh: a build of its own).
//
// Grouped mode: the rows of X belong to experts, one run of rows each (`ends`, made on the device), and W stacks the
// experts' matrices. A tile is 256 features (gated: 128) of one expert by up to 256 of its rows; an expert's rows are
// split evenly over as few tiles as hold them, and a tile's MMAs are only as wide as its rows (in steps of 32), so little
// is spent on padding. Rows of the next expert that a tile's last rows of 32 bring in are columns nobody stores. What bounds
// it: the loads where experts have few rows (16 KB of weights a CTA and k block, whatever the width), the MMAs from about
// 256 rows an expert on where k is long, the epilogue (0.9 us a chunk of 32 tokens) where it is not. us beside the library's grouped
// products (and a SwiGLU kernel behind the first), gated and down: 32 experts, 2,048 wide, 1,024 features, 64 rows an expert 58 and 35, 74
// and 45; 256 rows 69 and 44, 84 and 47; 1,024 rows 206 and 123, 234 and 107. 64 experts, 1,024 wide, 512 features, 64 rows 37 and 25,
// 48 and 28; 1,024 rows 143 and 106, 141 and 76: products over 1,024 and fewer features are behind the library's from about 512 rows an expert
// on, which the whole part shows past 4,096 tokens (8 of 64 experts, 8,192 tokens 489 and 514).
//
// Every wait on an mbarrier is bounded: after the limit the CTA raises bit 8 of the
// status word, stops issuing work, lets what is in flight land, meets its partner,
// frees its tensor memory and returns.
//
// The reference leaves these products to a library (`at::linear`,
// pulsarlm-core/src/engine/model/llama.cpp:67-69, 81, 91, 93).
#include <type_traits>

#include "gate_units.cuh"
#include "tcgen05_helpers.cuh"

namespace {

constexpr int kTileM = 128;    // features per CTA, 256 per pair
constexpr int kMostTokens = 256;  // tokens per tile (kPairN: this or 192), half of them loaded by each CTA
constexpr int kBlockK = 64;
constexpr int kThreads = 192;
constexpr int kStages = 6;
constexpr int kBytesA = kTileM * kBlockK * 2;
// Per CTA.
__host__ __device__ constexpr int stage_bytes(int tokens) { return kBytesA + tokens / 2 * kBlockK * 2; }

struct PairParams {
    void* y;  // [T, N] bf16 or fp32
    int t, n, k;  // n: output features (gated: W has 2n rows)
    int64_t ldy;
    int out_f32;
    float limit;  // (the clamped unit)
    int n_tiles;  // tiles along N (256 features each)
    int t_tiles;  // tiles along T (256 tokens each)
    int k_blocks;
    int total_tiles;
    int act;  // grouped, not gated: the plain activation of the rounded product (gate_units.cuh's codes, 0: none)
    const int32_t* ends;  // grouped: the row after each expert's last
    int n_experts;
    int32_t* status;
};

constexpr int kMostExperts = 512;  // of a grouped product (their tiles' running counts sit in shared memory)

// The rows of X one load brings in: half a tile's; grouped: boxes of 128, 64, 32 and 16 rows, of which a tile's half is made up.
template <bool GROUPED>
struct RowMaps {
    CUtensorMap box[GROUPED ? 4 : 1];
};

__device__ __forceinline__ uint32_t cluster_rank() {
    uint32_t rank;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
    return rank;
}
__device__ __forceinline__ void tcgen05_alloc_pair(uint32_t* slot, uint32_t columns) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(slot)),
                 "r"(columns)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tcgen05_dealloc_pair(uint32_t address, uint32_t columns) {
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(address), "r"(columns) : "memory");
}
// A tile load whose bytes are counted on the barrier at the same address in the pair's
// first CTA (both CTAs of the pair issue such loads for a stage).
__device__ __forceinline__ void tma_load_2d_pair(void* dst, const CUtensorMap* map, int x, int y, uint64_t* bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], "
        "[%2];"
        ::"r"(smem_u32(dst)), "l"(map), "r"(cluster_map(bar, 0)), "r"(x), "r"(y)
        : "memory");
}
__device__ __forceinline__ void tcgen05_mma_pair(uint32_t tmem_d, uint64_t desc_a, uint64_t desc_b, uint32_t idesc,
                                                 uint32_t accumulate) {
    const uint32_t zero = 0;  // no output lanes switched off
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, {%5, %5, %5, %5, %5, %5, %5, %5}, p;\n\t}"
        ::"r"(tmem_d), "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(accumulate), "r"(zero)
        : "memory");
}
// One arrival, once the MMAs issued so far have completed, on the barrier at this
// address in both CTAs of the pair.
__device__ __forceinline__ void tcgen05_commit_pair(uint64_t* bar) {
    const uint16_t both = 3;
    asm volatile(
        "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
        ::"r"(smem_u32(bar)), "h"(both)
        : "memory");
}
// One arrival on the barrier at this address in the pair's first CTA.
__device__ __forceinline__ void arrive_on_first(uint64_t* bar) {
    asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_map(bar, 0))
                 : "memory");
}

constexpr int kGateRow = 17;  // 16 token columns handed over per thread and chunk, padded against bank conflicts
constexpr int kGateBytes = 2 * 2 * (kTileM / 2) * kGateRow * 4;  // two buffers of [gate side, up side][64][17] floats

// An epilogue's chunk of 32 tokens on its way out: [32][PER features] of fp32 at most (grouped: bfloat16), two of them.
constexpr int out_bytes(int per, bool grouped) { return 2 * 32 * per * (grouped ? 2 : 4); }

template <typename T>
__device__ __forceinline__ T out_value(float v) {
    if constexpr (sizeof(T) == 4) {
        return v;
    } else {
        return __float2bfloat16_rn(v);
    }
}

// Rows t0 .. of a chunk [32][PER] in shared memory to y, 16 bytes a store where rows start on 16 bytes (by 128 threads).
template <int PER, typename T>
__device__ __forceinline__ void store_rows(const T* rows, T* y, int64_t ldy, int t0, int t_end, int n0, int n_end, bool vectors,
                                           int thread) {
    constexpr int kPer16 = 16 / sizeof(T), kLanes = PER / kPer16;
#pragma unroll
    for (int i = 0; i < 32 * kLanes / 128; ++i) {
        const int at = thread + 128 * i, t = t0 + at / kLanes, n = n0 + at % kLanes * kPer16;
        if (t < t_end && n < n_end) {
            const T* from = rows + at * kPer16;
            T* to = y + t * ldy + n;
            if (vectors && n + kPer16 <= n_end) {
                *reinterpret_cast<uint4*>(to) = *reinterpret_cast<const uint4*>(from);
            } else {
                for (int e = 0; e < kPer16 && n + e < n_end; ++e) {
                    to[e] = from[e];
                }
            }
        }
    }
}

// One tile: the features from n0 on (of the pair), the rows of W from w0 on are its first, rows t0 .. t_end of X, MMAs
// `wide` tokens wide.
struct PairTile {
    int n0, w0, t0, t_end, wide;
};

// Walks the tiles in ascending order. Grouped: expert by expert, within one the row tiles fastest, as in a plain product.
template <bool GROUPED, int PER_PAIR, int MOST>
struct PairTiles {
    const PairParams& p;
    const int* first;  // grouped: [n_experts + 1] tiles before each expert's, then rows before each expert's
    int expert = 0;
    __device__ __forceinline__ PairTiles(const PairParams& params, const int* counts): p(params), first(counts) {}
    __device__ __forceinline__ PairTile at(int tile) {
        if constexpr (!GROUPED) {
            const int n0 = (tile / p.t_tiles) * PER_PAIR;
            return {n0, n0, (tile % p.t_tiles) * MOST, p.t, MOST};
        } else {
            while (tile >= first[expert + 1]) {
                ++expert;
            }
            const int* row = first + kMostExperts + 1;
            const int begin = row[expert], end = row[expert + 1];
            const int row_tiles = (end - begin + MOST - 1) / MOST, in = tile - first[expert];
            const int rows = ((end - begin + row_tiles - 1) / row_tiles + 31) / 32 * 32;
            const int n0 = in / row_tiles * PER_PAIR, t0 = begin + in % row_tiles * rows, t_end = min(end, t0 + rows);
            return {n0, expert * p.n * (PER_PAIR == kTileM ? 2 : 1) + n0, t0, t_end, (t_end - t0 + 31) / 32 * 32};
        }
    }
};

// GATED: 0 the product alone, 1 silu(gate) * up, 2 the clamped unit of gate and up.
template <int GATED, int kPairN, bool GROUPED>
__global__ void __launch_bounds__(kThreads, 1)
gemm_pair_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ RowMaps<GROUPED> map_x,
                 const PairParams p) {
    constexpr uint32_t kColumns = 2 * kMostTokens;  // two accumulators, kPairN columns of each half (a power of two is allotted)
    constexpr int kStageBytes = stage_bytes(kPairN);
    constexpr uint32_t kIdesc = (1u << 4) | (1u << 7) | (1u << 10) | (static_cast<uint32_t>((2 * kTileM) >> 4) << 24);

    extern __shared__ unsigned char raw_smem[];
    unsigned char* tiles = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(raw_smem) + 1023) &
                                                            ~static_cast<uintptr_t>(1023));
    float* handover = reinterpret_cast<float*>(tiles + kStages * kStageBytes);  // gated: [2][2][64][17]
    constexpr int kPer = GATED ? kTileM / 2 : kTileM;      // output features per CTA and tile
    unsigned char* leaving = tiles + kStages * kStageBytes + (GATED ? kGateBytes : 0);  // [2][32][kPer]
    __shared__ __align__(8) uint64_t full_bar[kStages];   // waited on in the first CTA only
    __shared__ __align__(8) uint64_t empty_bar[kStages];
    __shared__ __align__(8) uint64_t acc_full[2];
    __shared__ __align__(8) uint64_t acc_empty[2];         // waited on in the first CTA only
    __shared__ uint32_t tmem_base_slot;
    __shared__ int abort_flag;
    __shared__ int first_tile[GROUPED ? 2 * (kMostExperts + 1) : 1];

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int rank = static_cast<int>(cluster_rank());
    const int pair = blockIdx.x >> 1;
    pl_grid_trigger();
    if (threadIdx.x == 0) {
        tensormap_prefetch(&map_w);
        tensormap_prefetch(&map_x.box[0]);
        for (int s = 0; s < kStages; ++s) {
            mbar_init(&full_bar[s], 1);
            mbar_init(&empty_bar[s], 1);
        }
        for (int a = 0; a < 2; ++a) {
            mbar_init(&acc_full[a], 1);
            mbar_init(&acc_empty[a], 8);  // the epilogue warps of both CTAs
        }
        abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        tcgen05_alloc_pair(&tmem_base_slot, kColumns);
    }
    tcgen05_fence_before();
    __syncthreads();
    tcgen05_fence_after();
    const uint32_t tmem_base = __shfl_sync(0xffffffffu, tmem_base_slot, 0);
    cluster_arrive_all();  // both CTAs' barriers exist before either signals the other's
    cluster_wait_all();
    pl_grid_wait();

    if constexpr (GROUPED) {
        if (warp == 0) {
            int before = 0;
            for (int base = 0; base < p.n_experts; base += 32) {
                const int e = base + lane;
                int upto = 0;
                if (e < p.n_experts) {
                    const int end = p.ends[e], rows = end - (e > 0 ? p.ends[e - 1] : 0);
                    first_tile[kMostExperts + 2 + e] = end;
                    upto = (rows + kPairN - 1) / kPairN * p.n_tiles;
                }
#pragma unroll
                for (int offset = 1; offset < 32; offset <<= 1) {
                    const int other = __shfl_up_sync(0xffffffffu, upto, offset);
                    upto += lane >= offset ? other : 0;
                }
                if (e < p.n_experts) {
                    first_tile[e + 1] = before + upto;
                }
                before += __shfl_sync(0xffffffffu, upto, 31);
            }
            if (lane == 0) {
                first_tile[0] = 0;
                first_tile[kMostExperts + 1] = 0;
            }
        }
        __syncthreads();
    }
    const int tile_begin = pair, tile_end = GROUPED ? first_tile[p.n_experts] : p.total_tiles, tile_step = gridDim.x >> 1;
    PairTiles<GROUPED, 2 * kPer, kPairN> places(p, first_tile);

    if (warp == 0) {
        // ------------------------------------------------ producer (both CTAs)
        int stage = 0;
        uint32_t phase = 0;
        bool ok = true;
        for (int tile = tile_begin; ok && tile < tile_end; tile += tile_step) {
            const PairTile place = places.at(tile);
            const int w0 = place.w0 + rank * kPer;
            const int t0 = place.t0 + rank * (place.wide / 2);
            for (int kb = 0; kb < p.k_blocks; ++kb) {
                if (!mbar_wait(&empty_bar[stage], phase ^ 1u, &abort_flag)) {
                    ok = false;
                    break;
                }
                unsigned char* a = tiles + stage * kStageBytes;
                if (elect_one()) {
                    if (rank == 0) {
                        mbar_expect_tx(&full_bar[stage], 2 * stage_bytes(place.wide));  // both CTAs' loads of this stage
                    }
                    tma_load_2d_pair(a, &map_w, kb * kBlockK, w0, &full_bar[stage]);
                    if (GATED) {  // the up rows of the same features under the gate rows
                        tma_load_2d_pair(a + kBytesA / 2, &map_w, kb * kBlockK, p.n + w0, &full_bar[stage]);
                    }
                    if constexpr (GROUPED) {
                        int row = 0;
#pragma unroll
                        for (int i = 0; i < 4; ++i) {
                            if (place.wide / 2 & (kMostTokens / 2 >> i)) {
                                tma_load_2d_pair(a + kBytesA + row * kBlockK * 2, &map_x.box[i], kb * kBlockK, t0 + row, &full_bar[stage]);
                                row += kMostTokens / 2 >> i;
                            }
                        }
                    } else {
                        tma_load_2d_pair(a + kBytesA, &map_x.box[0], kb * kBlockK, t0, &full_bar[stage]);
                    }
                }
                __syncwarp();
                if (++stage == kStages) {
                    stage = 0;
                    phase ^= 1u;
                }
            }
        }
    } else if (warp == 1 && rank == 0) {
        // ------------------------------------------------ MMA issuer (the pair's first CTA)
        int stage = 0;
        uint32_t phase = 0;
        bool ok = true;
        for (int tile = tile_begin; ok && tile < tile_end; tile += tile_step) {
            const int run = (tile - tile_begin) / tile_step;
            const int acc = run & 1;
            if (!mbar_wait_cluster(&acc_empty[acc], ((run >> 1) & 1u) ^ 1u, &abort_flag)) {
                break;
            }
            tcgen05_fence_after();
            const uint32_t tmem_d = tmem_base + acc * kMostTokens;
            const uint32_t idesc = kIdesc | (static_cast<uint32_t>(GROUPED ? places.at(tile).wide >> 3 : kPairN >> 3) << 17);
            for (int kb = 0; kb < p.k_blocks; ++kb) {
                if (!mbar_wait(&full_bar[stage], phase, &abort_flag)) {
                    ok = false;
                    break;
                }
                tcgen05_fence_after();
                const unsigned char* a = tiles + stage * kStageBytes;
                const uint64_t desc_a = smem_descriptor(a), desc_b = smem_descriptor(a + kBytesA);
                if (elect_one()) {
#pragma unroll
                    for (int k = 0; k < kBlockK / 16; ++k) {
                        tcgen05_mma_pair(tmem_d, desc_a + 2 * k, desc_b + 2 * k, idesc, (kb > 0 || k > 0) ? 1u : 0u);
                    }
                    tcgen05_commit_pair(&empty_bar[stage]);  // frees the stage in both CTAs
                }
                __syncwarp();
                if (++stage == kStages) {
                    stage = 0;
                    phase ^= 1u;
                }
            }
            if (!ok) {
                break;
            }
            if (elect_one()) {
                tcgen05_commit_pair(&acc_full[acc]);  // both CTAs' epilogues may read
            }
            __syncwarp();
        }
    } else if (warp >= 2) {
        // ------------------------------------------------ epilogue (warps 2..5, both CTAs)
        const int lane_group = warp & 3;  // the tensor-memory lanes a warp may read: 32 * (warp % 4)
        const int feature = lane_group * 32 + lane;
        const int thread = (warp - 2) * 32 + lane;
        const bool vectors = p.ldy * (p.out_f32 ? 4 : 2) % 16 == 0 && (reinterpret_cast<uintptr_t>(p.y) & 15) == 0;
        for (int tile = tile_begin; tile < tile_end; tile += tile_step) {
            const int run = (tile - tile_begin) / tile_step;
            const int acc = run & 1;
            // (All four warps go on or none does: they meet at barriers below. Behind this one the last tile's chunks
            // have left.)
            int go = mbar_wait(&acc_full[acc], (run >> 1) & 1u, &abort_flag) ? 1 : 0;
            asm volatile(
                "{\n\t.reg .pred p, q;\n\tsetp.ne.b32 p, %0, 0;\n\tbarrier.cta.red.and.pred q, 1, 128, p;\n\t"
                "selp.b32 %0, 1, 0, q;\n\t}"
                : "+r"(go)::"memory");
            if (!go) {
                break;
            }
            tcgen05_fence_after();
            const PairTile place = places.at(tile);
            const int n_first = place.n0 + rank * kPer;
            const int n = n_first + (GATED ? feature % kPer : feature);
            const int t0 = place.t0, t_end = place.t_end;
            const uint32_t tmem_row = tmem_base + (static_cast<uint32_t>(lane_group * 32) << 16) + acc * kMostTokens;
#pragma unroll 1
            for (int c0 = 0; c0 < kPairN && t0 + c0 < t_end; c0 += 32) {
                uint32_t v[32];
                tcgen05_ld32_nowait(tmem_row + c0, v);
                tcgen05_wait_ld();
                if (GATED) {
                    // Lanes 0..63 hold gate rows, lanes 64..127 the up rows of the same features.
                    // Each side hands the other half of its chunk: the gate threads then have
                    // both values for the chunk's first 16 tokens, the up threads for the last 16.
                    const bool is_up = feature >= kPer;
                    const int mine = is_up ? 16 : 0;  // the columns this thread finishes
                    float* buffer = handover + ((c0 >> 5) & 1) * (2 * kPer * kGateRow) +
                        (is_up ? 0 : kPer * kGateRow) + (feature % kPer) * kGateRow;
#pragma unroll
                    for (int c = 0; c < 16; ++c) {
                        buffer[c] = __uint_as_float(is_up ? v[c] : v[16 + c]);  // the half the partner finishes
                    }
                    asm volatile("bar.sync 1, 128;" ::: "memory");  // (two buffers: one barrier per chunk is enough)
                    if (n < p.n) {
                        // (loads, arithmetic and stores in separate sweeps: a store between two
                        // loads would keep the compiler from overlapping the elements' latencies)
                        const float* theirs = handover + ((c0 >> 5) & 1) * (2 * kPer * kGateRow) +
                            (is_up ? kPer * kGateRow : 0) + (feature % kPer) * kGateRow;
                        float other[16], act[16];
#pragma unroll
                        for (int c = 0; c < 16; ++c) {
                            other[c] = theirs[c];
                        }
#pragma unroll
                        for (int c = 0; c < 16; ++c) {
                            const float own = __uint_as_float(is_up ? v[16 + c] : v[c]);
                            // both products rounded as a product that stored them would round them
                            const float g = __bfloat162float(__float2bfloat16_rn(is_up ? other[c] : own));
                            const float u = __bfloat162float(__float2bfloat16_rn(is_up ? own : other[c]));
                            act[c] = GATED == 2 ? pl_clamped_unit<false>(g, u, p.limit) : __fdividef(g, 1.0f + __expf(-g)) * u;
                        }
                        auto put = [&](auto* rows) {
                            using T = std::remove_reference_t<decltype(*rows)>;
#pragma unroll
                            for (int c = 0; c < 16; ++c) {
                                rows[(mine + c) * kPer + feature % kPer] = out_value<T>(act[c]);
                            }
                        };
                        if (!GROUPED && p.out_f32) {
                            put(reinterpret_cast<float*>(leaving) + ((c0 >> 5) & 1) * 32 * kPer);
                        } else {
                            put(reinterpret_cast<__nv_bfloat16*>(leaving) + ((c0 >> 5) & 1) * 32 * kPer);
                        }
                    }
                } else {
                    auto put = [&](auto* rows) {
                        using T = std::remove_reference_t<decltype(*rows)>;
#pragma unroll
                        for (int c = 0; c < 32; ++c) {
                            float z = __uint_as_float(v[c]);
                            if (GROUPED && p.act != 0) {  // (of the product rounded as one that stored it would round it)
                                z = pl_plain_activation(__bfloat162float(__float2bfloat16_rn(z)), p.act);
                            }
                            rows[c * kPer + feature] = out_value<T>(z);
                        }
                    };
                    if (!GROUPED && p.out_f32) {
                        put(reinterpret_cast<float*>(leaving) + ((c0 >> 5) & 1) * 32 * kPer);
                    } else {
                        put(reinterpret_cast<__nv_bfloat16*>(leaving) + ((c0 >> 5) & 1) * 32 * kPer);
                    }
                }
                asm volatile("bar.sync 1, 128;" ::: "memory");  // (two chunks' places: one barrier per chunk is enough)
                if (!GROUPED && p.out_f32) {
                    store_rows<kPer>(reinterpret_cast<const float*>(leaving) + ((c0 >> 5) & 1) * 32 * kPer,
                                     static_cast<float*>(p.y), p.ldy, t0 + c0, t_end, n_first, p.n, vectors, thread);
                } else {
                    store_rows<kPer>(reinterpret_cast<const __nv_bfloat16*>(leaving) + ((c0 >> 5) & 1) * 32 * kPer,
                                     static_cast<__nv_bfloat16*>(p.y), p.ldy, t0 + c0, t_end, n_first, p.n, vectors, thread);
                }
            }
            tcgen05_fence_before();
            __syncwarp();
            if (lane == 0) {
                arrive_on_first(&acc_empty[acc]);
            }
        }
    }

    // ---------------------------------------------------- teardown
    __syncwarp();
    tcgen05_fence_before();
    __syncthreads();
    if (abort_flag) {
        if (threadIdx.x == 0) {
            if (p.status != nullptr) {
                atomicOr(p.status, 8);
            }
            for (uint32_t spin = 0; spin < (1u << 16); ++spin) {
                __nanosleep(64);  // loads in flight land meanwhile
            }
        }
        __syncthreads();
    }
    // Neither CTA leaves while its partner may still read its shared memory (MMAs) or
    // arrive on its barriers.
    cluster_arrive_all();
    cluster_wait_all();
    if (warp == 1) {
        tcgen05_fence_after();
        tcgen05_dealloc_pair(tmem_base, kColumns);
    }
}

int pair_count() {
    static int pairs = 0;
    if (pairs == 0) {
        int device = 0, sms = 0;
        cudaGetDevice(&device);
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
        pairs = sms / 2;
    }
    return pairs;
}

}  // namespace

// 1 when pl_gemm_bf16_pair takes these sizes (rows of X and W on 16-byte boundaries).
PL_API int pl_gemm_bf16_pair_supports(int t, int n, int k, int64_t ldx, int64_t ldw) {
    return t >= 1 && n >= 1 && k >= 8 && k % 8 == 0 && ldx % 8 == 0 && ldw % 8 == 0;
}

namespace {

template <int GATED, int TOKENS, bool GROUPED = false>
int launch_pair(const CUtensorMap& map_w, const RowMaps<GROUPED>& map_x, const PairParams& p, int used_pairs,
                cudaStream_t stream) {
    constexpr int smem =
        kStages * stage_bytes(TOKENS) + (GATED ? kGateBytes : 0) + out_bytes(GATED ? kTileM / 2 : kTileM, GROUPED) + 1024;
    if (const cudaError_t err = pl_allow_smem<gemm_pair_kernel<GATED, TOKENS, GROUPED>>(smem); err != cudaSuccess) {
        return pl_fail(3, "gemm_bf16_pair: cannot set shared memory size: %s", cudaGetErrorString(err));
    }
    cudaLaunchConfig_t config = {};
    config.gridDim = dim3(2 * used_pairs);
    config.blockDim = dim3(kThreads);
    config.dynamicSmemBytes = smem;
    config.stream = stream;
    cudaLaunchAttribute attributes[2];
    attributes[0].id = cudaLaunchAttributeClusterDimension;
    attributes[0].val.clusterDim.x = 2;
    attributes[0].val.clusterDim.y = 1;
    attributes[0].val.clusterDim.z = 1;
    attributes[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attributes[1].val.programmaticStreamSerializationAllowed = 1;
    config.attrs = attributes;
    config.numAttrs = pl_overlap_enabled() ? 2 : 1;
    const cudaError_t err = cudaLaunchKernelEx(&config, gemm_pair_kernel<GATED, TOKENS, GROUPED>, map_w, map_x, p);
    if (err != cudaSuccess) {
        return pl_fail(3, "gemm_bf16_pair: launch failed: %s", cudaGetErrorString(err));
    }
    return 0;
}

// Tokens of a tile: 256, or 192 where the pairs' rounds of tiles then take less time: a round of 192 takes 0.82 of one of
// 256 (0.235 us a k block against 0.277 in few rounds, 0.79 in many). Gated, 16,384 rows of 2,048: 552 tokens 45.1 against
// 51.2 us, 1,536 tokens 77.8 against 84.0, 512 tokens 45.1 against 41.0, 2,048 tokens 102.4 against 96.2; 28,672 rows of
// 4,096: 552 tokens 104.4 against 120.8, 1,024 tokens 180.2 against 162.0.
int tile_tokens(int t, int n_tiles) {
    const int64_t pairs = pair_count();
    auto rounds = [&](int tokens) {
        const int64_t tiles = static_cast<int64_t>(n_tiles) * ((t + tokens - 1) / tokens);
        return (tiles + pairs - 1) / pairs;
    };
    return rounds(192) * 41 < rounds(256) * 50 ? 192 : 256;
}

}  // namespace

// y[T, N] (bf16, or fp32 when out_f32) = x[T, K] w[N, K]^T with bf16 x and w, on
// pairs of SMs; meant for hundreds of tokens and more (a tile is 256 x 256). With
// `gated`, w is [2N, K] (a gate matrix over an up matrix) and
// y = silu(x gate^T) * (x up^T), both products rounded to bfloat16 first (a tile is
// then 128 output features x 256 tokens).
static int run_pair(const void* x, const void* w, void* y, int t, int n, int k, int64_t ldx, int64_t ldw, int64_t ldy,
                    int out_f32, int gated, float limit, int32_t* status, cudaStream_t stream) {
    PL_REQUIRE(pl_gemm_bf16_pair_supports(t, n, k, ldx, ldw),
               "gemm_bf16_pair: unsupported sizes t=%d n=%d k=%d ldx=%lld ldw=%lld (k and the leading dimensions "
               "must be multiples of 8)",
               t, n, k, static_cast<long long>(ldx), static_cast<long long>(ldw));
    PL_REQUIRE((reinterpret_cast<uintptr_t>(x) & 15) == 0 && (reinterpret_cast<uintptr_t>(w) & 15) == 0,
               "gemm_bf16_pair: operands must be 16-byte aligned");
    PL_REQUIRE(ldy >= n, "gemm_bf16_pair: ldy=%lld is smaller than n=%d", static_cast<long long>(ldy), n);
    const int per_pair = gated ? kTileM : 2 * kTileM;  // output features of a tile
    CUtensorMap map_w;
    RowMaps<false> map_x;
    if (const int code = make_map(&map_w, w, gated ? 2 * static_cast<int64_t>(n) : n, k, ldw,
                                  gated ? kTileM / 2 : kTileM, kBlockK)) {
        return code;
    }
    const int tokens = tile_tokens(t, (n + per_pair - 1) / per_pair);
    if (const int code = make_map(&map_x.box[0], x, t, k, ldx, tokens / 2, kBlockK)) {
        return code;
    }
    PairParams p = {};
    p.y = y;
    p.t = t;
    p.n = n;
    p.k = k;
    p.ldy = ldy;
    p.out_f32 = out_f32;
    p.limit = limit;
    p.n_tiles = (n + per_pair - 1) / per_pair;
    p.t_tiles = (t + tokens - 1) / tokens;
    p.k_blocks = (k + kBlockK - 1) / kBlockK;
    p.total_tiles = p.n_tiles * p.t_tiles;
    const int used_pairs = p.total_tiles < pair_count() ? p.total_tiles : pair_count();
    p.status = status;
    if (tokens == 192) {
        return gated == 2 ? launch_pair<2, 192>(map_w, map_x, p, used_pairs, stream)
            : gated       ? launch_pair<1, 192>(map_w, map_x, p, used_pairs, stream)
                          : launch_pair<0, 192>(map_w, map_x, p, used_pairs, stream);
    }
    return gated == 2 ? launch_pair<2, 256>(map_w, map_x, p, used_pairs, stream)
        : gated       ? launch_pair<1, 256>(map_w, map_x, p, used_pairs, stream)
                      : launch_pair<0, 256>(map_w, map_x, p, used_pairs, stream);
}

PL_API int pl_gemm_bf16_pair(const void* x, const void* w, void* y, int t, int n, int k, int64_t ldx, int64_t ldw,
                             int64_t ldy, int out_f32, int gated, int32_t* status, cudaStream_t stream) {
    return run_pair(x, w, y, t, n, k, ldx, ldw, ldy, out_f32, gated != 0, 0.0f, status, stream);
}

// Gated, with the clamped unit (gate_units.cuh) of the two rounded products in the place of silu(gate) * up.
PL_API int pl_gemm_bf16_pair_clamped(const void* x, const void* w, void* y, int t, int n, int k, int64_t ldx, int64_t ldw,
                                     int64_t ldy, int out_f32, float limit, int32_t* status, cudaStream_t stream) {
    return run_pair(x, w, y, t, n, k, ldx, ldw, ldy, out_f32, 2, limit, status, stream);
}

// 1 when pl_gemm_bf16_grouped takes these sizes (all operands contiguous, on 16-byte boundaries).
PL_API int pl_gemm_bf16_grouped_supports(int n, int k, int n_experts) {
    return n >= 1 && k >= 8 && k % 8 == 0 && n_experts >= 1 && n_experts <= kMostExperts;
}

// Rows of experts by their matrices: y[r] = x[r] w[e]^T for the rows r of expert e, ends[e - 1] <= r < ends[e] (ends int32
// [n_experts] on the device, ascending, the last at most `rows`). x bf16 [rows, k]; w bf16 [n_experts, n, k], gated
// [n_experts, 2n, k] (an expert's gate matrix over its up matrix); y bf16 [rows, n]. gated: 1 silu(gate) * up, 2 the clamped
// unit with `limit`, of the two products rounded to bfloat16; 0 with `act`: the plain activation of the rounded product.
PL_API int pl_gemm_bf16_grouped(const void* x, const void* w, void* y, const int32_t* ends, int rows, int n, int k, int n_experts,
                                int gated, float limit, int act, int32_t* status, cudaStream_t stream) {
    PL_REQUIRE(pl_gemm_bf16_grouped_supports(n, k, n_experts) && rows >= 0 && gated >= 0 && gated <= 2,
               "gemm_bf16_grouped: unsupported sizes rows=%d n=%d k=%d experts=%d", rows, n, k, n_experts);
    PL_REQUIRE(act == 0 || (gated == 0 && act >= 1 && act <= 3), "gemm_bf16_grouped: unknown activation %d", act);
    PL_REQUIRE(((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(w)) & 15) == 0,
               "gemm_bf16_grouped: operands must be 16-byte aligned");
    if (rows == 0) {
        return 0;
    }
    const int per_pair = gated ? kTileM : 2 * kTileM;
    const int64_t w_rows = static_cast<int64_t>(n_experts) * n * (gated ? 2 : 1);
    PL_REQUIRE(w_rows + 2 * kTileM <= INT32_MAX, "gemm_bf16_grouped: %lld rows of weights are too many",
               static_cast<long long>(w_rows));
    CUtensorMap map_w;
    RowMaps<true> map_x;
    if (const int code = make_map(&map_w, w, w_rows, k, k, gated ? kTileM / 2 : kTileM, kBlockK)) {
        return code;
    }
    for (int i = 0; i < 4; ++i) {
        if (const int code = make_map(&map_x.box[i], x, rows, k, k, kMostTokens / 2 >> i, kBlockK)) {
            return code;
        }
    }
    PairParams p = {};
    p.y = y;
    p.t = rows;
    p.n = n;
    p.k = k;
    p.ldy = n;
    p.limit = limit;
    p.n_tiles = (n + per_pair - 1) / per_pair;
    p.k_blocks = (k + kBlockK - 1) / kBlockK;
    p.act = act;
    p.ends = ends;
    p.n_experts = n_experts;
    p.status = status;
    // (how many tiles there are is known on the device: at most this many)
    const int64_t most = static_cast<int64_t>(p.n_tiles) * (static_cast<int64_t>(n_experts) + rows / kMostTokens);
    const int used_pairs = most < pair_count() ? static_cast<int>(most) : pair_count();
    return gated == 2 ? launch_pair<2, kMostTokens, true>(map_w, map_x, p, used_pairs, stream)
        : gated       ? launch_pair<1, kMostTokens, true>(map_w, map_x, p, used_pairs, stream)
                      : launch_pair<0, kMostTokens, true>(map_w, map_x, p, used_pairs, stream);
}
