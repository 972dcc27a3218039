// True 32-bit matrix product for the float32 engine: C[M, N] = A[M, K] * W[N, K]^T.
//
// CUDA-core FMAs only: no tensor cores, no TF32. Each output element is one chain
// of fmaf over k = 0 .. K-1 in ascending order, whatever M is, so a token's row
// does not depend on what else is in the batch or on how a prompt was cut. All kernels
// below make that same chain, so their results are equal bit for bit and which of them
// runs is a matter of time alone.
#include "common.cuh"

#include "mma_helpers.cuh"

namespace {

struct GemmF32Params {
    const float* a;
    const float* w;
    float* c;
    int m, n, k, lda, ldw, ldc, accumulate;
};

__device__ __forceinline__ void put(const GemmF32Params& p, int row, int col, float v) {
    if (row < p.m && col < p.n) {
        float* dst = p.c + static_cast<int64_t>(row) * p.ldc + col;
        *dst = p.accumulate ? *dst + v : v;
    }
}

// ---------------------------------------------------------------------------- any address and stride
// 256 threads; thread (ty, tx) of a 16x16 grid owns a 4x4 block of the 64x64 tile. For operands whose
// rows do not start on 16 bytes.
constexpr int kTileM = 64;
constexpr int kTileN = 64;
constexpr int kTileK = 16;

__global__ void __launch_bounds__(256) gemm_f32_any_kernel(const GemmF32Params p) {
    __shared__ float as[kTileK][kTileM + 1];
    __shared__ float ws[kTileK][kTileN + 1];
    const int tx = threadIdx.x % 16, ty = threadIdx.x / 16;
    const int m0 = blockIdx.y * kTileM, n0 = blockIdx.x * kTileN;

    float acc[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            acc[i][j] = 0.0f;
        }
    }

    for (int k0 = 0; k0 < p.k; k0 += kTileK) {
        // 64 rows x 16 k of each operand: 1024 elements, 4 per thread; consecutive
        // threads read consecutive k of one row.
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int e = threadIdx.x + i * 256;
            const int row = e / kTileK, kk = e % kTileK;
            const int gk = k0 + kk;
            as[kk][row] = (m0 + row < p.m && gk < p.k) ? p.a[static_cast<int64_t>(m0 + row) * p.lda + gk] : 0.0f;
            ws[kk][row] = (n0 + row < p.n && gk < p.k) ? p.w[static_cast<int64_t>(n0 + row) * p.ldw + gk] : 0.0f;
        }
        __syncthreads();
#pragma unroll
        for (int kk = 0; kk < kTileK; ++kk) {
            float av[4], wv[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                av[i] = as[kk][ty * 4 + i];
                wv[i] = ws[kk][tx * 4 + i];
            }
#pragma unroll
            for (int i = 0; i < 4; ++i) {
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    acc[i][j] = fmaf(av[i], wv[j], acc[i][j]);
                }
            }
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            put(p, m0 + ty * 4 + i, n0 + tx * 4 + j, acc[i][j]);
        }
    }
}

// ---------------------------------------------------------------------------- tiles
// Two chains a step: fma.rn.f32x2 rounds each half as fmaf does.
__device__ __forceinline__ void fma2(uint64_t& acc, uint64_t a, uint64_t b) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(a), "l"(b));
}
__device__ __forceinline__ uint64_t twice(float v) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %1};" : "=l"(r) : "f"(v));
    return r;
}

// Rows of four floats along k, zeros past the operand's rows and past k.
__device__ __forceinline__ float4 load_row4(const float* base, int ld, int row, int rows, int gk, int k) {
    float4 v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    if (row < rows) {
        const float* src = base + static_cast<int64_t>(row) * ld + gk;
        if (gk + 3 < k) {
            v = *reinterpret_cast<const float4*>(src);
        } else {
            if (gk < k) v.x = src[0];
            if (gk + 1 < k) v.y = src[1];
            if (gk + 2 < k) v.z = src[2];
        }
    }
    return v;
}

// A BM x BN tile per CTA, RM rows x RN columns a thread (both in runs of four), both operands in shared memory
// with k outermost, the next 16 k in registers meanwhile. A thread reads its RM + RN operands of a k
// AHEAD k before their fmafs. What bounds it: shared memory hands a warp one operand a lane and cycle while the
// SM's four schedulers do four fmafs a lane and cycle, so RM x RN / (RM + RN) has to stay above four (8 x 16: 5.3;
// 8 x 8: 4). For products of hundreds of rows and many tiles: 16384 x 2048, 509 rows 690 us (50 TFLOP/s).
template <int BM, int BN, int RM, int RN, int AHEAD, int CTAS>
__global__ void __launch_bounds__(BM * BN / (RM * RN), CTAS) gemm_f32_tile_kernel(const GemmF32Params p) {
    constexpr int kThreads = BM * BN / (RM * RN);
    constexpr int BK = 16;
    constexpr int kLdA = BM + 4, kLdW = BN + 4;
    constexpr int kTx = BN / RN;
    constexpr int kTy = BM / RM;
    constexpr int kLoadsA = BM * BK / 4 / kThreads, kLoadsW = BN * BK / 4 / kThreads;
    constexpr int kBufs = AHEAD + 1;
    static_assert(kLoadsA >= 1 && kLoadsW >= 1 && kTx * kTy == kThreads && RM % 4 == 0 && RN % 4 == 0, "tile");
    extern __shared__ __align__(16) float tile_smem[];
    float (*as)[BK][kLdA] = reinterpret_cast<float (*)[BK][kLdA]>(tile_smem);
    float (*ws)[BK][kLdW] = reinterpret_cast<float (*)[BK][kLdW]>(tile_smem + 2 * BK * kLdA);
    const int tid = threadIdx.x;
    const int tx = tid % kTx, ty = tid / kTx;
    const int m0 = blockIdx.x * BM, n0 = blockIdx.y * BN;

    uint64_t acc[RM][RN / 2];
#pragma unroll
    for (int i = 0; i < RM; ++i) {
#pragma unroll
        for (int j = 0; j < RN / 2; ++j) {
            acc[i][j] = 0;
        }
    }
    float4 la[kLoadsA], lw[kLoadsW];
    auto fetch = [&](int k0) {
#pragma unroll
        for (int i = 0; i < kLoadsA; ++i) {
            const int e = tid + i * kThreads;
            la[i] = load_row4(p.a, p.lda, m0 + e / 4, p.m, k0 + (e % 4) * 4, p.k);
        }
#pragma unroll
        for (int i = 0; i < kLoadsW; ++i) {
            const int e = tid + i * kThreads;
            lw[i] = load_row4(p.w, p.ldw, n0 + e / 4, p.n, k0 + (e % 4) * 4, p.k);
        }
    };
    auto stash = [&](int buffer) {
#pragma unroll
        for (int i = 0; i < kLoadsA; ++i) {
            const int e = tid + i * kThreads, row = e / 4, kk = (e % 4) * 4;
            as[buffer][kk][row] = la[i].x;
            as[buffer][kk + 1][row] = la[i].y;
            as[buffer][kk + 2][row] = la[i].z;
            as[buffer][kk + 3][row] = la[i].w;
        }
#pragma unroll
        for (int i = 0; i < kLoadsW; ++i) {
            const int e = tid + i * kThreads, row = e / 4, kk = (e % 4) * 4;
            ws[buffer][kk][row] = lw[i].x;
            ws[buffer][kk + 1][row] = lw[i].y;
            ws[buffer][kk + 2][row] = lw[i].z;
            ws[buffer][kk + 3][row] = lw[i].w;
        }
    };
    fetch(0);
    stash(0);
    __syncthreads();
    int buffer = 0;
    for (int k0 = 0; k0 < p.k; k0 += BK, buffer ^= 1) {
        const bool more = k0 + BK < p.k;
        if (more) {
            fetch(k0 + BK);
        }
        ulonglong2 wf[kBufs][RN / 4];
        float4 af[kBufs][RM / 4];
        auto pick = [&](int which, int kk) {
#pragma unroll
            for (int j = 0; j < RN / 4; ++j) {
                wf[which][j] = *reinterpret_cast<const ulonglong2*>(&ws[buffer][kk][j * (BN / (RN / 4)) + tx * 4]);
            }
#pragma unroll
            for (int i4 = 0; i4 < RM / 4; ++i4) {
                af[which][i4] = *reinterpret_cast<const float4*>(&as[buffer][kk][i4 * (BM / (RM / 4)) + ty * 4]);
            }
        };
#pragma unroll
        for (int kk = 0; kk < AHEAD; ++kk) {
            pick(kk, kk);
        }
#pragma unroll
        for (int kk = 0; kk < BK; ++kk) {
            const int now = kk % kBufs;
            if (kk + AHEAD < BK) {
                pick((kk + AHEAD) % kBufs, kk + AHEAD);
            }
#pragma unroll
            for (int i4 = 0; i4 < RM / 4; ++i4) {
                const float4 av = af[now][i4];
                const float a4[4] = {av.x, av.y, av.z, av.w};
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const uint64_t a2 = twice(a4[i]);
#pragma unroll
                    for (int j = 0; j < RN / 4; ++j) {
                        fma2(acc[i4 * 4 + i][2 * j], a2, wf[now][j].x);
                        fma2(acc[i4 * 4 + i][2 * j + 1], a2, wf[now][j].y);
                    }
                }
            }
        }
        if (more) {
            stash(buffer ^ 1);  // (last read a round ago; the round's barrier came since)
        }
        __syncthreads();
    }
    const bool vec = (p.ldc & 3) == 0 && (reinterpret_cast<uintptr_t>(p.c) & 15) == 0;
#pragma unroll
    for (int i = 0; i < RM; ++i) {
        const int row = m0 + (i / 4) * (BM / (RM / 4)) + ty * 4 + i % 4;
        if (row >= p.m) {
            continue;
        }
#pragma unroll
        for (int run = 0; run < RN / 4; ++run) {
            const int col = n0 + run * (BN / (RN / 4)) + tx * 4;
            float v[4];
            asm("mov.b64 {%0, %1}, %2;" : "=f"(v[0]), "=f"(v[1]) : "l"(acc[i][2 * run]));
            asm("mov.b64 {%0, %1}, %2;" : "=f"(v[2]), "=f"(v[3]) : "l"(acc[i][2 * run + 1]));
            if (vec && col + 3 < p.n) {
                float4* dst = reinterpret_cast<float4*>(p.c + static_cast<int64_t>(row) * p.ldc + col);
                float4 r = make_float4(v[0], v[1], v[2], v[3]);
                if (p.accumulate) {
                    const float4 old = *dst;
                    r = make_float4(old.x + r.x, old.y + r.y, old.z + r.z, old.w + r.w);
                }
                *dst = r;
            } else {
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    put(p, row, col + j, v[j]);
                }
            }
        }
    }
}

template <int BM, int BN, int RM, int RN, int AHEAD, int CTAS>
cudaError_t launch_tile(const GemmF32Params& p, cudaStream_t stream) {
    constexpr int kSmem = 2 * 16 * (BM + 4 + BN + 4) * static_cast<int>(sizeof(float));
    static_assert(kSmem <= 48 * 1024, "needs no opt-in");
    gemm_f32_tile_kernel<BM, BN, RM, RN, AHEAD, CTAS>
        <<<dim3((p.m + BM - 1) / BM, (p.n + BN - 1) / BN), BM * BN / (RM * RN), kSmem, stream>>>(p);
    return cudaGetLastError();
}

// ---------------------------------------------------------------------------- rows along k
// LN * CN weight rows and TM * RM rows of A a CTA, CN x RM of them a thread (weight rows LN apart, so that neighbours
// of a warp read neighbouring ones). Both operands arrive by cp.async as they lie, `stages` pieces of BK k in flight, and
// are read four k a load, AHEAD loads before their fmafs: no transposed copy, no registers held for it. What bounds it:
// the weights' stream where N is large and rows are few; shared memory's four bytes a lane and cycle (CN + RM operands
// for CN * RM fmafs) where rows are many; the chain of K dependent fmafs where a CTA is alone on its SM. So tiles grow
// with the rows, and with the columns once the SMs are full (form_for below). 16384 x 2048 and 8 / 16 / 32 / 300 rows:
// 40 / 50 / 76 / 488 us; with one weight row a thread and, above, 64 x 64 tiles through registers 51 / 90 / 130 / 589.
template <int LN, int CN, int TM, int RM, int BK, int AHEAD, int CTAS>
__global__ void __launch_bounds__(LN * TM, CTAS) gemm_f32_rows_kernel(const GemmF32Params p, const int stages) {
    constexpr int BN = LN * CN, BM = TM * RM;
    constexpr int kThreads = LN * TM;
    constexpr int kLd = BK + 4;  // (rows 4 banks apart: eight rows' 16-byte reads meet no bank twice)
    constexpr int kStageFloats = (BN + BM) * kLd;
    constexpr int kLanes = BK / 4, kRows = kThreads / kLanes;  // threads that copy a row's piece, rows copied at a time
    static_assert(kThreads % kLanes == 0 && BK / 4 > AHEAD, "tile");
    extern __shared__ __align__(16) float rows_smem[];
    const int tid = threadIdx.x;
    const int col = tid % LN, tm = tid / LN;
    const int n0 = blockIdx.x * BN, m0 = blockIdx.y * BM;
    const int pieces = (p.k + BK - 1) / BK;

    const int load_row = tid / kLanes, load_k = (tid % kLanes) * 4;
    auto load = [&](int piece, int slot) {
        const int gk = piece * BK + load_k;
        const int bytes = max(0, min(4, p.k - gk)) * 4;
        const int from = bytes > 0 ? gk : 0;  // (past k nothing is read, nor rows of A past the last; weight rows past
                                              // the last read it, and put() drops what comes of them)
        const uint32_t dst = static_cast<uint32_t>(
            __cvta_generic_to_shared(rows_smem + slot * kStageFloats + load_row * kLd + load_k));
        auto copy = [&](int i, const float* src, int bytes) {
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(
                             dst + i * kLd * static_cast<int>(sizeof(float))),
                         "l"(src + from), "r"(bytes)
                         : "memory");
        };
#pragma unroll
        for (int i = 0; i < BN; i += kRows) {
            if (BN % kRows == 0 || i + load_row < BN) {
                copy(i, p.w + static_cast<int64_t>(min(n0 + i + load_row, p.n - 1)) * p.ldw, bytes);
            }
        }
#pragma unroll
        for (int i = 0; i < BM; i += kRows) {
            if (BM % kRows == 0 || i + load_row < BM) {
                const int row = m0 + i + load_row;
                copy(BN + i, p.a + static_cast<int64_t>(min(row, p.m - 1)) * p.lda, row < p.m ? bytes : 0);
            }
        }
    };
    for (int s = 0; s < stages - 1; ++s) {
        if (s < pieces) {
            load(s, s);
        }
        cp_async_commit();
    }
    float acc[RM][CN];
#pragma unroll
    for (int i = 0; i < RM; ++i) {
#pragma unroll
        for (int j = 0; j < CN; ++j) {
            acc[i][j] = 0.0f;
        }
    }
    int slot = 0, next_slot = stages - 1;
    for (int piece = 0; piece < pieces; ++piece) {
        // The group of this piece is the oldest of stages - 1 in flight.
        if (stages == 8) {
            cp_async_wait<6>();
        } else if (stages == 6) {
            cp_async_wait<4>();
        } else if (stages == 4) {
            cp_async_wait<2>();
        } else {
            cp_async_wait<1>();
        }
        __syncthreads();
        if (piece + stages - 1 < pieces) {
            load(piece + stages - 1, next_slot);  // (into the stage that was read before the barrier)
        }
        cp_async_commit();
        next_slot = next_slot + 1 == stages ? 0 : next_slot + 1;
        const float* stage = rows_smem + slot * kStageFloats;
        slot = slot + 1 == stages ? 0 : slot + 1;
        const float* w_at = stage + col * kLd;
        const float* a_at = stage + (BN + tm * RM) * kLd;
        float4 w[AHEAD + 1][CN], a[AHEAD + 1][RM];
        auto fetch = [&](int which, int group) {
#pragma unroll
            for (int j = 0; j < CN; ++j) {
                w[which][j] = *reinterpret_cast<const float4*>(w_at + j * LN * kLd + group * 4);
            }
#pragma unroll
            for (int i = 0; i < RM; ++i) {
                a[which][i] = *reinterpret_cast<const float4*>(a_at + i * kLd + group * 4);
            }
        };
#pragma unroll
        for (int group = 0; group < AHEAD; ++group) {
            fetch(group, group);
        }
#pragma unroll
        for (int group = 0; group < BK / 4; ++group) {
            const int now = group % (AHEAD + 1);
            if (group + AHEAD < BK / 4) {
                fetch((group + AHEAD) % (AHEAD + 1), group + AHEAD);
            }
#pragma unroll
            for (int i = 0; i < RM; ++i) {
#pragma unroll
                for (int j = 0; j < CN; ++j) {
                    acc[i][j] = fmaf(a[now][i].x, w[now][j].x, acc[i][j]);
                }
            }
#pragma unroll
            for (int i = 0; i < RM; ++i) {
#pragma unroll
                for (int j = 0; j < CN; ++j) {
                    acc[i][j] = fmaf(a[now][i].y, w[now][j].y, acc[i][j]);
                }
            }
#pragma unroll
            for (int i = 0; i < RM; ++i) {
#pragma unroll
                for (int j = 0; j < CN; ++j) {
                    acc[i][j] = fmaf(a[now][i].z, w[now][j].z, acc[i][j]);
                }
            }
#pragma unroll
            for (int i = 0; i < RM; ++i) {
#pragma unroll
                for (int j = 0; j < CN; ++j) {
                    acc[i][j] = fmaf(a[now][i].w, w[now][j].w, acc[i][j]);
                }
            }
        }
    }
#pragma unroll
    for (int i = 0; i < RM; ++i) {
#pragma unroll
        for (int j = 0; j < CN; ++j) {
            put(p, m0 + tm * RM + i, n0 + col + j * LN, acc[i][j]);
        }
    }
}

// A CTA alone on its SM keeps ALONE pieces in flight, one among others SHARED.
template <int LN, int CN, int TM, int RM, int BK, int AHEAD, int ALONE, int SHARED, int CTAS = 1>
cudaError_t launch_rows(const GemmF32Params& p, cudaStream_t stream) {
    constexpr int BN = LN * CN, BM = TM * RM;
    constexpr int kStage = (BN + BM) * (BK + 4) * static_cast<int>(sizeof(float));
    static_assert(ALONE * kStage <= 227 * 1024 && SHARED <= ALONE, "stages");
    const dim3 grid((p.n + BN - 1) / BN, (p.m + BM - 1) / BM);
    const int stages = static_cast<int64_t>(grid.x) * grid.y <= 148 ? ALONE : SHARED;
    const cudaError_t set = pl_allow_smem<gemm_f32_rows_kernel<LN, CN, TM, RM, BK, AHEAD, CTAS>>(ALONE * kStage);
    if (set != cudaSuccess) {
        return set;
    }
    gemm_f32_rows_kernel<LN, CN, TM, RM, BK, AHEAD, CTAS><<<grid, LN * TM, stages * kStage, stream>>>(p, stages);
    return cudaGetLastError();
}

// ---------------------------------------------------------------------------- which form
// A form's tile, the k of one of its pieces, how many tiles of rows it is for (0: any), how many of its CTAs an SM holds, the time of a CTA
// alone on its SM and what each further one adds, in ps a k. Measured with weights that are not in L2, 2048 to 32000 columns of 2048 to
// 8192 k. k counts in whole pieces. What is chosen decides time alone. Tiles of up to 16 rows are for one of them, more would read
// the weights again; the 8-row form is also for two, which read them from L2 (16 rows, 3072 x 8192: 87 us by 16-row tiles, 72 so). The
// last 64-row form goes through registers in pieces of 16 k: for k up to 64 alone (200 rows, 3072 x 16: 3.7 us, by 32 x 32 tiles 7.4; at
// 2048 k a third slower than the one along k).
// Picked form / those before the table (us): 8 rows, 12288 x 2048: 32 / 47; 16 rows, 8192 x 2048: 33 / 59; 32 rows, 6144 x 4096: 90 /
// 119; 64 rows, 4096 x 2048: 47 / 69; 128 rows, 3072 x 2048: 76 / 99; 200 rows, 2048 x 8192: 301 / 389; 300 rows, 32000 x 2048: 904 /
// 1065; 700 rows, 4096 x 2048: 281 / 312. Within 5 % of even: up to 4 rows of 4096 columns and fewer, 509 rows of 16384 and 32000.
struct Form {
    int rows, columns, piece, row_tiles, resident, alone, more;
    cudaError_t (*launch)(const GemmF32Params&, cudaStream_t);
};
const Form kForms[] = {
    {1, 32, 128, 1, 3, 5700, 2900, launch_rows<32, 1, 1, 1, 128, 4, 4, 4>},
    {2, 16, 128, 1, 2, 4060, 1500, launch_rows<16, 1, 2, 1, 128, 4, 8, 8>},
    {2, 32, 128, 1, 3, 5700, 2900, launch_rows<32, 1, 1, 2, 128, 4, 4, 4>},
    {4, 16, 128, 1, 5, 4030, 1600, launch_rows<16, 1, 4, 1, 128, 4, 8, 4>},
    {4, 32, 64, 1, 5, 9000, 2500, launch_rows<16, 2, 2, 2, 64, 2, 4, 4>},
    {8, 16, 128, 1, 4, 4800, 3300, launch_rows<16, 1, 4, 2, 128, 4, 8, 4>},
    {8, 16, 128, 2, 4, 5400, 1750, launch_rows<16, 1, 4, 2, 128, 4, 8, 4>},
    {8, 32, 64, 1, 5, 9100, 3500, launch_rows<16, 2, 4, 2, 64, 2, 4, 4>},
    {16, 16, 128, 1, 3, 6800, 6300, launch_rows<16, 1, 8, 2, 128, 4, 8, 4>},
    {16, 32, 64, 1, 2, 10500, 7500, launch_rows<16, 2, 8, 2, 64, 2, 8, 8>},
    {16, 32, 64, 1, 4, 13100, 4000, launch_rows<16, 2, 4, 4, 64, 2, 4, 4>},
    {16, 64, 64, 1, 2, 20100, 4200, launch_rows<16, 4, 4, 4, 64, 1, 4, 4>},
    {32, 16, 128, 0, 2, 9800, 8300, launch_rows<16, 1, 8, 4, 128, 2, 4, 4>},
    {32, 32, 128, 0, 1, 14000, 14000, launch_rows<16, 2, 8, 4, 128, 1, 4, 4>},
    {32, 32, 64, 0, 3, 15100, 9500, launch_rows<16, 2, 8, 4, 64, 2, 4, 4>},
    {32, 64, 64, 0, 2, 23000, 15600, launch_rows<16, 4, 8, 4, 64, 1, 4, 4>},
    {32, 64, 32, 0, 2, 36600, 400, launch_rows<16, 4, 4, 8, 32, 1, 6, 6>},
    {64, 64, 32, 0, 4, 37000, 24300, launch_rows<16, 4, 8, 8, 32, 1, 3, 3, 2>},
    {64, 64, 16, 0, 4, 37000, 24300, launch_tile<64, 64, 4, 8, 1, 4>},
    {128, 64, 16, 0, 3, 62500, 39000, launch_tile<128, 64, 8, 8, 1, 3>},
    {128, 128, 16, 0, 2, 106000, 66000, launch_tile<128, 128, 8, 16, 2, 2>},
};

const Form& form_for(int m, int n, int k) {
    const Form* best = nullptr;
    double least = 0.0;
    for (const Form& f : kForms) {
        const int64_t row_tiles = (m + f.rows - 1) / f.rows, column_tiles = (static_cast<int64_t>(n) + f.columns - 1) / f.columns;
        // The second coordinate of a grid ends at 65,535: the rows' tiles in the forms along k, the columns' in those through
        // registers (pieces of 16). Tiles of 32 columns and more are for products that fill more than half of their rows,
        // those of 64 and 128 rows for more than 16.
        const bool along = f.piece > 16, shortest = !along && f.rows == 64;
        if ((along ? row_tiles : column_tiles) > 65535 || (f.row_tiles != 0 && row_tiles != f.row_tiles) ||
            (f.columns > 16 && f.rows <= 32 && f.rows >= 2 * m) || (f.rows > 32 && m <= 16) || (shortest && k > 64)) {
            continue;
        }
        const int64_t per_sm = (row_tiles * column_tiles + 147) / 148;
        auto together = [&](int64_t ctas) { return ctas > 0 ? f.alone + (ctas - 1) * f.more : 0; };
        const int64_t k_whole = (static_cast<int64_t>(k) + f.piece - 1) / f.piece * f.piece;
        const double time = static_cast<double>(per_sm / f.resident * together(f.resident) + together(per_sm % f.resident)) * k_whole;
        if (best == nullptr || time < least) {
            best = &f;
            least = time;
        }
    }
    return *best;  // (64-row tiles along k take any m from 17 on, 16-row and 8-row ones any below)
}

}  // namespace

PL_API int pl_gemm_f32(const float* a, const float* w, float* c, int m, int n, int k, int lda, int ldw, int ldc,
                       int accumulate, cudaStream_t stream) {
    PL_REQUIRE(m >= 0 && n > 0 && k > 0, "gemm_f32: bad sizes m=%d n=%d k=%d", m, n, k);
    PL_REQUIRE(lda >= k && ldw >= k && ldc >= n, "gemm_f32: leading dimensions too small (lda=%d ldw=%d ldc=%d)", lda,
               ldw, ldc);
    if (m == 0) {
        return 0;
    }
    PL_REQUIRE((m + kTileM - 1) / kTileM <= 65535, "gemm_f32: m=%d is too large for one launch", m);
    const GemmF32Params p{a, w, c, m, n, k, lda, ldw, ldc, accumulate};
    const bool rows16 = (lda & 3) == 0 && (ldw & 3) == 0 &&
        ((reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(w)) & 15) == 0;
    if (!rows16) {
        const dim3 grid((n + kTileN - 1) / kTileN, (m + kTileM - 1) / kTileM);
        gemm_f32_any_kernel<<<grid, 256, 0, stream>>>(p);
        PL_CHECK_LAUNCH("gemm_f32");
        return 0;
    }
    const cudaError_t err = form_for(m, n, k).launch(p, stream);
    if (err != cudaSuccess) {
        return pl_fail(3, "gemm_f32: launch failed: %s", cudaGetErrorString(err));
    }
    return 0;
}
