// Delta rules in steps of single tokens, bfloat16 engine: what the two
// recurrent mixers (gated_delta.cu, delta_rule.cu) share. A CTA has a whole head of one entry: its state [DIM, VDIM]
// lies in the threads' registers (four neighbouring columns, DIM * VDIM / 1024 rows each), so it is read once with 16-byte
// loads and written once, and the head's norm, its weight and the gate follow in the same kernel. What bounds it is the
// state's stream: 64 entries of 32 heads of 64 x 64 are 67 MB. The forms for longer portions give a head to several CTAs
// (that is what one entry's few heads need) which all make the token's vectors anew and leave the norm to a second kernel.
#pragma once

#include "common.cuh"

namespace {

constexpr int kStepThreads = 256;
// CTAs an SM holds: a CTA's loads answer once, so the state's stream is as wide as the CTAs in flight. Heads of 1,024 to 4,096 values
// (without the least) have two builds: with the registers that the compiler takes (48 to 69 a thread: four CTAs an SM, three of 128 x
// 32, five of 32 x 64), and with 40, a few of them in memory, and six. The latter takes 2 to 26 % longer for a CTA and is for steps that then go in
// fewer rounds; the general rule, whose rows need more, for those with a good third fewer. us, four and six CTAs: 32 heads of 64 x 64, 16
// entries 8.3 and 9.7, 24 entries 12.4 and 10.6, 32 entries 13.6 and 14.7, 64 entries 23.2 and 22.5, 256 entries 77.8 and 68.6 (the
// general rule 9.0 and 11.0, 13.6 and 11.9, 14.9 and 17.4, 26.4 and 27.1, 89.6 and 85.5); 16 heads of 128 x 32, 24 entries 7.7 and 9.1,
// 32 entries 11.7 and 9.9; 64 heads of 32 x 128, 16 entries 13.4 and 14.9, 256 entries 144 and 124. 128 x 128 is told of the two that it
// has anyway: 128 registers for 126, 64 entries of 16 heads 33.6 and 32.8. Others as the compiler has them (64 x 128 held to
// three: 36.0 and 37.3).
constexpr int kStepMany = 6;
constexpr bool step_has_two_builds(int dim, int vdim) { return dim * vdim > 1024 && dim * vdim <= 4096; }
// (0: nothing asked; asked for one the compiler takes 88 to 115 registers)
constexpr int step_ctas(int dim, int vdim) { return dim * vdim == 128 * 128 ? 2 : 0; }
inline bool step_many(int64_t ctas, int dim, int vdim, bool general) {
    const int few = dim == 128 ? 3 : dim == 32 && vdim == 64 ? 5 : 4;
    const int64_t rounds = (ctas + few * 148 - 1) / (few * 148), fewer = (ctas + kStepMany * 148 - 1) / (kStepMany * 148);
    return general ? 5 * rounds >= 7 * fewer : rounds > fewer;
}

// A token's vectors of a head, made by the first DIM threads, and its scalars.
template <int DIM, int VDIM>
struct DeltaStepShared {
    float q[DIM];            // meets the new state
    float x[DIM];            // meets the old one
    float g[DIM];            // decays it
    float p[DIM], k[DIM];    // (general rule: removed, written)
    float v[VDIM];
    float sums[kStepThreads / 32][VDIM];
    float b;                 // (last: everything before it starts on 16 bytes)
};

// parts[c] over all row groups for this thread's columns, in every thread.
template <int DIM, int VDIM>
__device__ __forceinline__ float4 step_column_sums(DeltaStepShared<DIM, VDIM>& s, float4 part) {
    constexpr int kQuads = VDIM / 4;
#pragma unroll
    for (int offset = 16; offset >= kQuads; offset >>= 1) {
        part.x += __shfl_xor_sync(0xffffffffu, part.x, offset);
        part.y += __shfl_xor_sync(0xffffffffu, part.y, offset);
        part.z += __shfl_xor_sync(0xffffffffu, part.z, offset);
        part.w += __shfl_xor_sync(0xffffffffu, part.w, offset);
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, quad = threadIdx.x % kQuads;
    if (lane < kQuads) {
        *reinterpret_cast<float4*>(&s.sums[warp][quad * 4]) = part;
    }
    __syncthreads();
    float4 total = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll
    for (int w = 0; w < kStepThreads / 32; ++w) {
        const float4 v = *reinterpret_cast<const float4*>(&s.sums[w][quad * 4]);
        total.x += v.x;
        total.y += v.y;
        total.z += v.z;
        total.w += v.w;
    }
    __syncthreads();
    return total;
}

// Walks `count` tokens of one entry and head; VECTORS(t) fills s.q .. s.b of token t (all threads call it; what it wrote
// is read after a barrier here); OUT(t, column, value, factor) takes the four outputs of a thread of the first row group.
template <int DIM, int VDIM, bool GENERAL, typename Vectors, typename Out>
__device__ __forceinline__ void delta_step_walk(DeltaStepShared<DIM, VDIM>& s, float* state, int count, float eps,
                                                const Vectors& vectors, const Out& store) {
    constexpr int kQuads = VDIM / 4, kGroups = kStepThreads / kQuads, kRows = DIM / kGroups;
    static_assert(kRows >= 1 && kRows * kGroups == DIM, "rows of a thread");
    const int quad = threadIdx.x % kQuads, group = threadIdx.x / kQuads;
    float4 S[kRows];
#pragma unroll
    for (int r = 0; r < kRows; ++r) {
        S[r] = *reinterpret_cast<const float4*>(state + (group + r * kGroups) * VDIM + quad * 4);
    }
    for (int t = 0; t < count; ++t) {
        vectors(t);
        __syncthreads();
        float4 part = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll
        for (int r = 0; r < kRows; ++r) {
            const int i = group + r * kGroups;
            const float x = s.x[i];
            if constexpr (!GENERAL) {
                const float g = s.g[i];
                S[r] = make_float4(S[r].x * g, S[r].y * g, S[r].z * g, S[r].w * g);
            }
            part = make_float4(fmaf(S[r].x, x, part.x), fmaf(S[r].y, x, part.y), fmaf(S[r].z, x, part.z), fmaf(S[r].w, x, part.w));
        }
        const float4 dot = step_column_sums<DIM, VDIM>(s, part);
        const float4 v = *reinterpret_cast<const float4*>(&s.v[quad * 4]);
        const float b = s.b;
        const float4 u = make_float4(b * (v.x - dot.x), b * (v.y - dot.y), b * (v.z - dot.z), b * (v.w - dot.w));
        part = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll
        for (int r = 0; r < kRows; ++r) {
            const int i = group + r * kGroups;
            if constexpr (GENERAL) {
                const float g = s.g[i], p = -s.p[i], k = s.k[i];
                S[r] = make_float4(fmaf(k, v.x, fmaf(p, dot.x, g * S[r].x)), fmaf(k, v.y, fmaf(p, dot.y, g * S[r].y)),
                                   fmaf(k, v.z, fmaf(p, dot.z, g * S[r].z)), fmaf(k, v.w, fmaf(p, dot.w, g * S[r].w)));
            } else {
                const float x = s.x[i];
                S[r] = make_float4(fmaf(x, u.x, S[r].x), fmaf(x, u.y, S[r].y), fmaf(x, u.z, S[r].z), fmaf(x, u.w, S[r].w));
            }
            const float q = s.q[i];
            part = make_float4(fmaf(S[r].x, q, part.x), fmaf(S[r].y, q, part.y), fmaf(S[r].z, q, part.z), fmaf(S[r].w, q, part.w));
        }
        const float4 o = step_column_sums<DIM, VDIM>(s, part);
        // the head's norm: the first row group's lanes hold every column once
        float square = fmaf(o.x, o.x, fmaf(o.y, o.y, fmaf(o.z, o.z, o.w * o.w)));
#pragma unroll
        for (int offset = kQuads / 2; offset > 0; offset >>= 1) {
            square += __shfl_xor_sync(0xffffffffu, square, offset);
        }
        if (group == 0) {
            const float factor = 1.0f / sqrtf(square / static_cast<float>(VDIM) + eps);
            store(t, quad * 4, make_float4(o.x * factor, o.y * factor, o.z * factor, o.w * factor));
        }
    }
#pragma unroll
    for (int r = 0; r < kRows; ++r) {
        *reinterpret_cast<float4*>(state + (group + r * kGroups) * VDIM + quad * 4) = S[r];
    }
}

// The sums over the first DIM threads of two values each, in all of them (and nothing of use in the others).
template <int DIM, int VDIM>
__device__ __forceinline__ float2 step_vector_sums(DeltaStepShared<DIM, VDIM>& s, float a, float b) {
    const int warp = threadIdx.x >> 5;
    a = pl_warp_sum(a);
    b = pl_warp_sum(b);
    if ((threadIdx.x & 31) == 0 && warp < DIM / 32) {
        s.sums[0][2 * warp] = a;
        s.sums[0][2 * warp + 1] = b;
    }
    __syncthreads();
    a = b = 0.0f;
#pragma unroll
    for (int w = 0; w < DIM / 32; ++w) {
        a += s.sums[0][2 * w];
        b += s.sums[0][2 * w + 1];
    }
    return make_float2(a, b);
}

}  // namespace
