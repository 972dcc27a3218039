// Paged causal attention on CUDA cores: the float32 engine's attention, and the
// kernel that takes every head size, group size and page size in bfloat16 too.
//
// A warp walks the keys of a (query token, query head) pair's request
// in chunks of 32 in ascending order, one key per lane for the scores, then
// accumulates the chunk's values with lane d owning output dims d, d+32, ... . The plain
// kernel gives a warp one pair at a time and reads keys and values from memory; float32 has a form with
// the chunks staged in shared memory for several pairs (below), the same sums in the same order.
// Scores, softmax and accumulation are fp32 (expf, not the fast intrinsic). The
// walk depends only on the query's position (and the window), so a query's result
// is the same whatever else is in the batch and however the prompt was cut.
// Prefill chunks and decode tokens are the same to it: every token carries its
// position and its request's block-table row. The reference's counterpart is
// attn_scalar_kernel, pulsarlm-core/src/kernels/paged_common.cu:26-137.
#include "common.cuh"

#include "mma_helpers.cuh"

namespace {

constexpr int kMaxAcc = 16;      // head_dim <= 512
constexpr int kMaxAccWide = 32;  // head_dim <= 1024

template <typename scalar_t>
__device__ __forceinline__ float dot_row(const float* __restrict__ q, const scalar_t* __restrict__ k, int head_dim);

template <>
__device__ __forceinline__ float dot_row<float>(const float* __restrict__ q, const float* __restrict__ k,
                                                int head_dim) {
    float s = 0.0f;
    if ((head_dim & 3) == 0 && (reinterpret_cast<uintptr_t>(k) & 15) == 0) {
        const float4* k4 = reinterpret_cast<const float4*>(k);
        for (int d = 0; d < head_dim / 4; ++d) {
            const float4 kv = k4[d];
            s = fmaf(q[4 * d + 0], kv.x, s);
            s = fmaf(q[4 * d + 1], kv.y, s);
            s = fmaf(q[4 * d + 2], kv.z, s);
            s = fmaf(q[4 * d + 3], kv.w, s);
        }
    } else {
        for (int d = 0; d < head_dim; ++d) {
            s = fmaf(q[d], k[d], s);
        }
    }
    return s;
}

template <>
__device__ __forceinline__ float dot_row<__nv_bfloat16>(const float* __restrict__ q,
                                                        const __nv_bfloat16* __restrict__ k, int head_dim) {
    float s = 0.0f;
    if ((head_dim & 7) == 0 && (reinterpret_cast<uintptr_t>(k) & 15) == 0) {
        const uint4* k8 = reinterpret_cast<const uint4*>(k);
        for (int d = 0; d < head_dim / 8; ++d) {
            const uint4 raw = k8[d];
            const uint32_t words[4] = {raw.x, raw.y, raw.z, raw.w};
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                // bf16 -> fp32 is a 16-bit shift of the bit pattern.
                s = fmaf(q[8 * d + 2 * i], __uint_as_float(words[i] << 16), s);
                s = fmaf(q[8 * d + 2 * i + 1], __uint_as_float(words[i] & 0xffff0000u), s);
            }
        }
    } else {
        for (int d = 0; d < head_dim; ++d) {
            s = fmaf(q[d], __bfloat162float(k[d]), s);
        }
    }
    return s;
}

template <typename scalar_t, int ACC>
__global__ void attention_simt_kernel(const scalar_t* __restrict__ q, int64_t q_row_stride,
                                      const scalar_t* __restrict__ k_pool, const scalar_t* __restrict__ v_pool,
                                      int64_t page_stride, int64_t head_stride, int page_size, int n_pages,
                                      const int32_t* __restrict__ table, int table_width,
                                      const int32_t* __restrict__ pos, const int32_t* __restrict__ entry,
                                      scalar_t* __restrict__ out, int64_t out_row_stride, int n_heads, int group,
                                      int head_dim, int window, float scale, float softcap,
                                      float* __restrict__ mass_sum, float* __restrict__ weight_sum,
                                      const float* __restrict__ query_weights, const float* __restrict__ sinks,
                                      const scalar_t* __restrict__ gate, int64_t gate_row_stride,
                                      const float* __restrict__ distance_bias, int bias_rows,
                                      const float* __restrict__ distance_slopes, int keep_first, int32_t* status) {
    extern __shared__ float q_shared[];  // [warps][head_dim]
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
    const int t = blockIdx.x;
    const int kv_head = blockIdx.y;
    const int p = pos[t];
    const int first = window > 0 ? max(0, p - window + 1) : 0;
    const PlTileWalk walk(first, keep_first, 32);
    const int chunks = walk.count(p, 32);
    const int32_t* row = table + static_cast<int64_t>(entry[t]) * table_width;
    float* qs = q_shared + warp * head_dim;
    const int n_acc = (head_dim + 31) / 32;

    for (int hg = warp; hg < group; hg += warps) {
        const int h = kv_head * group + hg;
        const scalar_t* qrow = q + t * q_row_stride + static_cast<int64_t>(h) * head_dim;
        __syncwarp();
        for (int d = lane; d < head_dim; d += 32) {
            qs[d] = pl_load(qrow + d);
        }
        __syncwarp();

        float m = -INFINITY, l = 0.0f;
        float acc[ACC];
#pragma unroll
        for (int i = 0; i < ACC; ++i) {
            acc[i] = 0.0f;
        }
        // Attention mass (optional): per page and head, this query's weight times its
        // largest scaled score over the page's keys it attends; per page, the weight once.
        int mass_page = -1;
        float mass_max = -INFINITY;
        auto add_mass = [&](int view_page, float page_max) {
            if (view_page < 0 || lane != 0 || !(page_max > -INFINITY)) {
                return;
            }
            const int page = row[view_page];
            if (page >= 0 && page < n_pages) {
                const float w = query_weights != nullptr ? query_weights[t] : 1.0f;
                atomicAdd(mass_sum + static_cast<int64_t>(page) * n_heads + h, w * page_max);
                if (h == 0) {
                    atomicAdd(weight_sum + page, w);
                }
            }
        };

        for (int w = 0; w < chunks; ++w) {
            const int base = walk.tile(w) * 32;
            const int j = base + lane;
            const bool valid = (j >= first || j < keep_first) && j <= p;
            int64_t offset = -1;
            float s = -INFINITY;
            if (valid) {
                const int page = row[j / page_size];
                if (page >= 0 && page < n_pages) {
                    offset = page * page_stride + kv_head * head_stride +
                        static_cast<int64_t>(j % page_size) * head_dim;
                    s = dot_row<scalar_t>(qs, k_pool + offset, head_dim) * scale;
                    if (softcap > 0.0f) {
                        s = softcap * tanhf(s / softcap);  // scores squashed into (-cap, cap) before the softmax
                    }
                    if (distance_bias != nullptr) {
                        // a learned bias by distance and head joins the scaled score (the scale does not touch it)
                        s += distance_bias[static_cast<int64_t>(h) * bias_rows + min(p - j, bias_rows - 1)];
                    }
                    if (distance_slopes != nullptr) {
                        s = fmaf(-distance_slopes[h], static_cast<float>(p - j), s);
                    }
                } else if (status != nullptr) {
                    atomicOr(status, 4);
                }
            }
            if (mass_sum != nullptr) {
                // Largest scaled score per page; a page may span several chunks, so the
                // running maximum is flushed only when the walk leaves the page.
                const int last = min(base + 31, p);
                for (int pg = (base < keep_first ? base : max(base, first)) / page_size; pg <= last / page_size; ++pg) {
                    const float chunk_max = pl_warp_max(valid && j / page_size == pg ? s : -INFINITY);
                    if (pg != mass_page) {
                        add_mass(mass_page, mass_max);
                        mass_page = pg;
                        mass_max = chunk_max;
                    } else {
                        mass_max = fmaxf(mass_max, chunk_max);
                    }
                }
            }
            const float m_new = fmaxf(m, pl_warp_max(s));
            // m_new is -inf only if a bad block table hid every key so far.
            const bool seen = m_new > -INFINITY;
            const float corr = seen ? expf(m - m_new) : 1.0f;  // 0 on the first chunk (m = -inf)
            const float pw = offset >= 0 && seen ? expf(s - m_new) : 0.0f;
            l = l * corr + pl_warp_sum(pw);
#pragma unroll
            for (int i = 0; i < ACC; ++i) {
                if (i < n_acc) {
                    acc[i] *= corr;
                }
            }
            const int count = min(32, p - base + 1);
            for (int jj = 0; jj < count; ++jj) {
                const float pj = __shfl_sync(0xffffffffu, pw, jj);
                const int64_t oj = __shfl_sync(0xffffffffu, offset, jj);
                if (oj < 0) {
                    continue;
                }
                const scalar_t* vrow = v_pool + oj;
#pragma unroll
                for (int i = 0; i < ACC; ++i) {
                    const int d = lane + 32 * i;
                    if (i < n_acc && d < head_dim) {
                        acc[i] = fmaf(pj, pl_load(vrow + d), acc[i]);
                    }
                }
            }
            m = m_new;
        }

        if (mass_sum != nullptr) {
            add_mass(mass_page, mass_max);
        }
        if (sinks != nullptr) {
            // A sink: one more term exp(sink) in the denominator, with no key and no value.
            const float sink = sinks[h];
            const float m_new = fmaxf(m, sink);
            const float corr = m > -INFINITY ? expf(m - m_new) : 0.0f;
            l = l * corr + expf(sink - m_new);
#pragma unroll
            for (int i = 0; i < ACC; ++i) {
                if (i < n_acc) {
                    acc[i] *= corr;
                }
            }
        }
        float inv = l > 0.0f ? 1.0f / l : 0.0f;
        if (gate != nullptr) {
            // The head's output times sigmoid of its gate logit.
            inv *= 1.0f / (1.0f + expf(-pl_load(gate + t * gate_row_stride + h)));
        }
        scalar_t* orow = out + t * out_row_stride + static_cast<int64_t>(h) * head_dim;
#pragma unroll
        for (int i = 0; i < ACC; ++i) {
            const int d = lane + 32 * i;
            if (i < n_acc && d < head_dim) {
                pl_store(orow + d, acc[i] * inv);
            }
        }
    }
}

// The same walk for the float32 engine with the keys and values of a chunk in shared memory, every sum in the
// order of the kernel above (their results are equal bit for bit). A CTA takes `run` neighbouring tokens of
// one kv head; a warp takes P of their (token, head) pairs, so a key or value read from shared memory serves P
// of them, and chunks arrive by cp.async two ahead. (Neighbours of several requests would be walked one request after
// the other: 65 single tokens of 600 keys took 707 us so, 455 by the kernel above. They have CTAs of one token.) What bounds the kernel above is the time a load takes to answer, once per key; here it is the operands
// that shared memory hands out (1.25 a fmaf of the scores at P = 4), with few CTAs the chain of a chunk's phases. 32
// heads of 64 over 8 kv heads, cold caches: 509 tokens of one prompt 779 -> 164 us, 8 single tokens of 600 keys
// 413 -> 36 us. (With the head size known to the compiler a single token's walk is a quarter shorter; four pairs a
// warp then take 132 registers, one CTA an SM instead of two, 195 us: those keep it a number.)
constexpr int kStagedDim = 128;

// Whether the `run` <= 32 tokens from `first` on are not all there or not all one request's. (By a whole warp.)
__device__ __forceinline__ bool run_is_mixed(const int32_t* entry, int first, int run, int n_tokens) {
    const int t = first + static_cast<int>(threadIdx.x & 31);
    return __any_sync(0xffffffffu, t < first + run && (t >= n_tokens || entry[t] != entry[first]));
}

constexpr int kStagedStages = 3;
constexpr int kOffsetRing = kStagedStages + 1;  // (where a chunk lies is known a step before its copies set out)

struct StagedParams {
    const float* q;
    int64_t q_row_stride;
    const float* k_pool;
    const float* v_pool;
    int64_t page_stride, head_stride;
    int page_size, n_pages;
    const int32_t* table;
    int table_width;
    const int32_t* pos;
    const int32_t* entry;
    float* out;
    int64_t out_row_stride;
    int n_tokens, group, head_dim, window, run;
    int mixed_run;  // 0: every token; else those of the runs of this many that are one request's (run > 1) or are not (run == 1)
    float scale, softcap;
    const float* sinks;
    const float* gate;
    int64_t gate_row_stride;
    const float* distance_bias;
    int bias_rows;
    const float* distance_slopes;
    int keep_first;
    int32_t* status;
};

inline int staged_smem_bytes(int pairs, int head_dim) {
    const int floats = pairs * head_dim + pairs * 32 + kStagedStages * 32 * (2 * head_dim + 4);
    return floats * 4 + kOffsetRing * 32 * 8;
}

template <int P, int ACC, int DIM>
__global__ void attention_f32_staged_kernel(const StagedParams a) {
    extern __shared__ __align__(16) float staged_smem[];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int hd = DIM > 0 ? DIM : a.head_dim, group = a.group;   // (DIM: a head size known to the compiler, or 0)
    const int pairs = a.run * group;
    const int k_ld = hd + 4;                             // (rows 4 banks apart: a lane reads a key of its own)
    float* qs = staged_smem;                             // [pairs][hd]
    float* ps = qs + pairs * hd;                         // [pairs][32]
    float* ks = ps + pairs * 32;                         // [stages][32][hd + 4]
    float* vs = ks + kStagedStages * 32 * k_ld;          // [stages][32][hd]
    int64_t* offsets = reinterpret_cast<int64_t*>(vs + kStagedStages * 32 * hd);  // [stages + 1][32]
    const int kv_head = blockIdx.y;
    // (the last tokens of a prompt have the longest walks: they start first)
    const int t_begin = static_cast<int>(gridDim.x - 1 - blockIdx.x) * a.run;
    const int t_end = min(t_begin + a.run, a.n_tokens);
    if (a.mixed_run > 0 &&
        run_is_mixed(a.entry, t_begin / a.mixed_run * a.mixed_run, a.mixed_run, a.n_tokens) != (a.run == 1)) {
        return;
    }

    for (int idx = tid; idx < (t_end - t_begin) * group * hd; idx += blockDim.x) {
        const int pair = idx / hd, d = idx - pair * hd;
        qs[idx] = a.q[(t_begin + pair / group) * a.q_row_stride + static_cast<int64_t>(kv_head * group + pair % group) * hd + d];
    }

    for (int seg = t_begin; seg < t_end;) {
        const int e = a.entry[seg];
        int seg_end = seg, p_max = -1, first_min = INT_MAX;
        while (seg_end < t_end && a.entry[seg_end] == e) {
            const int p = a.pos[seg_end];
            p_max = max(p_max, p);
            first_min = min(first_min, a.window > 0 ? max(0, p - a.window + 1) : 0);
            ++seg_end;
        }
        const PlTileWalk walk(first_min, a.keep_first, 32);
        const int chunks = walk.count(p_max, 32);
        const int32_t* row = a.table + static_cast<int64_t>(e) * a.table_width;

        // Where the 32 keys of the walk's place w lie (-1: no page, or past the last key), by the first warp; the
        // page is asked for a step before it is needed.
        auto ask = [&](int w) {
            const int j = w < chunks ? walk.tile(w) * 32 + lane : INT_MAX;
            return warp == 0 && j <= p_max ? row[j / a.page_size] : -1;
        };
        auto locate = [&](int w, int page) {
            if (warp == 0 && w < chunks) {
                const int j = walk.tile(w) * 32 + lane;
                offsets[w % kOffsetRing * 32 + lane] = page >= 0 && page < a.n_pages
                    ? page * a.page_stride + kv_head * a.head_stride + static_cast<int64_t>(j % a.page_size) * hd : -1;
            }
        };
        auto load = [&](int w) {
            if (w < chunks) {
                const int64_t* where = offsets + w % kOffsetRing * 32;
                const int stage = w % kStagedStages, per = hd / 4;
                for (int idx = tid; idx < 32 * per; idx += blockDim.x) {
                    const int key = idx / per, c = (idx - key * per) * 4;
                    const int64_t offset = where[key];
                    const bool there = offset >= 0;
                    cp_async_16_or_zero(ks + (stage * 32 + key) * k_ld + c, a.k_pool + (there ? offset + c : 0), there);
                    cp_async_16_or_zero(vs + (stage * 32 + key) * hd + c, a.v_pool + (there ? offset + c : 0), there);
                }
            }
            cp_async_commit();
        };

        int position[P], first[P];
        bool mine[P];
        float m[P], l[P], acc[P][ACC];
#pragma unroll
        for (int i = 0; i < P; ++i) {
            const int pair = warp * P + i;
            const int t = t_begin + pair / group;
            mine[i] = pair < pairs && t >= seg && t < seg_end;
            position[i] = mine[i] ? a.pos[t] : -1;
            first[i] = a.window > 0 ? max(0, position[i] - a.window + 1) : 0;
            m[i] = -INFINITY;
            l[i] = 0.0f;
#pragma unroll
            for (int n = 0; n < ACC; ++n) {
                acc[i][n] = 0.0f;
            }
        }

        __syncthreads();  // (the queries are there; nothing of an earlier request's chunks is read any more)
        locate(0, ask(0));
        locate(1, ask(1));
        locate(2, ask(2));
        int page = ask(3);
        __syncthreads();
        load(0);
        load(1);
        for (int w = 0; w < chunks; ++w) {
            cp_async_wait<1>();
            __syncthreads();  // the chunk has landed, and the one before it was read by everyone
            locate(w + 3, page);
            page = ask(w + 4);
            load(w + 2);
            const int chunk = walk.tile(w), base = chunk * 32, j = base + lane;
            bool takes[P], any = false;
#pragma unroll
            for (int i = 0; i < P; ++i) {
                const PlTileWalk own(first[i], a.keep_first, 32);
                takes[i] = mine[i] && (chunk < own.head || chunk >= own.start) && base <= position[i];
                any = any || takes[i];
            }
            if (!any) {
                continue;
            }
            const int stage = w % kStagedStages;
            const float* krow = ks + (stage * 32 + lane) * k_ld;
            const bool paged = offsets[w % kOffsetRing * 32 + lane] >= 0;
            float s[P];
#pragma unroll
            for (int i = 0; i < P; ++i) {
                s[i] = 0.0f;
            }
#pragma unroll(DIM > 0 ? DIM / 4 : 4)
            for (int d = 0; d < hd; d += 4) {
                const float4 kv = *reinterpret_cast<const float4*>(krow + d);
#pragma unroll
                for (int i = 0; i < P; ++i) {
                    // (a pair past the CTA's last reads another's query: nothing is made of it)
                    const float4 qv = *reinterpret_cast<const float4*>(qs + min(warp * P + i, pairs - 1) * hd + d);
                    s[i] = fmaf(qv.x, kv.x, s[i]);
                    s[i] = fmaf(qv.y, kv.y, s[i]);
                    s[i] = fmaf(qv.z, kv.z, s[i]);
                    s[i] = fmaf(qv.w, kv.w, s[i]);
                }
            }
            uint32_t seen_keys[P];
            bool whole = true;
#pragma unroll
            for (int i = 0; i < P; ++i) {
                const int h = kv_head * group + (warp * P + i) % group;
                const bool reach = takes[i] && (j >= first[i] || j < a.keep_first) && j <= position[i];
                if (reach && !paged && a.status != nullptr) {
                    atomicOr(a.status, 4);
                }
                const bool valid = reach && paged;
                float score = -INFINITY;
                if (valid) {
                    score = s[i] * a.scale;
                    if (a.softcap > 0.0f) {
                        score = a.softcap * tanhf(score / a.softcap);
                    }
                    if (a.distance_bias != nullptr) {
                        score += a.distance_bias[static_cast<int64_t>(h) * a.bias_rows + min(position[i] - j, a.bias_rows - 1)];
                    }
                    if (a.distance_slopes != nullptr) {
                        score = fmaf(-a.distance_slopes[h], static_cast<float>(position[i] - j), score);
                    }
                }
                seen_keys[i] = __ballot_sync(0xffffffffu, valid);
                whole = whole && (!takes[i] || seen_keys[i] == 0xffffffffu);
                float pw = 0.0f;
                if (takes[i]) {
                    const float m_new = fmaxf(m[i], pl_warp_max(score));
                    const bool seen = m_new > -INFINITY;  // (-inf only if a bad block table hid every key so far)
                    const float corr = seen ? expf(m[i] - m_new) : 1.0f;
                    pw = valid && seen ? expf(score - m_new) : 0.0f;
                    l[i] = l[i] * corr + pl_warp_sum(pw);
#pragma unroll
                    for (int n = 0; n < ACC; ++n) {
                        acc[i][n] *= corr;
                    }
                    m[i] = m_new;
                }
                if (warp * P + i < pairs) {
                    ps[(warp * P + i) * 32 + lane] = pw;
                }
            }
            __syncwarp();
            const float* vrows = vs + stage * 32 * hd;
            auto weigh = [&](int jj, const float (&pj)[P], bool check) {
                float v[ACC];
#pragma unroll
                for (int n = 0; n < ACC; ++n) {
                    const int d = lane + 32 * n;
                    v[n] = d < hd ? vrows[jj * hd + d] : 0.0f;
                }
#pragma unroll
                for (int i = 0; i < P; ++i) {
                    if (takes[i] && (!check || (seen_keys[i] >> jj & 1))) {
#pragma unroll
                        for (int n = 0; n < ACC; ++n) {
                            acc[i][n] = fmaf(pj[i], v[n], acc[i][n]);
                        }
                    }
                }
            };
#pragma unroll(P == 1 ? 8 : 2)
            for (int j4 = 0; j4 < 32; j4 += 4) {
                float4 p4[P];
#pragma unroll
                for (int i = 0; i < P; ++i) {
                    p4[i] = *reinterpret_cast<const float4*>(ps + min(warp * P + i, pairs - 1) * 32 + j4);
                }
                float pj[4][P];
#pragma unroll
                for (int i = 0; i < P; ++i) {
                    pj[0][i] = p4[i].x;
                    pj[1][i] = p4[i].y;
                    pj[2][i] = p4[i].z;
                    pj[3][i] = p4[i].w;
                }
                if (whole) {
#pragma unroll
                    for (int n = 0; n < 4; ++n) {
                        weigh(j4 + n, pj[n], false);
                    }
                } else {
#pragma unroll
                    for (int n = 0; n < 4; ++n) {
                        weigh(j4 + n, pj[n], true);
                    }
                }
            }
            __syncwarp();  // (the weights are written anew in the next chunk)
        }
        cp_async_wait<0>();

#pragma unroll
        for (int i = 0; i < P; ++i) {
            if (!mine[i]) {
                continue;
            }
            const int t = t_begin + (warp * P + i) / group, h = kv_head * group + (warp * P + i) % group;
            if (a.sinks != nullptr) {
                const float sink = a.sinks[h];
                const float m_new = fmaxf(m[i], sink);
                const float corr = m[i] > -INFINITY ? expf(m[i] - m_new) : 0.0f;
                l[i] = l[i] * corr + expf(sink - m_new);
#pragma unroll
                for (int n = 0; n < ACC; ++n) {
                    acc[i][n] *= corr;
                }
            }
            float inv = l[i] > 0.0f ? 1.0f / l[i] : 0.0f;
            if (a.gate != nullptr) {
                inv *= 1.0f / (1.0f + expf(-a.gate[t * a.gate_row_stride + h]));
            }
            float* orow = a.out + t * a.out_row_stride + static_cast<int64_t>(h) * hd;
#pragma unroll
            for (int n = 0; n < ACC; ++n) {
                const int d = lane + 32 * n;
                if (d < hd) {
                    orow[d] = acc[i][n] * inv;
                }
            }
        }
        seg = seg_end;
    }
}

// The same walk for few tokens without a window, its parts side by side: a CTA has one token and HEADS heads of a kv head, and
// KEYS keys at a time. A warp's 32 keys are one chunk of the walk: its threads make their keys' scores, then the chunk's largest; what
// the walk's maximum was before and after every chunk follows from those; the weights, their sums and the corrections are made
// chunk by chunk at once, and then a thread walks the keys for one column of one head. Every number is made by the same
// operations in the same order. Left in line is only the chain of fmafs over the keys, four cycles each; the walk above had every
// chunk's phases in it. What bounds it: shared memory's operands (a key and a query a fmaf of the scores, a value and a quarter of a
// weight a fmaf of the outputs). 8 tokens of 600 keys, 32 heads of 64 over 8, cold, in an engine step: 33.5 -> 20.1 us.
constexpr int kWideThreads = 256;

template <int HEADS, int KEYS>
inline constexpr int wide_smem_bytes(int hd) {
    return (HEADS * hd + HEADS * KEYS + 3 * HEADS * (KEYS / 32) + 2 * KEYS * (2 * hd + 4)) * 4 + HEADS * (KEYS / 32) * 4 + 3 * KEYS * 8;
}

template <int HEADS, int KEYS, int ACC>
__global__ void __launch_bounds__(kWideThreads) attention_f32_wide_kernel(const StagedParams a) {
    constexpr int kChunks = KEYS / 32, kSets = kWideThreads / KEYS, kOwn = (HEADS + kSets - 1) / kSets;
    extern __shared__ __align__(16) float wide_smem[];
    const int tid = threadIdx.x, lane = tid & 31;
    const int hd = a.head_dim, k_ld = hd + 4;
    float* ks = wide_smem;                                    // [2][KEYS][hd + 4]
    float* vs = ks + 2 * KEYS * k_ld;                         // [2][KEYS][hd]
    float* qs = vs + 2 * KEYS * hd;                           // [HEADS][hd]
    float* ps = qs + HEADS * hd;                              // [HEADS][KEYS]
    float* largest = ps + HEADS * KEYS;                       // [HEADS][chunks]
    float* sums = largest + HEADS * kChunks;
    float* corrections = sums + HEADS * kChunks;
    uint32_t* seen = reinterpret_cast<uint32_t*>(corrections + HEADS * kChunks);
    int64_t* offsets = reinterpret_cast<int64_t*>(seen + HEADS * kChunks);  // [3][KEYS]
    const int t = blockIdx.x, kv_head = blockIdx.y, head0 = kv_head * a.group + blockIdx.z * HEADS;
    const int position = a.pos[t];
    const int steps = position / KEYS + 1;
    const int32_t* row = a.table + static_cast<int64_t>(a.entry[t]) * a.table_width;

    for (int idx = tid; idx < HEADS * hd; idx += kWideThreads) {
        qs[idx] = a.q[t * a.q_row_stride + static_cast<int64_t>(head0) * hd + idx];
    }
    auto locate = [&](int w) {  // where a step's keys lie (-1: no page, or past the last key)
        const int j = w * KEYS + tid;
        if (tid < KEYS && w < steps) {
            const int page = j <= position ? row[j / a.page_size] : -1;
            offsets[w % 3 * KEYS + tid] = page >= 0 && page < a.n_pages
                ? page * a.page_stride + kv_head * a.head_stride + static_cast<int64_t>(j % a.page_size) * hd : -1;
        }
    };
    auto load = [&](int w) {
        if (w < steps) {
            const int64_t* where = offsets + w % 3 * KEYS;
            const int stage = w & 1, per = hd / 4;
            for (int idx = tid; idx < KEYS * per; idx += kWideThreads) {
                const int key = idx / per, c = (idx - key * per) * 4;
                const int64_t offset = where[key];
                const bool there = offset >= 0;
                cp_async_16_or_zero(ks + (stage * KEYS + key) * k_ld + c, a.k_pool + (there ? offset + c : 0), there);
                cp_async_16_or_zero(vs + (stage * KEYS + key) * hd + c, a.v_pool + (there ? offset + c : 0), there);
            }
        }
        cp_async_commit();
    };
    const int key = tid % KEYS, set = tid / KEYS, chunk = key / 32;  // (this thread's heads: set, set + kSets, ...)
    float m[kOwn], acc[ACC], l[ACC];
#pragma unroll
    for (int i = 0; i < kOwn; ++i) {
        m[i] = -INFINITY;
    }
#pragma unroll
    for (int n = 0; n < ACC; ++n) {
        acc[n] = l[n] = 0.0f;
    }
    locate(0);
    locate(1);
    __syncthreads();
    load(0);
    for (int w = 0; w < steps; ++w) {
        cp_async_wait<0>();
        __syncthreads();  // the step's keys have landed; the one before it was read by everyone
        load(w + 1);
        locate(w + 2);
        const int stage = w & 1, j = w * KEYS + key;
        const bool paged = offsets[w % 3 * KEYS + key] >= 0;
        const float* krow = ks + (stage * KEYS + key) * k_ld;
        float s[kOwn];
#pragma unroll
        for (int i = 0; i < kOwn; ++i) {
            s[i] = 0.0f;
        }
#pragma unroll 4
        for (int d = 0; d < hd; d += 4) {
            const float4 kv = *reinterpret_cast<const float4*>(krow + d);
#pragma unroll
            for (int i = 0; i < kOwn; ++i) {
                const float4 qv = *reinterpret_cast<const float4*>(qs + min(set + i * kSets, HEADS - 1) * hd + d);
                s[i] = fmaf(qv.x, kv.x, s[i]);
                s[i] = fmaf(qv.y, kv.y, s[i]);
                s[i] = fmaf(qv.z, kv.z, s[i]);
                s[i] = fmaf(qv.w, kv.w, s[i]);
            }
        }
        if (j <= position && !paged && set == 0 && a.status != nullptr) {
            atomicOr(a.status, 4);
        }
        const bool valid = j <= position && paged;
#pragma unroll
        for (int i = 0; i < kOwn; ++i) {
            const int h = set + i * kSets;
            float score = -INFINITY;
            if (valid && h < HEADS) {
                score = s[i] * a.scale;
                if (a.softcap > 0.0f) {
                    score = a.softcap * tanhf(score / a.softcap);
                }
                if (a.distance_bias != nullptr) {
                    score += a.distance_bias[static_cast<int64_t>(head0 + h) * a.bias_rows + min(position - j, a.bias_rows - 1)];
                }
                if (a.distance_slopes != nullptr) {
                    score = fmaf(-a.distance_slopes[head0 + h], static_cast<float>(position - j), score);
                }
            }
            s[i] = score;
            const float top = pl_warp_max(score);
            const uint32_t there = __ballot_sync(0xffffffffu, valid);
            if (lane == 0 && h < HEADS) {
                largest[h * kChunks + chunk] = top;
                seen[h * kChunks + chunk] = there;
            }
        }
        __syncthreads();
        // Chunks past the last key are not walked.
        const int chunks = min(kChunks, (position - w * KEYS) / 32 + 1);
#pragma unroll
        for (int i = 0; i < kOwn; ++i) {
            const int h = set + i * kSets;
            float before = m[i], after = m[i], running = m[i];
            for (int c = 0; c < chunks && h < HEADS; ++c) {
                const float next = fmaxf(running, largest[h * kChunks + c]);
                if (c == chunk) {
                    before = running;
                    after = next;
                }
                running = next;
            }
            m[i] = running;
            const bool any = after > -INFINITY;  // (-inf only if a bad block table hid every key so far)
            const float weight = valid && any ? expf(s[i] - after) : 0.0f;
            const float sum = pl_warp_sum(weight);
            if (h < HEADS) {
                ps[h * KEYS + key] = weight;
                if (lane == 0) {
                    sums[h * kChunks + chunk] = sum;
                    corrections[h * kChunks + chunk] = any ? expf(before - after) : 1.0f;
                }
            }
        }
        __syncthreads();
#pragma unroll
        for (int n = 0; n < ACC; ++n) {
            const int column = tid + n * kWideThreads, h = column / hd;
            if (column < HEADS * hd) {
                const float* values = vs + stage * KEYS * hd + column - h * hd;
                for (int c = 0; c < chunks; ++c) {
                    const float corr = corrections[h * kChunks + c];
                    const uint32_t mask = seen[h * kChunks + c];
                    l[n] = l[n] * corr + sums[h * kChunks + c];
                    acc[n] *= corr;
                    if (mask == 0xffffffffu) {
#pragma unroll
                        for (int j4 = 0; j4 < 32; j4 += 4) {
                            const float4 p4 = *reinterpret_cast<const float4*>(ps + h * KEYS + c * 32 + j4);
                            const float* v = values + (c * 32 + j4) * hd;
                            acc[n] = fmaf(p4.x, v[0], acc[n]);
                            acc[n] = fmaf(p4.y, v[hd], acc[n]);
                            acc[n] = fmaf(p4.z, v[2 * hd], acc[n]);
                            acc[n] = fmaf(p4.w, v[3 * hd], acc[n]);
                        }
                    } else {
                        for (int jj = 0; jj < 32; ++jj) {
                            if (mask >> jj & 1) {
                                acc[n] = fmaf(ps[h * KEYS + c * 32 + jj], values[(c * 32 + jj) * hd], acc[n]);
                            }
                        }
                    }
                }
            }
        }
    }
    // (the walk's last maximum, for the sink: every thread of set h has it for head h; the columns' threads make it again)
    __syncthreads();
#pragma unroll
    for (int i = 0; i < kOwn; ++i) {
        if (key == 0 && set + i * kSets < HEADS) {
            largest[set + i * kSets] = m[i];
        }
    }
    __syncthreads();
#pragma unroll
    for (int n = 0; n < ACC; ++n) {
        const int column = tid + n * kWideThreads, h = column / hd;
        if (column >= HEADS * hd) {
            continue;
        }
        if (a.sinks != nullptr) {
            const float sink = a.sinks[head0 + h], top = largest[h];
            const float m_new = fmaxf(top, sink);
            const float corr = top > -INFINITY ? expf(top - m_new) : 0.0f;
            l[n] = l[n] * corr + expf(sink - m_new);
            acc[n] *= corr;
        }
        float inv = l[n] > 0.0f ? 1.0f / l[n] : 0.0f;
        if (a.gate != nullptr) {
            inv *= 1.0f / (1.0f + expf(-a.gate[t * a.gate_row_stride + head0 + h]));
        }
        a.out[t * a.out_row_stride + static_cast<int64_t>(head0) * hd + column] = acc[n] * inv;
    }
}

template <int HEADS, int KEYS, int ACC>
cudaError_t launch_wide(const StagedParams& a, int n_kv_heads, cudaStream_t stream) {
    constexpr auto kernel = attention_f32_wide_kernel<HEADS, KEYS, ACC>;
    constexpr int kMost = wide_smem_bytes<HEADS, KEYS>(KEYS == 128 ? 64 : 128);
    static_assert(kMost <= 227 * 1024, "shared memory");
    if (const cudaError_t set = pl_allow_smem<kernel>(kMost); set != cudaSuccess) {
        return set;
    }
    kernel<<<dim3(a.n_tokens, n_kv_heads, a.group / HEADS), kWideThreads, wide_smem_bytes<HEADS, KEYS>(a.head_dim), stream>>>(a);
    return cudaGetLastError();
}

template <int P, int ACC, int DIM>
cudaError_t launch_staged(const StagedParams& a, int n_kv_heads, cudaStream_t stream) {
    const int pairs = a.run * a.group;
    const int warps = (pairs + P - 1) / P;
    const int smem = staged_smem_bytes(pairs, a.head_dim);
    constexpr auto kernel = attention_f32_staged_kernel<P, ACC, DIM>;
    const cudaError_t set = pl_allow_smem<kernel>(staged_smem_bytes(P == 1 ? 16 : 32, 32 * ACC));  // (the most of either form)
    if (set != cudaSuccess) {
        return set;
    }
    kernel<<<dim3((a.n_tokens + a.run - 1) / a.run, n_kv_heads), warps * 32, smem, stream>>>(a);
    return cudaGetLastError();
}

}  // namespace

// q [T, n_heads, head_dim] with q_row_stride elements between tokens; out likewise
// with out_row_stride. Token t is the query at position pos[t] of the request whose
// block-table row is table[entry[t]] of n_entries rows; it attends keys max(0, pos - window + 1) ..
// pos (window <= 0: from 0). Pools as in pl_rope_kv_write. mass_sum [n_pages,
// n_heads] and weight_sum [n_pages] (fp32, may be nullptr) are added to: for every
// page a query attends, query_weights[t] (1 when nullptr) times the query's largest
// scaled score in the page, per head, and the weight itself once per page
// (pulsarlm-core/inc/pulsarlm/kernels/ops.hpp:150-160). softcap > 0: every scaled
// score s becomes softcap * tanh(s / softcap) before the softmax (0: off). sinks (fp32
// [n_heads], may be nullptr): exp(sinks[h]) is added to head h's softmax denominator. gate
// ([T, n_heads] logits with gate_row_stride elements between rows, may be nullptr): head
// h's output for token t is multiplied by sigmoid(gate[t, h]). distance_bias (fp32 [n_heads,
// bias_rows], may be nullptr): distance_bias[h, min(pos - key's position, bias_rows - 1)] is added
// to head h's scaled score. distance_slopes (fp32 [n_heads], may be nullptr): distance_slopes[h] times the
// distance is taken off head h's scaled score. keep_first > 0: the request's first keep_first keys stay in reach
// besides the window's.
PL_API int pl_attention_simt(const void* q, int64_t q_row_stride, const void* k_pool, const void* v_pool,
                             int64_t page_stride, int64_t head_stride, int page_size, int n_pages,
                             const int32_t* table, int table_width, const int32_t* pos, const int32_t* entry,
                             void* out, int64_t out_row_stride, int n_tokens, int n_heads, int n_kv_heads,
                             int head_dim, int window, float scale, float softcap, int dtype, float* mass_sum,
                             float* weight_sum, const float* query_weights, const float* sinks, const void* gate,
                             int64_t gate_row_stride, const float* distance_bias, int bias_rows,
                             const float* distance_slopes, int keep_first, int n_entries, int32_t* status,
                             cudaStream_t stream) {
    PL_REQUIRE(n_tokens >= 0 && n_heads > 0 && n_kv_heads > 0 && head_dim > 0 && page_size > 0,
               "attention: bad sizes tokens=%d heads=%d kv_heads=%d head_dim=%d page=%d", n_tokens, n_heads,
               n_kv_heads, head_dim, page_size);
    PL_REQUIRE(n_heads % n_kv_heads == 0, "attention: %d query heads are not a multiple of %d kv heads", n_heads,
               n_kv_heads);
    PL_REQUIRE(head_dim <= 32 * kMaxAccWide, "attention: head_dim %d exceeds the supported maximum %d", head_dim,
               32 * kMaxAccWide);
    PL_REQUIRE(n_kv_heads <= 65535, "attention: %d kv heads exceed the grid limit", n_kv_heads);
    PL_REQUIRE(mass_sum == nullptr || weight_sum != nullptr, "attention: attention mass needs weight_sum too");
    PL_REQUIRE(distance_bias == nullptr || bias_rows > 0, "attention: a distance bias needs rows");
    if (n_tokens == 0) {
        return 0;
    }
    const int group = n_heads / n_kv_heads;
    // The staged form takes float32 rows of whole 16-byte pieces up to 128, up to 16 heads a kv head, no mass. Up to
    // 64 tokens a CTA has one token and a warp one head of it (nothing is shared between a step's single tokens, and a
    // short portion's few CTAs finish soonest so); beyond, as many neighbouring tokens as make 32 pairs, in runs that one
    // request's tokens fill; the tokens of the other runs (single tokens, ends of portions) one a CTA (300 keys, 32 heads of 64 over
    // 8: 128 single tokens 473 us by the plain kernel, 391 in runs, 64 so; 40 of them beside a portion of 90 422, 391, 111).
    // With one head a kv head and rows above 64 values a CTA of one token is one warp beside 100 KB, two of them an SM. There a
    // request's portion goes in runs from a few tokens on (32 heads of 128, 64 tokens: one a CTA 66 us, in a run 35), portions of eight
    // tokens and more on average in runs of whatever requests (20 of 12 tokens, 300 keys: plain 745 us, one a CTA 985, in runs
    // 406), and more than 64 single tokens by the plain kernel (200 of 300 keys: 604 us, one a CTA 811).
    const bool several = n_entries > 1, thin = group == 1 && head_dim > 64;
    if (dtype == PL_F32 && mass_sum == nullptr && head_dim % 4 == 0 && head_dim <= kStagedDim && group <= 16 &&
        page_stride % 4 == 0 && head_stride % 4 == 0 &&
        ((reinterpret_cast<uintptr_t>(k_pool) | reinterpret_cast<uintptr_t>(v_pool)) & 15) == 0 &&
        !(thin && n_tokens > 64 && n_tokens <= n_entries)) {
        const bool few = n_tokens <= 64 && (several || !thin || n_tokens <= 4);
        const bool apart = !few && several && !(thin && n_tokens / 8 >= n_entries);
        const int run = 32 / group;
        StagedParams a{static_cast<const float*>(q), q_row_stride, static_cast<const float*>(k_pool),
                       static_cast<const float*>(v_pool), page_stride, head_stride, page_size, n_pages, table,
                       table_width, pos, entry, static_cast<float*>(out), out_row_stride, n_tokens, group, head_dim,
                       window, run, apart ? run : 0, scale, softcap, sinks, static_cast<const float*>(gate),
                       gate_row_stride, distance_bias, bias_rows, distance_slopes, keep_first > 0 ? keep_first : 0,
                       status};
        cudaError_t failed = cudaSuccess;
        // Steps of few tokens without a window: the form whose parts are side by side, as long as every one of its CTAs (135 KB of
        // keys and values each) has an SM to itself, two heads a CTA where there are SMs for that, else four; and where the table has
        // room for more keys than one of its steps takes. 300 and 1,000 keys, us before and now: 32 heads of 64 over 8, 8 tokens 20.9
        // -> 13.7, 55.7 -> 29.6; 8 heads over 8, 8 tokens 27.0 -> 12.7, 74.1 -> 29.1; 32 heads of 128 over 8, 8 tokens 27.0 -> 21.6,
        // 73.3 -> 59.8; 16 over 2, 32 tokens 22.1 -> 16.8, 57.2 -> 37.5. With more CTAs than SMs: 32 over 8, 32 tokens 22.9 and 29.5.
        const int64_t pairs = static_cast<int64_t>(n_tokens) * n_kv_heads;
        const int heads = group % 4 == 0 && pairs * (group / 2) > 148 ? 4 : group % 2 == 0 ? 2 : 1;
        if (few && window <= 0 && pairs * (group / heads) <= 148 && static_cast<int64_t>(table_width) * page_size > 128) {
            failed = head_dim <= 64 ? (heads == 4   ? launch_wide<4, 128, 1>(a, n_kv_heads, stream)
                                       : heads == 2 ? launch_wide<2, 128, 1>(a, n_kv_heads, stream)
                                                    : launch_wide<1, 128, 1>(a, n_kv_heads, stream))
                                    : (heads == 4   ? launch_wide<4, 64, 2>(a, n_kv_heads, stream)
                                       : heads == 2 ? launch_wide<2, 64, 1>(a, n_kv_heads, stream)
                                                    : launch_wide<1, 64, 1>(a, n_kv_heads, stream));
            if (failed != cudaSuccess) {
                return pl_fail(3, "attention: launch failed: %s", cudaGetErrorString(failed));
            }
            return 0;
        }
        if (!few) {
            failed = head_dim <= 64 ? launch_staged<4, 2, 0>(a, n_kv_heads, stream)
                                    : launch_staged<4, 4, 0>(a, n_kv_heads, stream);
        }
        if (failed == cudaSuccess && (few || apart)) {
            a.run = 1;
            failed = head_dim == 64    ? launch_staged<1, 2, 64>(a, n_kv_heads, stream)
                     : head_dim == 128 ? launch_staged<1, 4, 128>(a, n_kv_heads, stream)
                     : head_dim <= 64  ? launch_staged<1, 2, 0>(a, n_kv_heads, stream)
                                       : launch_staged<1, 4, 0>(a, n_kv_heads, stream);
        }
        if (failed != cudaSuccess) {
            return pl_fail(3, "attention: launch failed: %s", cudaGetErrorString(failed));
        }
        PL_CHECK_LAUNCH("attention");
        return 0;
    }
    const int warps = group < 8 ? group : 8;
    const size_t smem = static_cast<size_t>(warps) * head_dim * sizeof(float);
    const dim3 grid(n_tokens, n_kv_heads);
    PL_DISPATCH_DTYPE(dtype, "attention", {
        // (rows above 512 take the build with twice the accumulators a lane)
        auto kernel = head_dim <= 32 * kMaxAcc ? attention_simt_kernel<scalar_t, kMaxAcc>
                                               : attention_simt_kernel<scalar_t, kMaxAccWide>;
        kernel<<<grid, warps * 32, smem, stream>>>(
            static_cast<const scalar_t*>(q), q_row_stride, static_cast<const scalar_t*>(k_pool),
            static_cast<const scalar_t*>(v_pool), page_stride, head_stride, page_size, n_pages, table, table_width,
            pos, entry, static_cast<scalar_t*>(out), out_row_stride, n_heads, group, head_dim, window, scale,
            softcap, mass_sum, weight_sum, query_weights, sinks, static_cast<const scalar_t*>(gate), gate_row_stride,
            distance_bias, bias_rows, distance_slopes, keep_first > 0 ? keep_first : 0, status);
    });
    PL_CHECK_LAUNCH("attention");
    return 0;
}
