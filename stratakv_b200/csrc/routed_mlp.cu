// A routed feed-forward (mixture of experts): router, sort of the (token, choice) pairs by expert, projections over
// the sorted pairs with each expert's own weights, and the weighted sum.
//
//   s = sigmoid(router . h)                     float sums, one score per expert (or softmax over all experts)
//   chosen: the `top` largest s + correction    (the lower index among equals; the correction chooses only); with
//                                               groups: the experts form equal groups of neighbours, a group scores
//                                               what its best expert does, and only the `keep` best groups' experts
//                                               can be chosen
//   weight of a chosen expert: s * scale        (renormalize: s divided by the chosen scores' sum + renorm_eps first)
//   share = sigmoid(shared_gate . h)            one number per token for a shared expert, if the layer has one
//
// Nothing is read back to the host: the number of pairs of every expert stays on the device (offsets [experts + 1]),
// and the projections are launched over an upper bound of row tiles, each of which looks up its expert.
#include "common.cuh"

namespace skv {

constexpr int ROUTE_THREADS = 256;
constexpr int ROUTE_MAX_EXPERTS = 1024;
constexpr int ROUTE_MAX_TOP = 16;

// The dot product of a weight row and a float row in shared memory, a warp's share of it: VEC, sixteen bytes of the weight
// at a time (rows of whole 16 bytes).
template <bool VEC>
__device__ __forceinline__ float route_dot(const float* __restrict__ w_row, const float* row, int hidden, int lane) {
    float acc = 0.0f;
    if (VEC) {
        for (int w = 4 * lane; w < hidden; w += 128) {
            const float4 a = *(const float4*)(w_row + w), b = *(const float4*)(row + w);
            acc = fmaf(a.x, b.x, acc); acc = fmaf(a.y, b.y, acc); acc = fmaf(a.z, b.z, acc); acc = fmaf(a.w, b.w, acc);
        }
    } else {
        for (int w = lane; w < hidden; w += 32) acc = fmaf(w_row[w], row[w], acc);
    }
    return acc;
}

template <bool VEC>
__device__ __forceinline__ float route_dot(const __nv_bfloat16* __restrict__ w_row, const float* row, int hidden, int lane) {
    float acc = 0.0f;
    if (VEC) {
        for (int w = 8 * lane; w < hidden; w += 256) {
            const uint4 raw = *(const uint4*)(w_row + w);
            const __nv_bfloat162* pairs = (const __nv_bfloat162*)&raw;
            const float4 lo = *(const float4*)(row + w), hi = *(const float4*)(row + w + 4);
            const float2 a = __bfloat1622float2(pairs[0]), b = __bfloat1622float2(pairs[1]);
            const float2 c = __bfloat1622float2(pairs[2]), d = __bfloat1622float2(pairs[3]);
            acc = fmaf(a.x, lo.x, acc); acc = fmaf(a.y, lo.y, acc); acc = fmaf(b.x, lo.z, acc); acc = fmaf(b.y, lo.w, acc);
            acc = fmaf(c.x, hi.x, acc); acc = fmaf(c.y, hi.y, acc); acc = fmaf(d.x, hi.z, acc); acc = fmaf(d.y, hi.w, acc);
        }
    } else {
        for (int w = lane; w < hidden; w += 32) acc = fmaf(__bfloat162float(w_row[w]), row[w], acc);
    }
    return acc;
}

// ---- router ------------------------------------------------------------------------------------------------------
// One token's choice by one warp, from its logits or sigmoids `score` and (sigmoids) its choice scores `choice`.
__device__ __forceinline__ void choose_experts(float* score, float* choice, const float* __restrict__ correction, int t, int lane,
                                               int experts, int top, float scale, int renormalize, int softmax, int groups,
                                               int keep, float renorm_eps, int* __restrict__ chosen, float* __restrict__ weights) {
    if (softmax) {
        // the logits become exp(z - max) / sum over all experts
        float top_logit = -INFINITY;
        for (int e = lane; e < experts; e += 32) top_logit = fmaxf(top_logit, score[e]);
        top_logit = warp_max(top_logit);
        float total = 0.0f;
        for (int e = lane; e < experts; e += 32) {
            const float w = expf(score[e] - top_logit);
            choice[e] = score[e];                     // (logits order experts whose shares are too small to tell apart)
            score[e] = w;
            total += w;
        }
        total = warp_sum(total);
        __syncwarp();
        for (int e = lane; e < experts; e += 32) {
            const float s = score[e] / total;
            score[e] = s;
            if (correction) choice[e] = s + correction[e];
            else if (groups > 1) choice[e] = s;
        }
        __syncwarp();
    }
    if (groups > 1) {
        // `keep` rounds: the group whose best expert scores most (the lower index among equals) is kept, which an
        // infinity in its members' places says; the members of all other groups then leave the choice
        const int size = experts / groups;
        for (int round = 0; round < keep; ++round) {
            float best = 0.0f;
            int best_at = -1;
            for (int g = lane; g < groups; g += 32) {
                bool taken = false;
                for (int e = 0; e < size; ++e) taken = taken || choice[g * size + e] == INFINITY;
                if (taken) continue;
                float top_score = choice[g * size];
                for (int e = 1; e < size; ++e) top_score = fmaxf(top_score, choice[g * size + e]);
                if (best_at < 0 || top_score > best) {
                    best = top_score;
                    best_at = g;
                }
            }
#pragma unroll
            for (int offset = 16; offset > 0; offset >>= 1) {
                const float other = __shfl_xor_sync(0xffffffffu, best, offset);
                const int other_at = __shfl_xor_sync(0xffffffffu, best_at, offset);
                if (other_at >= 0 && (best_at < 0 || other > best || (other == best && other_at < best_at))) {
                    best = other;
                    best_at = other_at;
                }
            }
            __syncwarp();
            if (best_at >= 0)
                for (int e = lane; e < size; e += 32) choice[best_at * size + e] = INFINITY;
            __syncwarp();
        }
        for (int e = lane; e < experts; e += 32) {
            const float c = choice[e];
            const float s = score[e];
            choice[e] = c == INFINITY ? (correction ? s + correction[e] : s) : __int_as_float(0x7fc00000);
        }
        __syncwarp();
    }
    // `top` rounds: the largest choice score left (the lower index among equals); an expert that has been taken is
    // marked with a value that is not a number, which the search passes over
    float picked_sum = 0.0f;
    for (int k = 0; k < top; ++k) {
        float best = 0.0f;
        int best_at = -1;
        for (int e = lane; e < experts; e += 32) {
            const float c = choice[e];
            if (c != c) continue;
            if (best_at < 0 || c > best) {
                best = c;
                best_at = e;
            }
        }
#pragma unroll
        for (int offset = 16; offset > 0; offset >>= 1) {
            const float other = __shfl_xor_sync(0xffffffffu, best, offset);
            const int other_at = __shfl_xor_sync(0xffffffffu, best_at, offset);
            if (other_at >= 0 && (best_at < 0 || other > best || (other == best && other_at < best_at))) {
                best = other;
                best_at = other_at;
            }
        }
        if (best_at < 0) best_at = k;                 // (only where the scores are not numbers)
        const float s = score[best_at];
        picked_sum += s;
        __syncwarp();
        if (lane == 0) {
            chosen[(size_t)t * top + k] = best_at;
            weights[(size_t)t * top + k] = s;
            choice[best_at] = __int_as_float(0x7fc00000);
        }
        __syncwarp();
    }
    if (lane < top) {
        float w = weights[(size_t)t * top + lane];
        if (renormalize) w = w / (picked_sum + renorm_eps);
        weights[(size_t)t * top + lane] = w * scale;
    }
}

template <typename T, bool VEC>
__global__ void __launch_bounds__(ROUTE_THREADS)
route_tokens_kernel(const T* __restrict__ h, const T* __restrict__ router, const float* __restrict__ correction,
                    const T* __restrict__ shared_gate, int hidden, int experts, int top, float scale, int renormalize,
                    int* __restrict__ chosen, float* __restrict__ weights, float* __restrict__ share, int softmax,
                    int groups, int keep, float renorm_eps) {
    extern __shared__ __align__(16) float route_smem[];
    float* row = route_smem;                  // [hidden]
    float* score = row + hidden;              // [experts]
    float* choice = score + experts;          // [experts]
    pdl_launch_dependents();
    pdl_wait();
    const int t = blockIdx.x;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int w = threadIdx.x; w < hidden; w += ROUTE_THREADS) row[w] = to_float(h[(size_t)t * hidden + w]);
    __syncthreads();
    const int dots = experts + (shared_gate ? 1 : 0);
    for (int e = warp; e < dots; e += ROUTE_THREADS / 32) {
        const T* w_row = e < experts ? router + (size_t)e * hidden : shared_gate;
        const float acc = warp_sum(route_dot<VEC>(w_row, row, hidden, lane));
        if (lane == 0) {
            const float s = softmax && e < experts ? acc : 1.0f / (1.0f + expf(-acc));
            if (e < experts) {
                score[e] = s;
                choice[e] = correction ? s + correction[e] : s;
            } else {
                share[t] = s;
            }
        }
    }
    __syncthreads();
    if (warp == 0)
        choose_experts(score, choice, correction, t, lane, experts, top, scale, renormalize, softmax, groups, keep, renorm_eps, chosen, weights);
}

#if SKV_DTYPE == SKV_BF16
// The same on tensor cores, for rows of whole 64 bytes: a block takes 16 tokens, its 16 warps share the hidden numbers out and
// add up in shared memory, then each warp chooses for one token.  Rows and weights are bfloat16, so the products are exact;
// every 16 of them are added to a float sum by an ordinary addition (mma_bf16_add), and the warps' sums in pairs: weights of a softmax
// err as the kernel above does (0.94 to 1.00 of it; 1.1 to 1.4 with 32 products at a time and the warps one after the other).  A block of one token's dot products (above) read
// the router once a token and was a chain of waits: E 8 of 2,048, 8 / 300 / 5,180 tokens
// 4.2 / 6.5 / 37 us, 3.6 / 4.5 / 12.5 here; 64 experts 16 / 32 / 208 and 8 / 9 / 29.
// The first weights are in registers, and the others asked into L2, ahead of the wait: in a step of few tokens they come
// from HBM.
constexpr int ROUTE_ROWS = 16, ROUTE_MMA_WARPS = 16;

template <int NT>
__global__ void __launch_bounds__(ROUTE_MMA_WARPS * 32)
route_tokens_mma_kernel(const __nv_bfloat16* __restrict__ h, const __nv_bfloat16* __restrict__ router,
                        const float* __restrict__ correction, const __nv_bfloat16* __restrict__ shared_gate, int n_tokens,
                        int hidden, int experts, int top, float scale, int renormalize, int* __restrict__ chosen,
                        float* __restrict__ weights, float* __restrict__ share, int softmax, int groups, int keep,
                        float renorm_eps) {
    constexpr int COLS = 8 * NT, PRE = NT == 4 ? 2 : 4;
    extern __shared__ __align__(16) float route_smem[];
    float* part = route_smem;                                         // [warps][ROWS][COLS]
    float* score = part + ROUTE_MMA_WARPS * ROUTE_ROWS * COLS;        // [ROWS][experts]
    float* choice = score + ROUTE_ROWS * experts;                     // [ROWS][experts]
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, tig = lane & 3;
    const int t0 = blockIdx.x * ROUTE_ROWS, dots = experts + (shared_gate ? 1 : 0), steps = hidden / 32;
    auto weight_row = [&](int col) {
        const int e = min(col, dots - 1);
        return e < experts ? router + (size_t)e * hidden : shared_gate;
    };
    uint4 w[PRE][NT];
    auto load_weights = [&](int n0, int s0) {
#pragma unroll
        for (int j = 0; j < NT; ++j) {
            const __nv_bfloat16* row = weight_row(n0 + 8 * j + g) + 8 * tig;
#pragma unroll
            for (int p = 0; p < PRE; ++p) w[p][j] = *(const uint4*)(row + 32 * min(s0 + ROUTE_MMA_WARPS * p, steps - 1));
        }
    };
    load_weights(0, warp);
    if (gridDim.x <= 4)
        for (long long at = threadIdx.x * 128LL; at < 2LL * experts * hidden; at += ROUTE_MMA_WARPS * 32 * 128LL)
            asm volatile("prefetch.global.L2 [%0];" :: "l"((const char*)router + at));
    pdl_launch_dependents();
    pdl_wait();
    const __nv_bfloat16* rows[2];
#pragma unroll
    for (int i = 0; i < 2; ++i) rows[i] = h + (size_t)min(t0 + 8 * i + g, n_tokens - 1) * hidden + 8 * tig;
    for (int n0 = 0; n0 < dots; n0 += COLS) {
        float acc[NT][4] = {};
        for (int s0 = warp; s0 < steps; s0 += ROUTE_MMA_WARPS * PRE) {
            uint4 a[PRE][2];
#pragma unroll
            for (int p = 0; p < PRE; ++p)
#pragma unroll
                for (int i = 0; i < 2; ++i) a[p][i] = *(const uint4*)(rows[i] + 32 * min(s0 + ROUTE_MMA_WARPS * p, steps - 1));
            if (n0 > 0 || s0 > warp) load_weights(n0, s0);
#pragma unroll
            for (int p = 0; p < PRE; ++p) {
                if (s0 + ROUTE_MMA_WARPS * p >= steps) break;
#pragma unroll
                for (int j = 0; j < NT; ++j) {
                    const uint32_t first[1][4] = {{a[p][0].x, a[p][1].x, a[p][0].y, a[p][1].y}}, second[1][4] = {{a[p][0].z, a[p][1].z, a[p][0].w, a[p][1].w}};
                    mma_bf16_add<1>(acc[j], first, w[p][j].x, w[p][j].y);
                    mma_bf16_add<1>(acc[j], second, w[p][j].z, w[p][j].w);
                }
            }
        }
#pragma unroll
        for (int j = 0; j < NT; ++j) {
            float* at = part + ((size_t)warp * ROUTE_ROWS + g) * COLS + 8 * j + 2 * tig;
            *(float2*)at = make_float2(acc[j][0], acc[j][1]);
            *(float2*)(at + 8 * COLS) = make_float2(acc[j][2], acc[j][3]);
        }
        __syncthreads();
        for (int i = threadIdx.x; i < ROUTE_ROWS * COLS; i += ROUTE_MMA_WARPS * 32) {
            const int row = i / COLS, e = n0 + i % COLS;
            if (e >= dots || t0 + row >= n_tokens) continue;
            float sums[ROUTE_MMA_WARPS];                              // (added in pairs: fewer roundings at the sum's full size)
#pragma unroll
            for (int k = 0; k < ROUTE_MMA_WARPS; ++k) sums[k] = part[k * ROUTE_ROWS * COLS + i];
#pragma unroll
            for (int half = ROUTE_MMA_WARPS / 2; half > 0; half /= 2)
#pragma unroll
                for (int k = 0; k < half; ++k) sums[k] += sums[k + half];
            const float sum = sums[0];
            const float s = softmax && e < experts ? sum : 1.0f / (1.0f + expf(-sum));
            if (e < experts) {
                score[row * experts + e] = s;
                choice[row * experts + e] = correction ? s + correction[e] : s;
            } else {
                share[t0 + row] = s;
            }
        }
        __syncthreads();
    }
    if (t0 + warp < n_tokens)
        choose_experts(score + warp * experts, choice + warp * experts, correction, t0 + warp, lane, experts, top, scale,
                       renormalize, softmax, groups, keep, renorm_eps, chosen, weights);
}
#endif

// ---- counting sort of the pairs by expert ----------------------------------------------------------------------------
// One block.  offsets [experts + 1]; order[p] = token of sorted pair p; place[pair] = where the pair went.
__global__ void __launch_bounds__(1024)
sort_by_expert_kernel(const int* __restrict__ chosen, int pairs, int top, int experts, int* __restrict__ offsets,
                      int* __restrict__ order, int* __restrict__ place) {
    __shared__ int counts[ROUTE_MAX_EXPERTS];
    __shared__ int cursor[ROUTE_MAX_EXPERTS];
    __shared__ int warp_totals[32];
    pdl_launch_dependents();
    pdl_wait();
    for (int e = threadIdx.x; e < experts; e += blockDim.x) counts[e] = 0;
    __syncthreads();
    for (int p = threadIdx.x; p < pairs; p += blockDim.x) {
        const int e = chosen[p];
        if (e >= 0 && e < experts) atomicAdd(&counts[e], 1);
    }
    __syncthreads();
    // exclusive scan of counts over up to 1024 experts: a thread per expert
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int mine = threadIdx.x < experts ? counts[threadIdx.x] : 0;
    int inclusive = mine;
#pragma unroll
    for (int offset = 1; offset < 32; offset <<= 1) {
        const int below = __shfl_up_sync(0xffffffffu, inclusive, offset);
        if (lane >= offset) inclusive += below;
    }
    if (lane == 31) warp_totals[warp] = inclusive;
    __syncthreads();
    if (warp == 0) {
        int total = warp_totals[lane];
#pragma unroll
        for (int offset = 1; offset < 32; offset <<= 1) {
            const int below = __shfl_up_sync(0xffffffffu, total, offset);
            if (lane >= offset) total += below;
        }
        warp_totals[lane] = total;
    }
    __syncthreads();
    const int start = inclusive - mine + (warp > 0 ? warp_totals[warp - 1] : 0);
    if (threadIdx.x < experts) {
        cursor[threadIdx.x] = start;
        offsets[threadIdx.x] = start;
        if (threadIdx.x == experts - 1) offsets[experts] = start + mine;
    }
    __syncthreads();
    // Within an expert the pairs keep no particular order: every pair's result is computed from its own row alone,
    // so where it lies among its expert's rows changes nothing.
    for (int p = threadIdx.x; p < pairs; p += blockDim.x) {
        const int e = chosen[p];
        if (e < 0 || e >= experts) { place[p] = 0; continue; }
        const int at = atomicAdd(&cursor[e], 1);
        order[at] = p / top;
        place[p] = at;
    }
}

// ---- projections over the sorted pairs -----------------------------------------------------------------------------
constexpr int EXP_ROWS = 32, EXP_OUTS = 64, EXP_K = 32;

// Row tile `tile` of the launch: which expert, and which of its rows.  Tiles are counted expert by expert, each expert
// having ceil(rows / EXP_ROWS) of them; a tile beyond the last gets no expert.
__device__ __forceinline__ void find_tile(const int* __restrict__ offsets, int experts, int tile, int* expert, int* first,
                                          int* last) {
    int seen = 0;
    *expert = -1;
    for (int e = 0; e < experts; ++e) {
        const int lo = offsets[e], hi = offsets[e + 1];
        const int tiles = (hi - lo + EXP_ROWS - 1) / EXP_ROWS;
        if (tile < seen + tiles) {
            *expert = e;
            *first = lo + (tile - seen) * EXP_ROWS;
            *last = hi;
            return;
        }
        seen += tiles;
    }
}

// GATED: an expert's weight holds 2 N rows, in tiles of 16 (8 gate rows, then the 8 up rows that go with them, as the
// dense gated feed-forward packs them); out[., o] = act(gate_o . a) * (up_o . a).
template <typename TIn, typename TOut, bool GATED>
__global__ void __launch_bounds__(256)
expert_linear_kernel(const TIn* __restrict__ a, int a_stride, const int* __restrict__ rows, const TIn* __restrict__ w,
                     const int* __restrict__ offsets, TOut* __restrict__ out, int experts, int N, int K, act_t act_word) {
    __shared__ float as[EXP_ROWS][EXP_K + 1];
    __shared__ float ws[EXP_OUTS][EXP_K + 1];
    __shared__ float us[GATED ? EXP_OUTS : 1][EXP_K + 1];
    __shared__ int source[EXP_ROWS];
    __shared__ int tile_info[3];
    pdl_launch_dependents();
    pdl_wait();
    if (threadIdx.x == 0) find_tile(offsets, experts, blockIdx.y, &tile_info[0], &tile_info[1], &tile_info[2]);
    __syncthreads();
    const int expert = tile_info[0], first = tile_info[1], last = tile_info[2];
    if (expert < 0) return;
    const int count = min(EXP_ROWS, last - first);
    if (threadIdx.x < EXP_ROWS) {
        const int p = first + threadIdx.x;
        source[threadIdx.x] = threadIdx.x < count ? (rows ? rows[p] : p) : -1;
    }
    __syncthreads();
    const int o0 = blockIdx.x * EXP_OUTS;
    const int act = act_word < 0 ? -1 : (int)(act_word & 0xff);
    const float limit = act_param(act_word);
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    const TIn* w_e = w + (size_t)expert * (GATED ? 2 : 1) * N * K;
    float acc[2][4] = {};
    float up[GATED ? 2 : 1][4] = {};
    for (int k0 = 0; k0 < K; k0 += EXP_K) {
        for (int idx = threadIdx.x; idx < EXP_ROWS * EXP_K; idx += 256) {
            const int r = idx / EXP_K, k = idx % EXP_K;
            const int src = source[r];
            as[r][k] = src >= 0 && k0 + k < K ? to_float(a[(size_t)src * a_stride + k0 + k]) : 0.0f;
        }
        for (int idx = threadIdx.x; idx < EXP_OUTS * EXP_K; idx += 256) {
            const int r = idx / EXP_K, k = idx % EXP_K;
            const int o = o0 + r;
            if (GATED) {
                const size_t gate_row = (size_t)(o >> 3) * 16 + (o & 7);
                ws[r][k] = o < N && k0 + k < K ? to_float(w_e[gate_row * K + k0 + k]) : 0.0f;
                us[r][k] = o < N && k0 + k < K ? to_float(w_e[(gate_row + 8) * K + k0 + k]) : 0.0f;
            } else {
                ws[r][k] = o < N && k0 + k < K ? to_float(w_e[(size_t)o * K + k0 + k]) : 0.0f;
            }
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < EXP_K; ++k) {
            const float a0 = as[ty][k], a1 = as[ty + 16][k];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const float b = ws[tx + 16 * j][k];
                acc[0][j] = fmaf(a0, b, acc[0][j]);
                acc[1][j] = fmaf(a1, b, acc[1][j]);
                if (GATED) {
                    const float c = us[tx + 16 * j][k];
                    up[0][j] = fmaf(a0, c, up[0][j]);
                    up[1][j] = fmaf(a1, c, up[1][j]);
                }
            }
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        const int r = ty + 16 * i;
        if (r >= count) continue;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int o = o0 + tx + 16 * j;
            if (o >= N) continue;
            float v = acc[i][j];
            if (GATED && act == ACT_SWIGLU_CLAMP) {
                out[(size_t)(first + r) * N + o] = from_float<TOut>(clamped_swiglu(v, up[i][j], limit));
                continue;
            }
            if (act == ACT_RELU2) v = relu_squared(v);
            else if (act == ACT_GELU_TANH) v = gelu_tanh(v);
            else if (act == ACT_SILU) v = v / (1.0f + expf(-v));
            if (GATED) v *= up[i][j];
            out[(size_t)(first + r) * N + o] = from_float<TOut>(v);
        }
    }
}

#if SKV_DTYPE == SKV_BF16
// ---- projections of few pairs ----------------------------------------------------------------------------------------
// A block owns 16 weight rows of one expert and streams them once for up to 8 of its rows (the tokens of the mma
// m16n8k16; more rows go round again, with the weights from L2).  Rows are read where the tokens lie (rows: the token of
// each sorted pair), with their weight where `weigh` says so: weights[pair] of the pair that place[] put at this row, on
// the input rounded as scatter_rows rounds it.  A round's loads are all on their way at once: eight steps of 32 k a warp,
// the rows' first, since loads return in the order they were asked for.
// Bound by HBM: the chosen experts' weights.  The 128-row tiles of the tensor-memory form read the same bytes at half
// the rate when a tile holds one to four rows, and need the rows gathered first.  Up and down projection of 8 gated experts of
// 2816 x 2048, gathering included: 1 token x 2 26 + 18 -> 10 + 5 us, 4 tokens 49 + 34 -> 22 + 14, 16 tokens 45 + 23 -> 31 + 20;
// of 7168 x 4096, 16 tokens: 190 + 90 -> 138 + 74 us (6.8 TB/s).
constexpr int FEW_WARPS = 8, FEW_STEPS = 8;
struct FewWeigh { const int* place; const float* weights; int top; };

template <bool GATED, bool FLOAT_OUT>
__global__ void __launch_bounds__(FEW_WARPS * 32, 2)
expert_few_kernel(const __nv_bfloat16* __restrict__ a, int a_stride, const int* __restrict__ rows, const __nv_bfloat16* __restrict__ w,
                  const int* __restrict__ offsets, void* __restrict__ out, int N, int K, act_t act_word, const FewWeigh weigh) {
    __shared__ float part[FEW_WARPS][16][9];
    pdl_launch_dependents();
    pdl_wait();
    const int expert = blockIdx.y, lo = offsets[expert], hi = offsets[expert + 1];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const int n_rows = GATED ? 2 * N : N, n0 = blockIdx.x * 16, steps = (K + 31) >> 5;
    const __nv_bfloat16* w_e = w + (size_t)expert * n_rows * K + 8 * t;
    const __nv_bfloat16 *wa_row = w_e + (size_t)min(n0 + g, n_rows - 1) * K, *wb_row = w_e + (size_t)min(n0 + g + 8, n_rows - 1) * K;
    const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
    for (int first = lo; first < hi; first += 8) {
        const int p = first + g;
        const bool has = p < hi;
        const int source = has && rows ? rows[p] : p;
        const __nv_bfloat16* x_row = a + (size_t)(has ? source : 0) * a_stride + 8 * t;
        float factor = 1.0f;
        if (weigh.place && has)
            for (int k = 0; k < weigh.top; ++k)
                if (weigh.place[source * weigh.top + k] == p) factor = weigh.weights[source * weigh.top + k];
        float acc[4] = {};
        for (int s0 = warp; s0 < steps; s0 += FEW_WARPS * FEW_STEPS) {
            uint4 x[FEW_STEPS], wa[FEW_STEPS], wb[FEW_STEPS];
#pragma unroll
            for (int u = 0; u < FEW_STEPS; ++u) {
                const int k = (s0 + u * FEW_WARPS) * 32;
                x[u] = has && k + 8 * t < K ? *(const uint4*)(x_row + k) : zero;
            }
#pragma unroll
            for (int u = 0; u < FEW_STEPS; ++u) {
                const int k = (s0 + u * FEW_WARPS) * 32;
                wa[u] = k + 8 * t < K ? __ldg((const uint4*)(wa_row + k)) : zero;
                wb[u] = k + 8 * t < K ? __ldg((const uint4*)(wb_row + k)) : zero;
            }
#pragma unroll
            for (int u = 0; u < FEW_STEPS; ++u) {
                if (weigh.place) {
                    __nv_bfloat162* pairs = (__nv_bfloat162*)&x[u];
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const float2 f = __bfloat1622float2(pairs[i]);
                        pairs[i] = __floats2bfloat162_rn(f.x * factor, f.y * factor);
                    }
                }
                mma_bf16_16816(acc, wa[u].x, wb[u].x, wa[u].y, wb[u].y, x[u].x, x[u].y);
                mma_bf16_16816(acc, wa[u].z, wb[u].z, wa[u].w, wb[u].w, x[u].z, x[u].w);
            }
        }
        part[warp][g][2 * t] = acc[0]; part[warp][g][2 * t + 1] = acc[1];
        part[warp][g + 8][2 * t] = acc[2]; part[warp][g + 8][2 * t + 1] = acc[3];
        __syncthreads();
        for (int i = threadIdx.x; i < (GATED ? 64 : 128); i += FEW_WARPS * 32) {
            const int r = GATED ? i & 7 : i & 15, m = GATED ? i >> 3 : i >> 4, o = GATED ? (n0 >> 1) + r : n0 + r;
            if (first + m >= hi || o >= N) continue;
            float v = 0.0f, up = 0.0f;
#pragma unroll
            for (int q = 0; q < FEW_WARPS; ++q) {
                v += part[q][r][m];
                if (GATED) up += part[q][r + 8][m];
            }
            const int act = act_word < 0 ? -1 : (int)(act_word & 0xff);
            if (GATED && act == ACT_SWIGLU_CLAMP) {
                v = clamped_swiglu(v, up, act_param(act_word));
            } else {
                if (act == ACT_RELU2) v = relu_squared(v);
                else if (act == ACT_GELU_TANH) v = gelu_tanh(v);
                else if (act == ACT_SILU) v = v / (1.0f + expf(-v));
                if (GATED) v *= up;
            }
            if (FLOAT_OUT) ((float*)out)[(size_t)(first + m) * N + o] = v;
            else ((__nv_bfloat16*)out)[(size_t)(first + m) * N + o] = __float2bfloat16_rn(v);
        }
        __syncthreads();
    }
}
#endif

// ---- rows in sorted order --------------------------------------------------------------------------------------------
// out[p] = a[rows[p]] for every sorted pair p: the tensor-core projection reads whole tiles of neighbouring rows.
// Rows are K numbers, K * sizeof(T) a multiple of 16 bytes; a warp copies a row.
template <typename T>
__global__ void __launch_bounds__(256)
gather_rows_kernel(const T* __restrict__ a, int a_stride, const int* __restrict__ rows, T* __restrict__ out, int pairs, int K) {
    pdl_launch_dependents();
    pdl_wait();
    const int p = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (p >= pairs) return;
    const uint4* src = (const uint4*)(a + (size_t)rows[p] * a_stride);
    uint4* dst = (uint4*)(out + (size_t)p * K);
    const int pieces = K * (int)sizeof(T) / 16;
    for (int i = lane; i < pieces; i += 32) dst[i] = src[i];
}

// out[place[pair]] = a[token of the pair] * weights[pair] for every (token, choice) pair: the tokens' rows in sorted order
// where the weights multiply the experts' inputs.  VEC: rows of whole 16 bytes.  A warp makes a row.
template <typename T, bool VEC>
__global__ void __launch_bounds__(256)
scatter_rows_kernel(const T* __restrict__ a, const int* __restrict__ place, const float* __restrict__ weights, int top,
                    T* __restrict__ out, int pairs, int K) {
    pdl_launch_dependents();
    pdl_wait();
    const int pair = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (pair >= pairs) return;
    const T* src = a + (size_t)(pair / top) * K;
    T* dst = out + (size_t)place[pair] * K;
    const float w = weights[pair];
    if (VEC) {
        constexpr int EACH = 16 / (int)sizeof(T);
        for (int i = lane; i < K / EACH; i += 32) {
            const uint4 raw = ((const uint4*)src)[i];
            const T* x = (const T*)&raw;
            T y[EACH];
#pragma unroll
            for (int e = 0; e < EACH; ++e) y[e] = from_float<T>(to_float(x[e]) * w);
            ((uint4*)dst)[i] = *(const uint4*)y;
        }
    } else {
        for (int i = lane; i < K; i += 32) dst[i] = from_float<T>(to_float(src[i]) * w);
    }
}

// ---- the weighted sum ----------------------------------------------------------------------------------------------
// grid (tokens, column blocks); VEC: hidden is a multiple of 4 and every pointer is 16-byte aligned.
template <bool VEC>
__global__ void __launch_bounds__(256)
combine_experts_kernel(const float* __restrict__ results, const int* __restrict__ place, const float* __restrict__ weights,
                       const float* __restrict__ shared, const float* __restrict__ share, float* __restrict__ x,
                       int hidden, int top, int add) {
    __shared__ int where[ROUTE_MAX_TOP];
    __shared__ float weight[ROUTE_MAX_TOP];
    pdl_launch_dependents();
    pdl_wait();
    const int t = blockIdx.x;
    if (threadIdx.x < top) {
        where[threadIdx.x] = place[(size_t)t * top + threadIdx.x];
        weight[threadIdx.x] = weights ? weights[(size_t)t * top + threadIdx.x] : 1.0f;
    }
    __syncthreads();
    const float gate = shared ? (share ? share[t] : 1.0f) : 0.0f;
    const int first = blockIdx.y * 256 + threadIdx.x, step = gridDim.y * 256;
    if (VEC) {
        for (int w = 4 * first; w < hidden; w += 4 * step) {
            const size_t at = (size_t)t * hidden + w;
            float4 total = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            for (int k = 0; k < top; ++k) {
                const float4 r = *(const float4*)(results + (size_t)where[k] * hidden + w);
                total.x = fmaf(weight[k], r.x, total.x); total.y = fmaf(weight[k], r.y, total.y);
                total.z = fmaf(weight[k], r.z, total.z); total.w = fmaf(weight[k], r.w, total.w);
            }
            if (shared) {
                const float4 r = *(const float4*)(shared + at);
                total.x = fmaf(gate, r.x, total.x); total.y = fmaf(gate, r.y, total.y);
                total.z = fmaf(gate, r.z, total.z); total.w = fmaf(gate, r.w, total.w);
            }
            if (add) {
                const float4 r = *(const float4*)(x + at);
                total = make_float4(r.x + total.x, r.y + total.y, r.z + total.z, r.w + total.w);
            }
            *(float4*)(x + at) = total;
        }
        return;
    }
    for (int w = first; w < hidden; w += step) {
        float total = 0.0f;
        for (int k = 0; k < top; ++k) total = fmaf(weight[k], results[(size_t)where[k] * hidden + w], total);
        if (shared) total = fmaf(gate, shared[(size_t)t * hidden + w], total);
        const size_t at = (size_t)t * hidden + w;
        x[at] = add ? x[at] + total : total;
    }
}

#if SKV_DTYPE == SKV_BF16
// gemm_tcgen05.cu: the tensor-memory GEMM over rows sorted by group
int grouped_linear_tcgen05(const void* a, const void* w, const int* offsets, void* out, int out_is_float, int rows,
                           int groups, int N, int K, act_t act, int gated, int* flag, cudaStream_t stream);
#endif

}  // namespace skv

using namespace skv;

// h [n, hidden], router [experts, hidden], shared_gate [hidden] or null in the compute dtype; correction float
// [experts] or null.  chosen int [n, top], weights float [n, top], share float [n] (with shared_gate).
SKV_EXPORT int skv_route_tokens(const void* h, const void* router, const float* correction, const void* shared_gate,
                                int n, int hidden, int experts, int top, float scale, int renormalize, int* chosen,
                                float* weights, float* share, int softmax, int groups, int keep, float renorm_eps,
                                cudaStream_t stream) {
    if (n <= 0) return 0;
    if (hidden <= 0 || experts <= 0 || experts > ROUTE_MAX_EXPERTS || top <= 0 || top > experts || top > ROUTE_MAX_TOP)
        return fail("skv_route_tokens", "1 to 16 of 1 to 1024 experts are served");
    if (!h || !router || !chosen || !weights || (shared_gate && !share))
        return fail("skv_route_tokens", "the rows, the router and places for the choice are needed");
    if (groups > 1 && (experts % groups != 0 || keep <= 0 || keep > groups || keep * (experts / groups) < top))
        return fail("skv_route_tokens", "groups must divide the experts, and the kept groups must hold the choices");
    const size_t smem = (size_t)(hidden + 2 * experts) * sizeof(float);
    if (smem > 200 * 1024) return fail("skv_route_tokens", "the hidden size is too large");
#if SKV_DTYPE == SKV_BF16
    if (hidden % 32 == 0 && (((uintptr_t)h | (uintptr_t)router | (uintptr_t)shared_gate) & 15) == 0) {
        const int dots = experts + (shared_gate ? 1 : 0), tiles = dots <= 8 ? 1 : dots <= 16 ? 2 : 4;
        auto wide = tiles == 1 ? route_tokens_mma_kernel<1> : tiles == 2 ? route_tokens_mma_kernel<2> : route_tokens_mma_kernel<4>;
        const size_t room = (size_t)ROUTE_ROWS * (ROUTE_MMA_WARPS * 8 * tiles + 2 * experts) * sizeof(float);
        if (room > 48 * 1024 && cudaFuncSetAttribute(wide, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)room) != cudaSuccess)
            return fail("skv_route_tokens", "cannot reserve shared memory for the scores");
        return launch_pdl("skv_route_tokens", wide, dim3((n + ROUTE_ROWS - 1) / ROUTE_ROWS), dim3(ROUTE_MMA_WARPS * 32), room, stream,
                          (const __nv_bfloat16*)h, (const __nv_bfloat16*)router, correction, (const __nv_bfloat16*)shared_gate, n,
                          hidden, experts, top, scale, renormalize, chosen, weights, share, softmax, groups, keep, renorm_eps);
    }
#endif
    const bool vec = (hidden * sizeof(skv_t)) % 16 == 0 && (((uintptr_t)router | (uintptr_t)shared_gate) & 15) == 0;
    auto kernel = vec ? route_tokens_kernel<skv_t, true> : route_tokens_kernel<skv_t, false>;
    if (smem > 48 * 1024 && cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess)
        return fail("skv_route_tokens", "cannot reserve shared memory for a row");
    return launch_pdl("skv_route_tokens", kernel, dim3(n), dim3(ROUTE_THREADS), smem, stream, (const skv_t*)h,
                      (const skv_t*)router, correction, (const skv_t*)shared_gate, hidden, experts, top, scale,
                      renormalize, chosen, weights, share, softmax, groups, keep, renorm_eps);
}

SKV_EXPORT int skv_sort_by_expert(const int* chosen, int pairs, int top, int experts, int* offsets, int* order,
                                  int* place, cudaStream_t stream) {
    if (experts <= 0 || experts > ROUTE_MAX_EXPERTS || top <= 0) return fail("skv_sort_by_expert", "1 to 1024 experts are served");
    if (pairs < 0 || !chosen || !offsets || !order || !place) return fail("skv_sort_by_expert", "the choice and places for the result are needed");
    return launch_pdl("skv_sort_by_expert", sort_by_expert_kernel, dim3(1), dim3(1024), 0, stream, chosen, pairs, top,
                      experts, offsets, order, place);
}

// a [a_rows, a_stride] and w [experts, N, K] in the compute dtype; rows int [pairs] or null (row p reads a[p]);
// out [pairs, N] float (out_is_float) or the compute dtype; act: an activation's word (its code, and a parameter's bits
// in the high half) or -1 for none.
// gated: w is [experts, 2 N, K], tiles of 8 gate rows and their 8 up rows; out = act(gate . a) * (up . a).
// In bfloat16, rows that lie in sorted order already (rows null, a_stride = K) with K a multiple of 8 go to the
// tensor-memory GEMM's grouped form; `flag` is where its bounded waits report that they gave up.
// Few pairs in bfloat16 (skv_expert_few_serves) read each chosen expert's weights once, wherever the rows lie; `place`
// [tokens, top] and `weights` [tokens, top] (both or neither; with rows) multiply each row by its pair's weight first.
// `fullest`: the most rows one expert may have (as many as there are tokens), 0 where it is not known.
SKV_EXPORT int skv_expert_few_serves(int pairs, int experts, int K, int fullest) {
#if SKV_DTYPE == SKV_BF16
    // up to four rows an expert on average: 16 tokens x 2 of 8 experts of 7168 x 4096 take 138 + 74 us here and 190 + 90 in the
    // tensor-memory form's tiles, 1 token 42 + 22 and 87 + 62.  Short rows leave a block little to stream (64 experts, rows of
    // 512: 64 pairs 41 us against 46, 128 pairs 52 against 46): they come here up to a pair an expert.
    // Where all tokens choose the same experts these go over their rows eight a round: with 2 of 8 experts of 2816 x 2048 or 4 of 64
    // of 1408 x 2048 chosen by all of 16 / 32 / 64 tokens 16 + 9 / - / - and 24 + 16 / 36 + 23 / 62 + 35 us, in tiles 17 + 14 / - / -
    // and 16 + 11 / 16 + 11 / 16 + 12 (8 of 128 of 1024 x 2048, 16 tokens: 35 + 29 and 19 + 12).  So more than two rounds are not
    // risked, though choices at random gain there too (4 of 64, 16 / 64 tokens: 83 + 51 / 121 + 71 against 110 + 63 / 150 + 81).
    return pairs <= (K >= 1024 ? 4 : 1) * experts && K % 8 == 0 && fullest <= 16;
#else
    return 0;
#endif
}

SKV_EXPORT int skv_expert_linear(const void* a, int a_stride, int a_rows, const int* rows, const void* w,
                                 const int* offsets, void* out, int out_is_float, int pairs, int experts, int N, int K,
                                 act_t act, int gated, const int* place, const float* weights, int top, int fullest,
                                 int* flag, cudaStream_t stream) {
    if (pairs <= 0) return 0;
    if (experts <= 0 || experts > ROUTE_MAX_EXPERTS || N <= 0 || K <= 0 || a_stride < K || a_rows <= 0)
        return fail("skv_expert_linear", "sizes do not agree");
    if (!a || !w || !offsets || !out) return fail("skv_expert_linear", "rows, weights, offsets and a place for the result are needed");
    if (act >= 0 && (act & 0xff) >= (gated ? ACT_COUNT : ACT_SWIGLU_CLAMP)) return fail("skv_expert_linear", "this activation is not served");
    if (gated && (act < 0 || N % 8 != 0)) return fail("skv_expert_linear", "a gated weight needs an activation and whole tiles of 8 rows");
    if ((place == nullptr) != (weights == nullptr) || (place && (!rows || top <= 0 || pairs % top)))
        return fail("skv_expert_linear", "weighted rows need their tokens, places and weights");
#if SKV_DTYPE == SKV_BF16
    if (skv_expert_few_serves(pairs, experts, K, fullest) && a_stride % 8 == 0 && !(((uintptr_t)a | (uintptr_t)w) & 15)) {
        const dim3 grid(((gated ? 2 * N : N) + 15) / 16, experts);
        const FewWeigh weigh = {place, weights, top};
        auto kernel = gated ? (out_is_float ? expert_few_kernel<true, true> : expert_few_kernel<true, false>)
                            : (out_is_float ? expert_few_kernel<false, true> : expert_few_kernel<false, false>);
        return launch_pdl("skv_expert_linear", kernel, grid, dim3(FEW_WARPS * 32), 0, stream, (const __nv_bfloat16*)a, a_stride, rows,
                          (const __nv_bfloat16*)w, offsets, out, N, K, act, weigh);
    }
#endif
    if (place) return fail("skv_expert_linear", "rows are weighted on their way in only for few pairs in bfloat16");
#if SKV_DTYPE == SKV_BF16
    if (!rows && a_stride == K && K % 8 == 0 && a_rows >= pairs && !(((uintptr_t)a | (uintptr_t)w) & 15) &&
        (!gated || (!out_is_float && (act & 0xff) != ACT_RELU2)))
        return grouped_linear_tcgen05(a, w, offsets, out, out_is_float, pairs, experts, gated ? 2 * N : N, K,
                                      gated ? act : (act >= 0 ? (act | ACT_ON_STORE) : (act_t)0), gated,
                                      flag, stream);
#endif
    const int row_tiles = (pairs + EXP_ROWS - 1) / EXP_ROWS + experts;       // no expert leaves more than one part tile
    if (row_tiles > 65535) return fail("skv_expert_linear", "too many rows for one launch");
    const dim3 grid((N + EXP_OUTS - 1) / EXP_OUTS, row_tiles);
    if (gated) {
        if (out_is_float)
            return launch_pdl("skv_expert_linear", expert_linear_kernel<skv_t, float, true>, grid, dim3(256), 0, stream,
                              (const skv_t*)a, a_stride, rows, (const skv_t*)w, offsets, (float*)out, experts, N, K, act);
        return launch_pdl("skv_expert_linear", expert_linear_kernel<skv_t, skv_t, true>, grid, dim3(256), 0, stream,
                          (const skv_t*)a, a_stride, rows, (const skv_t*)w, offsets, (skv_t*)out, experts, N, K, act);
    }
    if (out_is_float)
        return launch_pdl("skv_expert_linear", expert_linear_kernel<skv_t, float, false>, grid, dim3(256), 0, stream,
                          (const skv_t*)a, a_stride, rows, (const skv_t*)w, offsets, (float*)out, experts, N, K, act);
    return launch_pdl("skv_expert_linear", expert_linear_kernel<skv_t, skv_t, false>, grid, dim3(256), 0, stream,
                      (const skv_t*)a, a_stride, rows, (const skv_t*)w, offsets, (skv_t*)out, experts, N, K, act);
}

// out [pairs, K] = a[rows[p]] (compute dtype; K * element size a multiple of 16 bytes, both 16-byte aligned).
SKV_EXPORT int skv_gather_rows(const void* a, int a_stride, const int* rows, void* out, int pairs, int K,
                               cudaStream_t stream) {
    if (pairs <= 0) return 0;
    if (!a || !rows || !out || K <= 0 || a_stride < K) return fail("skv_gather_rows", "rows, their indices and a place for them are needed");
    if ((K * sizeof(skv_t)) % 16 || (a_stride * sizeof(skv_t)) % 16 || (((uintptr_t)a | (uintptr_t)out) & 15))
        return fail("skv_gather_rows", "rows must be whole 16-byte pieces");
    return launch_pdl("skv_gather_rows", gather_rows_kernel<skv_t>, dim3((pairs + 7) / 8), dim3(256), 0, stream,
                      (const skv_t*)a, a_stride, rows, (skv_t*)out, pairs, K);
}

// a [pairs / top, K] and out [pairs, K] in the compute dtype: out[place[p]] = a[p / top] * weights[p].
SKV_EXPORT int skv_scatter_rows(const void* a, const int* place, const float* weights, int top, void* out, int pairs, int K,
                                cudaStream_t stream) {
    if (pairs <= 0) return 0;
    if (!a || !place || !weights || !out || K <= 0 || top <= 0) return fail("skv_scatter_rows", "rows, their places and weights are needed");
    const bool vec = (K * sizeof(skv_t)) % 16 == 0 && (((uintptr_t)a | (uintptr_t)out) & 15) == 0;
    auto kernel = vec ? scatter_rows_kernel<skv_t, true> : scatter_rows_kernel<skv_t, false>;
    return launch_pdl("skv_scatter_rows", kernel, dim3((pairs + 7) / 8), dim3(256), 0, stream, (const skv_t*)a, place, weights,
                      top, (skv_t*)out, pairs, K);
}

// weights null: every choice counts as it is.
SKV_EXPORT int skv_combine_experts(const float* results, const int* place, const float* weights, const float* shared,
                                   const float* share, float* x, int n, int hidden, int top, int add,
                                   cudaStream_t stream) {
    if (n <= 0) return 0;
    if (hidden <= 0 || top <= 0 || top > ROUTE_MAX_TOP) return fail("skv_combine_experts", "1 to 16 choices a token are served");
    if (!results || !place || !x || (share && !shared))
        return fail("skv_combine_experts", "results, places, weights and the stream are needed");
    const bool vec = hidden % 4 == 0 && (((uintptr_t)results | (uintptr_t)shared | (uintptr_t)x) & 15) == 0;
    // a row of a step of few tokens is cut into blocks of columns that run side by side
    const int blocks = (hidden + (vec ? 1023 : 255)) / (vec ? 1024 : 256), room = (2 * sm_count() + n - 1) / n;
    auto kernel = vec ? combine_experts_kernel<true> : combine_experts_kernel<false>;
    return launch_pdl("skv_combine_experts", kernel, dim3(n, blocks < room ? blocks : room), dim3(256), 0, stream, results, place,
                      weights, shared, share, x, hidden, top, add);
}
