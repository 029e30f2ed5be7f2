// Attention with the head sizes as run-time arguments and the optional mechanisms that the
// head-size-specialised kernels do not have: biases on the projections, a norm on each value head,
// values narrower or wider than keys, a bias on the score that grows with the logarithm of the
// distance, and a gate per head on the output.  Two kernels:
//
//   qkv_finish:        float rows [q | k | v | ...] of the fused projection -> queries in the compute
//                      dtype, keys and (normalised) values in their places of the paged cache; a warp per
//                      (token, head);
//   attention_general: one warp per (token, head) over the sequence's own cached keys, online softmax
//                      by chunks of 32 keys, everything after the loads in float.
//
// score(i, j) = (q_i . k_j) * scale - r1[head] * ln(1 + r2[head] * (i - j))      (r1 null: no such term)
//               then cap * tanh(score / cap)                                      (cap 0: no cap)
// visible:      0 <= i - j < window   (window 0: every earlier key)
// out(i)      = softmax(score) . v  *  sigmoid(gate[i, head])                    (gate null: no gate; with
//               gate_per_element the logit of every output number: gate[i, head * vdim + d])
//
// qkv_finish can also divide every query and key head by its root mean square (unit norm, no weight, or with a
// weight on the keys, which is how a compressed latent per position is normed before it is cached), and multiply
// the queries of position p by 1 + coef * ln(floor((p + 1) / every) + 1).  A row may hold queries only (keys and
// values of another layer are used) or no values (vdim 0: the cached latent serves as key and value).
//
// Cache layout per entry: keys [block][kv_head][block_size][dim], values [block][kv_head][block_size][vdim].
// These kernels are the same in every build of the library (no compile-time head size); they serve the
// float32 path and every shape the specialised bfloat16 kernels do not take.
#include "common.cuh"

namespace skv {

constexpr int GEN_WARPS = 4;
constexpr int GEN_MAX_VDIM = 512;             // a lane keeps vdim / 32 accumulators: 8 up to 256, else 16

constexpr int FINISH_WARPS = 8;

// Optional steps of qkv_finish, all off when zero: the unit norm of query heads and of key heads (eps qk_eps; the
// keys' with a weight [kv_heads * dim] if k_weight is given) and the queries' temperature by position.
struct FinishExtras {
    int key_dim;               // width of a key head where it differs from a query head's (a cached latent); else dim
    int q_norm, k_norm;
    float qk_eps;
    const float* k_weight;
    float q_temp_coef;
    int q_temp_every;
};

template <typename T>
__device__ __forceinline__ void finish_store4(T* out, float4 v, float factor) {
    if (sizeof(T) == 4) {
        *(float4*)out = make_float4(v.x * factor, v.y * factor, v.z * factor, v.w * factor);
    } else {
        const __nv_bfloat162 lo = __floats2bfloat162_rn(v.x * factor, v.y * factor);
        const __nv_bfloat162 hi = __floats2bfloat162_rn(v.z * factor, v.w * factor);
        *(uint2*)out = make_uint2(*(const uint32_t*)&lo, *(const uint32_t*)&hi);
    }
}

__device__ __forceinline__ float4 finish_load4(const float* x, const float* bias) {
    float4 v = *(const float4*)x;
    if (bias) {
        const float4 b = *(const float4*)bias;
        v.x += b.x; v.y += b.y; v.z += b.z; v.w += b.w;
    }
    return v;
}

// One warp per (token, head): the token's query heads, then its key heads, then its value heads.
// value_norm != 0 divides each value head by sqrt(mean(v^2) + eps).  VEC: head sizes (at most 256) and the row
// stride are multiples of 4 and every pointer is 16-byte aligned; a lane then holds up to eight numbers of the
// head, whose loads go out before the lookups that say where the head is to be written.
template <typename T, bool VEC>
__global__ void __launch_bounds__(FINISH_WARPS * 32)
qkv_finish_kernel(const float* __restrict__ qkv, int row_stride, const float* __restrict__ q_bias,
                  const float* __restrict__ k_bias, const float* __restrict__ v_bias,
                  const int* __restrict__ positions, const int* __restrict__ token_seq,
                  const int* __restrict__ block_table, int table_width, T* __restrict__ q_out,
                  T* __restrict__ k_cache, T* __restrict__ v_cache, int n_tokens, int num_heads, int num_kv_heads,
                  int dim, int vdim, int block_size, int value_norm, float value_eps, int write_kv,
                  const FinishExtras extras) {
    pdl_launch_dependents();
    pdl_wait();
    const int lane = threadIdx.x & 31;
    const int per_token = num_heads + (vdim > 0 ? 2 : 1) * num_kv_heads;
    const long long item = (long long)blockIdx.x * FINISH_WARPS + (threadIdx.x >> 5);
    if (item >= (long long)n_tokens * per_token) return;        // whole warps leave together
    const int t = (int)(item / per_token), which = (int)(item - (long long)t * per_token);
    const bool is_query = which < num_heads, is_key = !is_query && which < num_heads + num_kv_heads;
    if (!is_query && !write_kv) return;
    const int g = is_query ? which : (is_key ? which - num_heads : which - num_heads - num_kv_heads);
    const int kdim = extras.key_dim;
    const int n = is_query ? dim : (is_key ? kdim : vdim);
    const float* x = qkv + (size_t)t * row_stride + (is_query ? (size_t)g * dim
                     : is_key ? (size_t)num_heads * dim + (size_t)g * kdim
                              : (size_t)num_heads * dim + (size_t)num_kv_heads * kdim + (size_t)g * vdim);
    const float* bias_base = is_query ? q_bias : (is_key ? k_bias : v_bias);
    const float* bias = bias_base ? bias_base + (size_t)g * n : nullptr;
    const bool normed = (!is_query && !is_key && value_norm) || (is_query && extras.q_norm) || (is_key && extras.k_norm);
    const float norm_eps = is_query || is_key ? extras.qk_eps : value_eps;
    const float* weight = is_key && extras.k_weight ? extras.k_weight + (size_t)g * n : nullptr;
    float temperature = 1.0f;
    if (is_query && extras.q_temp_every > 0)
        temperature = 1.0f + extras.q_temp_coef * logf((float)((positions[t] + 1) / extras.q_temp_every) + 1.0f);

    float4 held[2];
    if (VEC) {
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            const int i = 4 * lane + 128 * u;
            held[u] = i < n ? finish_load4(x + i, bias ? bias + i : nullptr) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        }
    }
    T* out;
    if (is_query) {
        out = q_out + ((size_t)t * num_heads + g) * dim;
    } else {
        const int pos = positions[t];
        const int block = block_table[(size_t)token_seq[t] * table_width + pos / block_size];
        const size_t row = ((size_t)block * num_kv_heads + g) * block_size + (pos % block_size);
        out = (is_key ? k_cache : v_cache) + row * n;
    }
    float factor = 1.0f;
    if (VEC) {
        if (normed) {
            float squares = 0.0f;
#pragma unroll
            for (int u = 0; u < 2; ++u)
                squares += held[u].x * held[u].x + held[u].y * held[u].y + held[u].z * held[u].z + held[u].w * held[u].w;
            factor = 1.0f / sqrtf(warp_sum(squares) / (float)n + norm_eps);
        }
        factor *= temperature;
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            const int i = 4 * lane + 128 * u;
            if (i < n) {
                if (weight) {
                    const float4 w4 = *(const float4*)(weight + i);
                    held[u].x *= w4.x; held[u].y *= w4.y; held[u].z *= w4.z; held[u].w *= w4.w;
                }
                finish_store4<T>(out + i, held[u], factor);
            }
        }
        return;
    }
    if (normed) {
        float squares = 0.0f;
        for (int d = lane; d < n; d += 32) {
            const float v = x[d] + (bias ? bias[d] : 0.0f);
            squares = fmaf(v, v, squares);
        }
        factor = 1.0f / sqrtf(warp_sum(squares) / (float)n + norm_eps);
    }
    factor *= temperature;
    for (int d = lane; d < n; d += 32)
        out[d] = from_float<T>((x[d] + (bias ? bias[d] : 0.0f)) * factor * (weight ? weight[d] : 1.0f));
}

// Rows of a paged cache with one head, copied into a plain matrix: out[i, :] = the row of position positions[i] of
// sequence seqs[i] (for a mixer that needs its sequences' cached vectors side by side, as a GEMM's input).
template <typename T>
__global__ void __launch_bounds__(256)
paged_gather_kernel(const T* __restrict__ cache, const int* __restrict__ block_table, int table_width,
                    const int* __restrict__ positions, const int* __restrict__ seqs, T* __restrict__ out, int n_rows,
                    int width, int block_size) {
    pdl_launch_dependents();
    pdl_wait();
    const int lane = threadIdx.x & 31;
    const long long i = (long long)blockIdx.x * 8 + (threadIdx.x >> 5);
    if (i >= n_rows) return;
    const int pos = positions[i];
    const int block = block_table[(size_t)seqs[i] * table_width + pos / block_size];
    const T* from = cache + ((size_t)block * block_size + pos % block_size) * width;
    T* to = out + (size_t)i * width;
    for (int d = lane; d < width; d += 32) to[d] = from[d];
}

__device__ __forceinline__ float general_dot(const float* __restrict__ q, const float* __restrict__ row, int dim) {
    float sum = 0.0f;
    if ((dim & 3) == 0) {
        for (int d = 0; d < dim; d += 4) {
            const float4 k = *(const float4*)(row + d);
            sum = fmaf(q[d], k.x, sum); sum = fmaf(q[d + 1], k.y, sum);
            sum = fmaf(q[d + 2], k.z, sum); sum = fmaf(q[d + 3], k.w, sum);
        }
    } else {
        for (int d = 0; d < dim; ++d) sum = fmaf(q[d], row[d], sum);
    }
    return sum;
}

__device__ __forceinline__ float general_dot(const float* __restrict__ q, const __nv_bfloat16* __restrict__ row, int dim) {
    float sum = 0.0f;
    if ((dim & 7) == 0) {
        for (int d = 0; d < dim; d += 8) {
            const uint4 raw = *(const uint4*)(row + d);
            const __nv_bfloat162* pairs = (const __nv_bfloat162*)&raw;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const float2 k = __bfloat1622float2(pairs[i]);
                sum = fmaf(q[d + 2 * i], k.x, sum);
                sum = fmaf(q[d + 2 * i + 1], k.y, sum);
            }
        }
    } else {
        for (int d = 0; d < dim; ++d) sum = fmaf(q[d], __bfloat162float(row[d]), sum);
    }
    return sum;
}

template <typename T, int GEN_ACC>
__global__ void __launch_bounds__(GEN_WARPS * 32)
attention_general_kernel(const T* __restrict__ q, const T* __restrict__ k_cache, const T* __restrict__ v_cache,
                         const int* __restrict__ block_table, int table_width, const int* __restrict__ positions,
                         const int* __restrict__ token_seq, T* __restrict__ out, int n_tokens, int num_heads,
                         int num_kv_heads, int dim, int vdim, int block_size, float scale, int window,
                         const float* __restrict__ r1, const float* __restrict__ r2, const float* __restrict__ gate,
                         int gate_stride, int out_stride, float softcap, int gate_per_element,
                         const float* __restrict__ sink, int v_stride, int splits, float* __restrict__ partial_o,
                         float* __restrict__ partial_ml) {
    extern __shared__ __align__(16) float general_q[];          // [GEN_WARPS][dim rounded up to 4]
    pdl_launch_dependents();
    pdl_wait();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const long long work = (long long)blockIdx.x * GEN_WARPS + warp;
    if (work >= (long long)n_tokens * num_heads * splits) return;        // whole warps leave together
    // With splits > 1 a warp takes one part of its (token, head)'s keys and leaves its sums, their maximum and its
    // unnormalised output for attention_general_merge_kernel; the heads of a token stay side by side in a block.
    const long long item = splits > 1 ? (work / ((long long)num_heads * splits)) * num_heads + work % num_heads : work;
    const int split = splits > 1 ? (int)((work / num_heads) % splits) : 0;
    const int t = (int)(item / num_heads), head = (int)(item % num_heads);
    const int kv_head = head / (num_heads / num_kv_heads);
    const int pos = positions[t];
    const int* table = block_table + (size_t)token_seq[t] * table_width;
    const int lo = window > 0 ? max(0, pos - window + 1) : 0;
    const float slope = r1 ? r1[head] : 0.0f, reach = r1 ? r2[head] : 0.0f;

    float* qs = general_q + (size_t)warp * ((dim + 3) & ~3);
    const T* q_row = q + ((size_t)t * num_heads + head) * dim;
    for (int d = lane; d < dim; d += 32) qs[d] = to_float(q_row[d]);
    __syncwarp();

    float acc[GEN_ACC];
#pragma unroll
    for (int i = 0; i < GEN_ACC; ++i) acc[i] = 0.0f;
    float running_max = -INFINITY, running_sum = 0.0f;

    // this warp's keys: all of lo .. pos, or its part of them in whole runs of 32
    int first_key = lo, last_key = pos;
    if (splits > 1) {
        const int runs = (pos - lo + 32) / 32, per_split = (runs + splits - 1) / splits;
        first_key = lo + split * per_split * 32;
        last_key = min(pos, first_key + per_split * 32 - 1);
    }
    for (int j0 = first_key; j0 <= last_key; j0 += 32) {
        const int j = j0 + lane;
        const bool valid = j <= last_key;
        size_t row = 0;                                // row of this key in units of one head's vector
        float score = -INFINITY;
        if (valid) {
            const int block = table[j / block_size];
            row = ((size_t)block * num_kv_heads + kv_head) * block_size + (j % block_size);
            score = general_dot(qs, k_cache + row * dim, dim) * scale;
            if (r1) score -= slope * log1pf(reach * (float)(pos - j));
            if (softcap > 0.0f) score = softcap * tanhf(score / softcap);
        }
        const float new_max = fmaxf(running_max, warp_max(score));
        const float p = valid ? expf(score - new_max) : 0.0f;
        const float rescale = expf(running_max - new_max);     // 0 on the first chunk
        running_sum = running_sum * rescale + warp_sum(p);
        running_max = new_max;
#pragma unroll
        for (int i = 0; i < GEN_ACC; ++i) acc[i] *= rescale;
        const int count = min(32, last_key - j0 + 1);
        for (int jj = 0; jj < count; ++jj) {
            const float pj = __shfl_sync(0xffffffffu, p, jj);
            const unsigned long long rj = __shfl_sync(0xffffffffu, (unsigned long long)row, jj);
            const T* v_row = v_cache + (size_t)rj * v_stride;
#pragma unroll
            for (int i = 0; i < GEN_ACC; ++i) {
                const int d = lane + 32 * i;
                if (d < vdim) acc[i] = fmaf(pj, to_float(v_row[d]), acc[i]);
            }
        }
    }
    if (splits > 1) {
        float* o_part = partial_o + ((size_t)item * splits + split) * vdim;
#pragma unroll
        for (int i = 0; i < GEN_ACC; ++i) {
            const int d = lane + 32 * i;
            if (d < vdim) o_part[d] = acc[i];
        }
        if (lane == 0) {
            partial_ml[((size_t)item * splits + split) * 2] = running_max;      // -infinity: this part had no keys
            partial_ml[((size_t)item * splits + split) * 2 + 1] = running_sum;
        }
        return;
    }
    // a sink counts once in the denominator: it has no key and no value, and is not scaled
    if (sink) running_sum += expf(sink[head] - running_max);
    float factor = 1.0f / running_sum;
    if (gate && !gate_per_element) factor *= 1.0f / (1.0f + expf(-gate[(size_t)t * gate_stride + head]));
    const float* gate_row = gate && gate_per_element ? gate + (size_t)t * gate_stride + (size_t)head * vdim : nullptr;
    T* out_row = out + (size_t)t * out_stride + (size_t)head * vdim;
#pragma unroll
    for (int i = 0; i < GEN_ACC; ++i) {
        const int d = lane + 32 * i;
        if (d < vdim) {
            float value = acc[i] * factor;
            if (gate_row) value *= 1.0f / (1.0f + expf(-gate_row[d]));
            out_row[d] = from_float<T>(value);
        }
    }
    // columns that pad a row for the projection after it are zero
    if (head == num_heads - 1)
        for (int c = num_heads * vdim + lane; c < out_stride; c += 32) out[(size_t)t * out_stride + c] = from_float<T>(0.0f);
}

// The parts of a (token, head) that attention_general_kernel or latent_attention_kernel left with splits > 1, put together:
// the largest maximum, the sums and outputs brought to it, the sink, the gate.  A block per (token, head): the first warp
// makes the parts' weights while the numbers of the first 16 parts are on their way, then a thread adds up its numbers (in the step, 256
// (token, head) of 256 numbers: 6.0 -> 3.8 us).  (A warp per (token, head) that walked the parts one after the other took 20 us for 256 of
// them over 16 parts.)
constexpr int MERGE_THREADS = 256, MERGE_MAX_SPLITS = 1024, MERGE_AHEAD = 16;
template <typename T>
__global__ void __launch_bounds__(MERGE_THREADS)
attention_general_merge_kernel(const float* __restrict__ partial_o, const float* __restrict__ partial_ml,
                               T* __restrict__ out, int n_tokens, int num_heads, int vdim, int splits,
                               const float* __restrict__ gate, int gate_stride, int out_stride, int gate_per_element,
                               const float* __restrict__ sink) {
    __shared__ float weights[MERGE_MAX_SPLITS];
    pdl_launch_dependents();
    pdl_wait();
    const long long item = blockIdx.x;
    const int t = (int)(item / num_heads), head = (int)(item % num_heads);
    // the first numbers of the first parts are on their way while their weights are made (a part without keys left nothing: what is
    // read of it is not used)
    const float* o_parts = partial_o + (size_t)item * splits * vdim;
    float ahead[MERGE_AHEAD];
#pragma unroll
    for (int s = 0; s < MERGE_AHEAD; ++s) ahead[s] = s < splits && (int)threadIdx.x < vdim ? o_parts[(size_t)s * vdim + threadIdx.x] : 0.0f;
    if (threadIdx.x < 32) {
        const int lane = threadIdx.x;
        const float* ml = partial_ml + (size_t)item * splits * 2;
        float top = -INFINITY;
        for (int s = lane; s < splits; s += 32) top = fmaxf(top, ml[2 * s]);      // (the first part always has the first key)
        top = warp_max(top);
        float total = 0.0f;
        for (int s = lane; s < splits; s += 32) {
            const float m = ml[2 * s], w = m == -INFINITY ? 0.0f : expf(m - top);
            weights[s] = w;
            if (w != 0.0f) total += ml[2 * s + 1] * w;
        }
        total = warp_sum(total);
        if (sink) total += expf(sink[head] - top);
        float factor = 1.0f / total;
        if (gate && !gate_per_element) factor *= 1.0f / (1.0f + expf(-gate[(size_t)t * gate_stride + head]));
        for (int s = lane; s < splits; s += 32) weights[s] *= factor;
    }
    __syncthreads();
    const float* gate_row = gate && gate_per_element ? gate + (size_t)t * gate_stride + (size_t)head * vdim : nullptr;
    T* out_row = out + (size_t)t * out_stride + (size_t)head * vdim;
    for (int d = threadIdx.x; d < vdim; d += MERGE_THREADS) {
        float value = 0.0f;
        const bool first = d == (int)threadIdx.x;
        if (first) {
#pragma unroll
            for (int s = 0; s < MERGE_AHEAD; ++s) {
                const float w = s < splits ? weights[s] : 0.0f;
                if (w != 0.0f) value = fmaf(ahead[s], w, value);
            }
        }
        for (int s0 = first ? MERGE_AHEAD : 0; s0 < splits; s0 += 4) {
            float part[4], w[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {                              // (a part without keys left nothing to read)
                w[u] = s0 + u < splits ? weights[s0 + u] : 0.0f;
                part[u] = w[u] != 0.0f ? o_parts[(size_t)(s0 + u) * vdim + d] : 0.0f;
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) value = fmaf(part[u], w[u], value);
        }
        if (gate_row) value *= 1.0f / (1.0f + expf(-gate_row[d]));
        out_row[d] = from_float<T>(value);
    }
    if (head == num_heads - 1)
        for (int c = num_heads * vdim + threadIdx.x; c < out_stride; c += MERGE_THREADS) out[(size_t)t * out_stride + c] = from_float<T>(0.0f);
}

#if SKV_DTYPE == SKV_BF16
// Part of the keys of one token for 32 of its query heads on tensor cores, where all heads share one cached row of `dim`
// numbers whose first `vdim` are the value (a latent with a rotated part behind it).  Tiles of 64 keys go through shared
// memory once for all heads (cp.async, two stages); eight warps make the scores (16 heads x 16 keys each), then four rows
// of the softmax each, then 16 heads x 64 numbers of the output each.  Scores, softmax and sums are float; a probability
// is split into three bfloat16 that add up to it, against values that are bfloat16 anyway, so nothing is rounded that
// attention_general_kernel kept, and sums are added by mma_bf16_add (relative errors before the output's rounding, rows of 288, two
// parts of 8,000: 2.1e-7, that kernel 7.2e-7; sums left in the tensor core 110e-7, at 1 to 7 % less time).  That kernel, a warp
// per (token, head, part), read every key once per head: with its merge 8 sequences x 32 heads over 780 rows of 272
// numbers took 69 us and take 14, 1 sequence over 8,000 rows 150 and 30, 64 over 500 187 and 31.
constexpr int LAT_KEYS = 64, LAT_HEADS = 32, LAT_MAX_DIM = 320, LAT_MAX_VDIM = 256, LAT_S_PITCH = LAT_KEYS + 4, LAT_P_PITCH = LAT_KEYS + 8;

__device__ __forceinline__ void lat_ldmatrix(uint32_t (&r)[4], const void* p) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];\n" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(smem_u32(p)) : "memory");
}
__device__ __forceinline__ void lat_ldmatrix_trans(uint32_t (&r)[4], const void* p) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];\n" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(smem_u32(p)) : "memory");
}

__global__ void __launch_bounds__(256)
latent_attention_kernel(const __nv_bfloat16* __restrict__ q, const __nv_bfloat16* __restrict__ cache, const int* __restrict__ block_table,
                        int table_width, const int* __restrict__ positions, const int* __restrict__ token_seq, int num_heads, int dim,
                        int vdim, int block_size, float scale, int splits, float* __restrict__ partial_o, float* __restrict__ partial_ml) {
    extern __shared__ __align__(16) unsigned char lat_smem[];
    const int pitch = dim + 8;                                          // rows 16 bytes apart modulo 128: eight of them hit all banks
    __nv_bfloat16* qs = (__nv_bfloat16*)lat_smem;                       // [LAT_HEADS][pitch]
    __nv_bfloat16* keys = qs + LAT_HEADS * pitch;                       // [2][LAT_KEYS][pitch]
    __nv_bfloat16* probs = keys + 2 * LAT_KEYS * pitch;                 // [3][LAT_HEADS][LAT_P_PITCH]
    float* scores = (float*)(probs + 3 * LAT_HEADS * LAT_P_PITCH);      // [LAT_HEADS][LAT_S_PITCH]
    float* rescale = scores + LAT_HEADS * LAT_S_PITCH;                  // [LAT_HEADS]
    pdl_launch_dependents();
    pdl_wait();
    const int t = blockIdx.x / splits, split = blockIdx.x % splits, head0 = blockIdx.y * LAT_HEADS;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, quad = lane & 3;
    const int count = positions[t] + 1, tiles = (count + LAT_KEYS - 1) / LAT_KEYS, per_split = (tiles + splits - 1) / splits;
    const int first = split * per_split, last = min(tiles, first + per_split);
    const int live_heads = min(LAT_HEADS, num_heads - head0);
    const size_t item0 = (size_t)t * num_heads + head0;
    if (first >= last) {
        if (tid < live_heads) {
            partial_ml[((item0 + tid) * splits + split) * 2] = -INFINITY;
            partial_ml[((item0 + tid) * splits + split) * 2 + 1] = 0.0f;
        }
        return;
    }
    const int* table = block_table + (size_t)token_seq[t] * table_width;
    const int pieces = dim / 8;                                         // 16-byte pieces of a row
    auto fetch = [&](int tile, int stage) {
        for (int i = tid; i < LAT_KEYS * pieces; i += 256) {
            const int row = i / pieces, piece = i - row * pieces, j = tile * LAT_KEYS + row;
            const bool live = j < count;                                // (rows beyond the last key are zeros: stale ones may hold anything)
            const int safe = live ? j : 0;
            const __nv_bfloat16* from = cache + ((size_t)table[safe / block_size] * block_size + safe % block_size) * dim + 8 * piece;
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" :: "r"(smem_u32(keys + ((size_t)stage * LAT_KEYS + row) * pitch + 8 * piece)),
                         "l"(from), "r"(live ? 16 : 0) : "memory");
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    fetch(first, 0);
    for (int i = tid; i < LAT_HEADS * pieces; i += 256) {
        const int row = i / pieces, piece = i - row * pieces;
        *(uint4*)(qs + row * pitch + 8 * piece) = row < live_heads ? *(const uint4*)(q + (item0 + row) * dim + 8 * piece) : make_uint4(0u, 0u, 0u, 0u);
    }
    const int m_tile = warp & 1, part = warp >> 1;                      // 16 heads; 16 keys of the scores, 64 numbers of the output
    float acc[8][4] = {};
    float running_max[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY}, running_sum[4] = {};
    for (int tile = first; tile < last; ++tile) {
        const int stage = (tile - first) & 1;
        if (tile + 1 < last) {
            fetch(tile + 1, stage ^ 1);
            asm volatile("cp.async.wait_group 1;" ::: "memory");
        } else {
            asm volatile("cp.async.wait_group 0;" ::: "memory");
        }
        __syncthreads();
        const __nv_bfloat16* k_tile = keys + (size_t)stage * LAT_KEYS * pitch;
        {
            float s[2][4] = {};
            const __nv_bfloat16* q_at = qs + (16 * m_tile + (lane & 15)) * pitch + 8 * (lane >> 4);
            const __nv_bfloat16* k_at = k_tile + (16 * part + (lane & 7) + 8 * (lane >> 4)) * pitch + 8 * ((lane >> 3) & 1);
            for (int d = 0; d < dim; d += 16) {
                uint32_t a[1][4], b[4];
                lat_ldmatrix(a[0], q_at + d);
                lat_ldmatrix(b, k_at + d);
                mma_bf16_add<1>(s[0], a, b[0], b[1]);
                mma_bf16_add<1>(s[1], a, b[2], b[3]);
            }
#pragma unroll
            for (int n = 0; n < 2; ++n)
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const int row = 16 * m_tile + g + 8 * (e >> 1), key = 16 * part + 8 * n + 2 * quad + (e & 1);
                    scores[row * LAT_S_PITCH + key] = tile * LAT_KEYS + key < count ? s[n][e] * scale : -INFINITY;
                }
        }
        __syncthreads();
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int row = 4 * warp + i;
            const float2 s = *(const float2*)(scores + row * LAT_S_PITCH + 2 * lane);
            const float new_max = fmaxf(running_max[i], warp_max(fmaxf(s.x, s.y)));
            const float base = new_max == -INFINITY ? 0.0f : new_max;   // (scores that are all -infinity so far weigh nothing)
            const float p[2] = {expf(s.x - base), expf(s.y - base)};
            const float factor = expf(running_max[i] - base);           // 0 on the first tile
            running_sum[i] = running_sum[i] * factor + warp_sum(p[0] + p[1]);
            running_max[i] = new_max;
            if (lane == 0) rescale[row] = factor;
            uint32_t parts[3];
            split3(p[0], p[1], parts);
#pragma unroll
            for (int k = 0; k < 3; ++k) *(uint32_t*)(probs + (k * LAT_HEADS + row) * LAT_P_PITCH + 2 * lane) = parts[k];
        }
        __syncthreads();
        const float low = rescale[16 * m_tile + g], high = rescale[16 * m_tile + g + 8];
#pragma unroll
        for (int n = 0; n < 8; ++n) { acc[n][0] *= low; acc[n][1] *= low; acc[n][2] *= high; acc[n][3] *= high; }
#pragma unroll
        for (int k = 0; k < LAT_KEYS; k += 16) {
            uint32_t a[3][4];
#pragma unroll
            for (int p = 0; p < 3; ++p) lat_ldmatrix(a[p], probs + (p * LAT_HEADS + 16 * m_tile + (lane & 15)) * LAT_P_PITCH + k + 8 * (lane >> 4));
#pragma unroll
            for (int n = 0; n < 8; n += 2) {
                const int c = 64 * part + 8 * n;
                if (c >= vdim) continue;
                uint32_t b[4];
                lat_ldmatrix_trans(b, k_tile + (k + (lane & 15)) * pitch + c + 8 * (lane >> 4));
                mma_bf16_add<3>(acc[n], a, b[0], b[1]);
                mma_bf16_add<3>(acc[n + 1], a, b[2], b[3]);
            }
        }
        __syncthreads();                                                // (the stage, the scores and the probabilities are free again)
    }
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const int row = 16 * m_tile + g + 8 * h;
        if (row >= live_heads) continue;
        float* o_part = partial_o + ((item0 + row) * splits + split) * vdim;
#pragma unroll
        for (int n = 0; n < 8; ++n) {
            const int c = 64 * part + 8 * n + 2 * quad;
            if (c < vdim) *(float2*)(o_part + c) = make_float2(acc[n][2 * h], acc[n][2 * h + 1]);
        }
    }
    if (lane == 0) {
#pragma unroll
        for (int i = 0; i < 4; ++i)
            if (4 * warp + i < live_heads) {
                partial_ml[((item0 + 4 * warp + i) * splits + split) * 2] = running_max[i];
                partial_ml[((item0 + 4 * warp + i) * splits + split) * 2 + 1] = running_sum[i];
            }
    }
}
#endif

}  // namespace skv

using namespace skv;

// `qkv`: float [n_tokens, row_stride], a row holding heads*dim query, kv_heads*dim key and kv_heads*vdim value
// numbers (whatever follows them is not read).  Biases are float and may be null.
SKV_EXPORT int skv_qkv_finish(const float* qkv, int row_stride, const float* q_bias, const float* k_bias,
                              const float* v_bias, const int* positions, const int* token_seq,
                              const int* block_table, int table_width, void* q_out, void* k_cache, void* v_cache,
                              int n_tokens, int num_heads, int num_kv_heads, int dim, int vdim, int block_size,
                              int value_norm, float value_eps, int write_kv, int q_norm, int k_norm, float qk_eps,
                              const float* k_weight, float q_temp_coef, int q_temp_every, int key_dim,
                              cudaStream_t stream) {
    if (n_tokens <= 0) return 0;
    if (num_heads < 0 || num_kv_heads <= 0 || dim <= 0 || vdim < 0 || block_size <= 0 || (num_heads > 0 && !q_out))
        return fail("skv_qkv_finish", "head counts, head sizes and block_size must be positive");
    if (key_dim <= 0) key_dim = dim;
    if (row_stride < (write_kv ? num_heads * dim + num_kv_heads * (key_dim + vdim) : num_heads * dim))
        return fail("skv_qkv_finish", "a row is shorter than its queries, keys and values");
    if (q_temp_every < 0) return fail("skv_qkv_finish", "the temperature's period must not be negative");
    const FinishExtras extras = {key_dim, q_norm, k_norm, qk_eps, k_weight, q_temp_coef, q_temp_every};
    const long long items = (long long)n_tokens * (num_heads + (vdim > 0 ? 2 : 1) * num_kv_heads);
    const long long blocks = (items + FINISH_WARPS - 1) / FINISH_WARPS;
    if (blocks > 0x7fffffffLL) return fail("skv_qkv_finish", "too many tokens in one step");
    const bool vec = dim % 4 == 0 && vdim % 4 == 0 && key_dim % 4 == 0 && dim <= 256 && vdim <= 256 && key_dim <= 256 &&
                     row_stride % 4 == 0 &&
                     (((uintptr_t)qkv | (uintptr_t)q_bias | (uintptr_t)k_bias | (uintptr_t)v_bias | (uintptr_t)q_out |
                       (uintptr_t)k_cache | (uintptr_t)v_cache | (uintptr_t)k_weight) & 15) == 0;
    auto kernel = vec ? qkv_finish_kernel<skv_t, true> : qkv_finish_kernel<skv_t, false>;
    return launch_pdl("skv_qkv_finish", kernel, dim3((unsigned)blocks), dim3(FINISH_WARPS * 32), 0, stream, qkv,
                      row_stride, q_bias, k_bias, v_bias, positions, token_seq, block_table, table_width,
                      (skv_t*)q_out, (skv_t*)k_cache, (skv_t*)v_cache, n_tokens, num_heads, num_kv_heads, dim, vdim,
                      block_size, value_norm, value_eps, write_kv, extras);
}

// cache: [blocks][1][block_size][width] in the compute dtype; out [n_rows, width].
SKV_EXPORT int skv_paged_gather(const void* cache, const int* block_table, int table_width, const int* positions,
                                const int* seqs, void* out, int n_rows, int width, int block_size, cudaStream_t stream) {
    if (n_rows <= 0) return 0;
    if (width <= 0 || block_size <= 0 || table_width <= 0) return fail("skv_paged_gather", "sizes must be positive");
    return launch_pdl("skv_paged_gather", paged_gather_kernel<skv_t>, dim3((n_rows + 7) / 8), dim3(256), 0, stream,
                      (const skv_t*)cache, block_table, table_width, positions, seqs, (skv_t*)out, n_rows, width, block_size);
}

// Whether attention over one cached row of `dim` numbers for all heads, the first `vdim` of them the value, has a tensor-core form
// for parts of the keys: rows in whole steps of 16 numbers that fit its tiles.
SKV_EXPORT int skv_attention_latent_serves(int dim, int vdim) {
#if SKV_DTYPE == SKV_BF16
    return dim % 16 == 0 && dim <= LAT_MAX_DIM && vdim % 16 == 0 && vdim <= LAT_MAX_VDIM && vdim <= dim;
#else
    return 0;
#endif
}

// `r1`, `r2`: float [num_heads] or both null.  `gate`: float, the gate's logit of (token t, head h) at
// gate[t * gate_stride + h], or null.  `out` rows are out_stride >= heads * vdim apart; what lies beyond a row's
// heads is set to zero.  `sink`: float [num_heads] or null; exp(sink[h]) is added to the softmax's denominator.
// `value_stride`: numbers between the values' rows (0: vdim), so that the head of a wider cached row can be the value.
SKV_EXPORT int skv_attention_general(const void* q, const void* k_cache, const void* v_cache, const int* block_table,
                                     int table_width, const int* positions, const int* token_seq, void* out,
                                     int n_tokens, int num_heads, int num_kv_heads, int dim, int vdim, int block_size,
                                     float scale, int window, const float* r1, const float* r2, const float* gate,
                                     int gate_stride, int out_stride, float softcap, int gate_per_element,
                                     const float* sink, int value_stride, int splits, float* partial_o,
                                     float* partial_ml, cudaStream_t stream) {
    if (n_tokens <= 0) return 0;
    if (splits < 1 || splits > 1024 || (splits > 1 && (!partial_o || !partial_ml)))
        return fail("skv_attention_general", "1 to 1024 parts of the keys, and with more than one the scratch for them");
    if (num_heads <= 0 || num_kv_heads <= 0 || num_heads % num_kv_heads != 0)
        return fail("skv_attention_general", "heads must be a positive multiple of kv heads");
    if (dim <= 0 || vdim <= 0 || vdim > GEN_MAX_VDIM) return fail("skv_attention_general", "value heads of 1 to 512 numbers are served");
    if (softcap < 0.0f) return fail("skv_attention_general", "the cap on the scores must not be negative");
    if (value_stride <= 0) value_stride = vdim;
    if (value_stride < vdim) return fail("skv_attention_general", "the values' rows cannot be closer together than they are wide");
    if (block_size <= 0 || window < 0) return fail("skv_attention_general", "bad block size or window");
    if (out_stride < num_heads * vdim) return fail("skv_attention_general", "a row of the output is shorter than its heads");
    if ((r1 == nullptr) != (r2 == nullptr)) return fail("skv_attention_general", "the distance bias needs both of its numbers per head");
    const size_t smem = (size_t)GEN_WARPS * ((dim + 3) & ~3) * sizeof(float);
    if (smem > 48 * 1024) return fail("skv_attention_general", "the key size is too large");
    const long long items = (long long)n_tokens * num_heads;
    const long long blocks = (items * splits + GEN_WARPS - 1) / GEN_WARPS;
    if (blocks > 0x7fffffffLL) return fail("skv_attention_general", "too many tokens in one step");
#if SKV_DTYPE == SKV_BF16
    // One cached row for all heads whose head is the value, in parts, with nothing that changes a score: the tensor-core
    // form, where the sizes are its own and the partial outputs' rows 8-byte aligned
    const bool latent = splits > 1 && num_kv_heads == 1 && k_cache == v_cache && value_stride == dim && skv_attention_latent_serves(dim, vdim) &&
                        window == 0 && !r1 && softcap == 0.0f && items * splits <= 0x7fffffffLL &&
                        (((uintptr_t)q | (uintptr_t)k_cache | (uintptr_t)partial_o) & 15) == 0;
    if (latent) {
        const size_t room = (size_t)((LAT_HEADS + 2 * LAT_KEYS) * (dim + 8) + 3 * LAT_HEADS * LAT_P_PITCH) * 2 + (size_t)LAT_HEADS * (LAT_S_PITCH + 1) * 4;
        constexpr size_t most = (size_t)((LAT_HEADS + 2 * LAT_KEYS) * (LAT_MAX_DIM + 8) + 3 * LAT_HEADS * LAT_P_PITCH) * 2 + (size_t)LAT_HEADS * (LAT_S_PITCH + 1) * 4;
        if (int code = reserve_shared_once<latent_attention_kernel>("skv_attention_general", most)) return code;
        if (int code = launch_pdl("skv_attention_general(latent)", latent_attention_kernel,
                                  dim3((unsigned)(n_tokens * splits), (unsigned)((num_heads + LAT_HEADS - 1) / LAT_HEADS)), dim3(256), room, stream,
                                  (const __nv_bfloat16*)q, (const __nv_bfloat16*)k_cache, block_table, table_width, positions, token_seq,
                                  num_heads, dim, vdim, block_size, scale, splits, partial_o, partial_ml))
            return code;
        return launch_pdl("skv_attention_general(merge)", attention_general_merge_kernel<skv_t>,
                          dim3((unsigned)items), dim3(MERGE_THREADS), 0, stream,
                          (const float*)partial_o, (const float*)partial_ml, (skv_t*)out, n_tokens, num_heads, vdim, splits,
                          gate, gate_stride, out_stride, gate_per_element, sink);
    }
#endif
    auto kernel = vdim <= 256 ? attention_general_kernel<skv_t, 8> : attention_general_kernel<skv_t, 16>;
    // A warp per (token, head) reads its keys straight through L1, where the heads of a key head find them: behind a projection whose weights wait
    // in shared memory and whose blocks it overlapped it had 60 KB of L1 left.  8 sequences x 32 heads of 256 over 8 with their projection, 8 parts of 300
    // / 2,000 keys: 92 / 304 us overlapping, 75 / 256 so; 32 heads of 96, 52 / 180 and 36 / 141.  (The float32 projections are as they were.)
#if SKV_DTYPE == SKV_BF16
    const auto launch = [&](auto... args) { return launch_alone(args...); };
#else
    const auto launch = [&](auto... args) { return launch_pdl(args...); };
#endif
    if (int code = launch("skv_attention_general", kernel, dim3((unsigned)blocks),
                              dim3(GEN_WARPS * 32), smem, stream, (const skv_t*)q, (const skv_t*)k_cache,
                              (const skv_t*)v_cache, block_table, table_width, positions, token_seq, (skv_t*)out, n_tokens,
                              num_heads, num_kv_heads, dim, vdim, block_size, scale, window, r1, r2, gate, gate_stride,
                              out_stride, softcap, gate_per_element, sink, value_stride, splits, partial_o, partial_ml))
        return code;
    if (splits == 1) return 0;
    return launch_pdl("skv_attention_general(merge)", attention_general_merge_kernel<skv_t>,
                      dim3((unsigned)items), dim3(MERGE_THREADS), 0, stream,
                      (const float*)partial_o, (const float*)partial_ml, (skv_t*)out, n_tokens, num_heads, vdim, splits,
                      gate, gate_stride, out_stride, gate_per_element, sink);
}
