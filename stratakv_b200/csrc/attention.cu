// Causal grouped-query attention over the paged cache, one warp per (token, head), or several where there are few.
//
// Replaces the reference's paged_attention_decode_kernel (src/cuda/gemm_cuda.cu:
// 304-429), which serves one query token, with a kernel for any number of new
// tokens per sequence: a token at absolute position p attends to cached keys
// lo..p of its own sequence (lo = 0, or p - window + 1 with a window), its own key
// included because the cache write runs first.  As in the reference,
// kv_head = q_head / (heads / kv_heads), the scale multiplies the finished dot
// product, and max, exp, sums and the weighted sum of values are in float
// (src/layers/attention.cpp:261-338); the softmax is the online form, by chunks of
// 32 keys.  expf is the accurate one: nothing here is built with fast-math.
//
// Cache layout per entry: [block][kv_head][block_size][head_dim]; a token's keys
// are found through block_table[seq][position / block_size].
#include "head_size.cuh"

namespace skv {

constexpr int HD = SKV_HEAD_DIM;
constexpr int DIMS_PER_LANE = (HD + 31) / 32;
constexpr int ATT_WARPS = 4;

template <typename T, int VEC> struct RowDot;

// dot(q, key row) with 16-byte loads of the row.
__device__ __forceinline__ float row_dot(const float* __restrict__ q, const float* __restrict__ row) {
    float sum = 0.0f;
#pragma unroll
    for (int d = 0; d < HD; d += 4) {
        const float4 k = *(const float4*)(row + d);
        sum = fmaf(q[d], k.x, sum);
        sum = fmaf(q[d + 1], k.y, sum);
        sum = fmaf(q[d + 2], k.z, sum);
        sum = fmaf(q[d + 3], k.w, sum);
    }
    return sum;
}

__device__ __forceinline__ float row_dot(const float* __restrict__ q, const __nv_bfloat16* __restrict__ row) {
    float sum = 0.0f;
#pragma unroll
    for (int d = 0; d < HD; d += 8) {
        const uint4 raw = *(const uint4*)(row + d);
        const __nv_bfloat162* pairs = (const __nv_bfloat162*)&raw;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float2 k = __bfloat1622float2(pairs[i]);
            sum = fmaf(q[d + 2 * i], k.x, sum);
            sum = fmaf(q[d + 2 * i + 1], k.y, sum);
        }
    }
    return sum;
}

// PARTS warps of a block share one (token, head): warp w takes the chunks w, w + PARTS, ... of 32 keys, and the first
// warp merges their softmaxes in order.  PARTS = 1: a block's warps serve ATT_WARPS (token, head) pairs.
// Bound by a warp's chain of loads per chunk, not by bytes: a decode step of 3 sequences x 32 heads of 64 over 250 keys
// took 65 us with one warp each and takes 11 with eight, one sequence over 2,000 keys 487 and 67, 40 sequences over 600
// keys 168 and (four warps each) 107.
template <typename T, int PARTS>
__global__ void __launch_bounds__((PARTS == 1 ? ATT_WARPS : PARTS) * 32)
attention_kernel(const T* __restrict__ q, const T* __restrict__ k_cache, const T* __restrict__ v_cache,
                 const int* __restrict__ block_table, int table_width, const int* __restrict__ positions,
                 const int* __restrict__ token_seq, T* __restrict__ out, int n_tokens, int num_heads,
                 int num_kv_heads, int block_size, float scale, int window) {
    __shared__ __align__(16) float q_smem[PARTS == 1 ? ATT_WARPS : 1][HD];
    __shared__ float part_acc[PARTS][HD], part_max[PARTS], part_sum[PARTS];
    pdl_launch_dependents();
    pdl_wait();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const long long item = PARTS == 1 ? (long long)blockIdx.x * ATT_WARPS + warp : (long long)blockIdx.x;
    if (item >= (long long)n_tokens * num_heads) return;       // whole warps (with PARTS > 1: whole blocks) leave together
    const int t = (int)(item / num_heads), head = (int)(item % num_heads);
    const int kv_head = head / (num_heads / num_kv_heads);
    const int pos = positions[t];
    const int* table = block_table + (size_t)token_seq[t] * table_width;
    const int lo = window > 0 ? max(0, pos - window + 1) : 0;

    float* qs = q_smem[PARTS == 1 ? warp : 0];
    const T* q_row = q + ((size_t)t * num_heads + head) * HD;
    for (int d = PARTS == 1 ? lane : threadIdx.x; d < HD; d += PARTS * 32) qs[d] = to_float(q_row[d]);
    if (PARTS == 1) __syncwarp(); else __syncthreads();

    float acc[DIMS_PER_LANE];
#pragma unroll
    for (int i = 0; i < DIMS_PER_LANE; ++i) acc[i] = 0.0f;
    float running_max = -INFINITY, running_sum = 0.0f;

    for (int j0 = PARTS == 1 ? lo : lo + 32 * warp; j0 <= pos; j0 += 32 * PARTS) {
        const int j = j0 + lane;
        const bool valid = j <= pos;
        int row = 0;                                   // row index in units of HD elements
        float score = -INFINITY;
        if (valid) {
            const int block = table[j / block_size];
            row = (block * num_kv_heads + kv_head) * block_size + (j % block_size);
            score = row_dot(qs, k_cache + (size_t)row * HD) * scale;
        }
        const float new_max = fmaxf(running_max, warp_max(score));
        const float base = new_max == -INFINITY ? 0.0f : new_max;      // (a part whose scores so far are all -infinity weighs nothing)
        const float p = valid ? expf(score - base) : 0.0f;
        const float rescale = expf(running_max - base);        // 0 on the first chunk
        running_sum = running_sum * rescale + warp_sum(p);
        running_max = new_max;
#pragma unroll
        for (int i = 0; i < DIMS_PER_LANE; ++i) acc[i] *= rescale;
        const int count = min(32, pos - j0 + 1);
#pragma unroll 4
        for (int jj = 0; jj < count; ++jj) {
            const float pj = __shfl_sync(0xffffffffu, p, jj);
            const int rj = __shfl_sync(0xffffffffu, row, jj);
            const T* v_row = v_cache + (size_t)rj * HD;
#pragma unroll
            for (int i = 0; i < DIMS_PER_LANE; ++i) {
                const int d = lane + 32 * i;
                if (d < HD) acc[i] = fmaf(pj, to_float(v_row[d]), acc[i]);
            }
        }
    }
    if (PARTS > 1) {
#pragma unroll
        for (int i = 0; i < DIMS_PER_LANE; ++i)
            if (lane + 32 * i < HD) part_acc[warp][lane + 32 * i] = acc[i];
        if (lane == 0) { part_max[warp] = running_max; part_sum[warp] = running_sum; }
        __syncthreads();
        if (warp > 0) return;
        // (a part without keys, or with scores of -infinity alone, weighs exp(-inf) = 0)
        const float own_max = lane < PARTS ? part_max[lane] : -INFINITY;
        const float top = warp_max(own_max);
        const float weight = expf(own_max - top);
        running_sum = warp_sum(lane < PARTS ? part_sum[lane] * weight : 0.0f);
#pragma unroll
        for (int i = 0; i < DIMS_PER_LANE; ++i) acc[i] = 0.0f;
#pragma unroll
        for (int part = 0; part < PARTS; ++part) {
            const float scale_part = __shfl_sync(0xffffffffu, weight, part);
#pragma unroll
            for (int i = 0; i < DIMS_PER_LANE; ++i)
                if (lane + 32 * i < HD) acc[i] = fmaf(scale_part, part_acc[part][lane + 32 * i], acc[i]);
        }
    }
    T* out_row = out + ((size_t)t * num_heads + head) * HD;
    const float inverse = 1.0f / running_sum;
#pragma unroll
    for (int i = 0; i < DIMS_PER_LANE; ++i) {
        const int d = lane + 32 * i;
        if (d < HD) out_row[d] = from_float<T>(acc[i] * inverse);
    }
}

}  // namespace skv

using namespace skv;

SKV_EXPORT int skv_library_head_dim() { return SKV_HEAD_DIM; }

SKV_EXPORT int skv_attention(const void* q, const void* k_cache, const void* v_cache, const int* block_table,
                             int table_width, const int* positions, const int* token_seq, void* out,
                             int n_tokens, int num_heads, int num_kv_heads, int head_dim, int block_size,
                             float scale, int window, cudaStream_t stream) {
    if (n_tokens <= 0) return 0;
    if (head_dim != HD) return fail("skv_attention", "this library was built for another head size");
    if (num_heads <= 0 || num_kv_heads <= 0 || num_heads % num_kv_heads != 0)
        return fail("skv_attention", "heads must be a positive multiple of kv heads");
    if (block_size <= 0 || window < 0) return fail("skv_attention", "bad block size or window");
    const long long items = (long long)n_tokens * num_heads;
    if (items > 0x7fffffffLL) return fail("skv_attention", "too many tokens in one step");
    // while a warp each leaves the GPU's 64 warps an SM idle, eight or four warps share a (token, head)
    const int parts = items * 8 <= (long long)sm_count() * 64 ? 8 : items * 4 <= (long long)sm_count() * 64 ? 4 : 1;
    const long long blocks = parts > 1 ? items : (items + ATT_WARPS - 1) / ATT_WARPS;
    auto kernel = parts == 8 ? attention_kernel<skv_t, 8> : parts == 4 ? attention_kernel<skv_t, 4> : attention_kernel<skv_t, 1>;
    return launch_pdl("skv_attention", kernel, dim3((unsigned)blocks), dim3((parts > 1 ? parts : ATT_WARPS) * 32), 0,
                      stream, (const skv_t*)q, (const skv_t*)k_cache, (const skv_t*)v_cache, block_table,
                      table_width, positions, token_seq, (skv_t*)out, n_tokens, num_heads, num_kv_heads,
                      block_size, scale, window);
}
