// What follows the fused projection of a latent-attention layer whose queries and keys have a rotated part.
//
// A float row of the projection holds, per head, `dim` unrotated and `rope_dim` rotated query numbers, and (for a layer
// with a cache of its own, at latent_offset) `latent_dim` numbers of the compressed vector and `rope_dim` numbers of
// the one key part that all heads share.  Per token, a block
//   - copies the unrotated query parts to q_plain [tokens, heads * dim] (the keys' up-projection is folded into them
//     by the per-head product that follows),
//   - rotates the rotated query parts and puts them behind the (not yet written) folded part of every head of
//     q_folded [tokens, heads * (latent_dim + rope_dim)]
//     (or, where the step makes every head's keys instead of folding: both parts, head by head, to
//     q_whole [tokens, heads * (dim + rope_dim)], and nothing to the other two),
//   - divides the compressed vector by its root mean square, multiplies by the norm's weight, rotates the key part,
//     and writes both into the token's row of the paged cache [blocks][1][block_size][latent_dim + rope_dim].
// Rotation: of the first `rotated` numbers of a part, number i is paired with number i + rotated/2;
// (u, v) -> (u cos - v sin, v cos + u sin) with (cos, sin) = table[position][i].  Float math; the outputs are rounded
// to the compute dtype.
#include "common.cuh"

namespace skv {

constexpr int LATENT_FINISH_THREADS = 256;

// The value of number r of a part x after the rotation (r < part width).
__device__ __forceinline__ float turned(const float* x, int r, int rotated, const float* cos_sin) {
    if (r >= rotated) return x[r];
    const int half = rotated >> 1;
    if (r < half) return x[r] * cos_sin[2 * r] - x[r + half] * cos_sin[2 * r + 1];
    const int i = r - half;
    return x[r] * cos_sin[2 * i] + x[i] * cos_sin[2 * i + 1];
}

template <typename T>
__global__ void __launch_bounds__(LATENT_FINISH_THREADS)
latent_finish_kernel(const float* __restrict__ fused, int row_stride, T* __restrict__ q_plain, T* __restrict__ q_folded,
                     T* __restrict__ q_whole, T* __restrict__ cache, const int* __restrict__ positions, const int* __restrict__ token_seq,
                     const int* __restrict__ block_table, int table_width, int heads, int dim, int rope_dim,
                     int latent_dim, int block_size, const float* __restrict__ rotation, int rotated, int table_len,
                     int latent_offset, const float* __restrict__ latent_gamma, float eps, int write_cache) {
    __shared__ float reduce[33];
    pdl_launch_dependents();
    pdl_wait();
    const int t = blockIdx.x;
    const float* row = fused + (size_t)t * row_stride;
    const int pos = positions[t];
    const float* cos_sin = rotation ? rotation + (size_t)min(pos, table_len - 1) * rotated : nullptr;
    const int turn = rotation ? rotated : 0;
    const int q_head = dim + rope_dim, key_dim = latent_dim + rope_dim;
    for (int idx = threadIdx.x; idx < heads * q_head; idx += LATENT_FINISH_THREADS) {
        const int head = idx / q_head, j = idx - head * q_head;
        const float value = j < dim ? row[idx] : turned(row + (size_t)head * q_head + dim, j - dim, turn, cos_sin);
        if (q_whole) q_whole[(size_t)t * heads * q_head + idx] = from_float<T>(value);
        else if (j < dim) q_plain[((size_t)t * heads + head) * dim + j] = from_float<T>(value);
        else q_folded[((size_t)t * heads + head) * key_dim + latent_dim + (j - dim)] = from_float<T>(value);
    }
    if (!write_cache) return;
    const float* latent = row + latent_offset;
    float squares = 0.0f;
    for (int j = threadIdx.x; j < latent_dim; j += LATENT_FINISH_THREADS) squares = fmaf(latent[j], latent[j], squares);
    const float factor = 1.0f / sqrtf(block_sum(squares, reduce) / (float)latent_dim + eps);
    const int block = block_table[(size_t)token_seq[t] * table_width + pos / block_size];
    T* out = cache + ((size_t)block * block_size + pos % block_size) * key_dim;
    for (int j = threadIdx.x; j < key_dim; j += LATENT_FINISH_THREADS) {
        const float value = j < latent_dim ? latent[j] * factor * latent_gamma[j]
                                           : turned(latent + latent_dim, j - latent_dim, turn, cos_sin);
        out[j] = from_float<T>(value);
    }
}

// The same four neighbouring numbers a thread (every size and half the rotated part multiples of 4, rows 16-byte aligned), a
// token's queries in slices where tokens are few: a block of them is a chain of waits, not work.  With more than one slice the last
// one is the latent's.  32 heads of 48 + 16 over a latent of 256, 8 / 500 / 5,180 tokens: 7.2 / 10.5 / 62 us above, 2.1 / 5.0 / 36 here.
__device__ __forceinline__ void store_quad(float* p, float4 v) { *(float4*)p = v; }
__device__ __forceinline__ void store_quad(__nv_bfloat16* p, float4 v) {
    const __nv_bfloat162 lo = __floats2bfloat162_rn(v.x, v.y), hi = __floats2bfloat162_rn(v.z, v.w);
    *(uint2*)p = make_uint2(*(const uint32_t*)&lo, *(const uint32_t*)&hi);
}

// Numbers r .. r + 3 of a part x after the rotation.
__device__ __forceinline__ float4 turned_quad(const float* x, int r, int rotated, const float* cos_sin) {
    const float4 a = *(const float4*)(x + r);
    if (r >= rotated) return a;
    const int half = rotated >> 1;
    const bool lower = r < half;
    const int i = lower ? r : r - half;
    const float4 b = *(const float4*)(x + (lower ? r + half : i));
    const float4 c0 = *(const float4*)(cos_sin + 2 * i), c1 = *(const float4*)(cos_sin + 2 * i + 4);
    const float sign = lower ? -1.0f : 1.0f;
    return make_float4(a.x * c0.x + sign * (b.x * c0.y), a.y * c0.z + sign * (b.y * c0.w), a.z * c1.x + sign * (b.z * c1.y),
                       a.w * c1.z + sign * (b.w * c1.w));
}

template <typename T>
__global__ void __launch_bounds__(LATENT_FINISH_THREADS)
latent_finish_wide_kernel(const float* __restrict__ fused, int row_stride, T* __restrict__ q_plain, T* __restrict__ q_folded,
                          T* __restrict__ q_whole, T* __restrict__ cache, const int* __restrict__ positions, const int* __restrict__ token_seq,
                          const int* __restrict__ block_table, int table_width, int heads, int dim, int rope_dim,
                          int latent_dim, int block_size, const float* __restrict__ rotation, int rotated, int table_len,
                          int latent_offset, const float* __restrict__ latent_gamma, float eps, int write_cache, int q_slices) {
    __shared__ float reduce[33];
    const int c0 = 4 * threadIdx.x;
    float4 gamma = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    if (write_cache && c0 < latent_dim) gamma = *(const float4*)(latent_gamma + c0);
    pdl_launch_dependents();
    pdl_wait();
    const int t = blockIdx.x, slice = blockIdx.y;
    const float* row = fused + (size_t)t * row_stride;
    const int pos = positions[t];
    const float* cos_sin = rotation ? rotation + (size_t)min(pos, table_len - 1) * rotated : nullptr;
    const int turn = rotation ? rotated : 0;
    const int q_head = dim + rope_dim, key_dim = latent_dim + rope_dim;
    if (slice < q_slices) {
        for (int idx = 4 * (slice * LATENT_FINISH_THREADS + threadIdx.x); idx < heads * q_head; idx += 4 * q_slices * LATENT_FINISH_THREADS) {
            const int head = idx / q_head, j = idx - head * q_head;
            const float4 value = j < dim ? *(const float4*)(row + idx) : turned_quad(row + (size_t)head * q_head + dim, j - dim, turn, cos_sin);
            T* to = q_whole ? q_whole + (size_t)t * heads * q_head + idx
                  : j < dim ? q_plain + ((size_t)t * heads + head) * dim + j
                            : q_folded + ((size_t)t * heads + head) * key_dim + latent_dim + (j - dim);
            store_quad(to, value);
        }
    }
    if (!write_cache || slice != (int)gridDim.y - 1) return;
    const float* latent = row + latent_offset;
    float4 own = c0 < key_dim ? *(const float4*)(latent + c0) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    const int block = block_table[(size_t)token_seq[t] * table_width + pos / block_size];
    float squares = 0.0f;
    for (int j = c0; j < latent_dim; j += 4 * LATENT_FINISH_THREADS) {
        const float4 v = j == c0 ? own : *(const float4*)(latent + j);
        squares = fmaf(v.x, v.x, fmaf(v.y, v.y, fmaf(v.z, v.z, fmaf(v.w, v.w, squares))));
    }
    const float factor = 1.0f / sqrtf(block_sum(squares, reduce) / (float)latent_dim + eps);
    T* out = cache + ((size_t)block * block_size + pos % block_size) * key_dim;
    for (int j = c0; j < key_dim; j += 4 * LATENT_FINISH_THREADS) {
        if (j < latent_dim) {
            if (j != c0) { own = *(const float4*)(latent + j); gamma = *(const float4*)(latent_gamma + j); }
            store_quad(out + j, make_float4(own.x * factor * gamma.x, own.y * factor * gamma.y, own.z * factor * gamma.z, own.w * factor * gamma.w));
        } else {
            store_quad(out + j, turned_quad(latent + latent_dim, j - latent_dim, turn, cos_sin));
        }
    }
}

}  // namespace skv

using namespace skv;

// q_whole: null, or the one place for the queries (then q_plain and q_folded may be null).
// rotation: float [table_len][rotated / 2][2] or null (then nothing is rotated).  With write_cache 0 a row need hold
// its queries only, and latent_gamma may be null.
SKV_EXPORT int skv_latent_finish(const float* fused, int row_stride, void* q_plain, void* q_folded, void* q_whole, void* cache,
                                 const int* positions, const int* token_seq, const int* block_table, int table_width,
                                 int n_tokens, int heads, int dim, int rope_dim, int latent_dim, int block_size,
                                 const float* rotation, int rotated, int table_len, int latent_offset,
                                 const float* latent_gamma, float eps, int write_cache, cudaStream_t stream) {
    if (n_tokens <= 0) return 0;
    if (heads <= 0 || dim <= 0 || rope_dim < 0 || latent_dim <= 0 || block_size <= 0)
        return fail("skv_latent_finish", "head count, sizes and block_size must be positive");
    if (rotation && (rotated <= 0 || rotated % 2 || rotated > rope_dim || table_len <= 0))
        return fail("skv_latent_finish", "the rotated numbers must be an even count within the rotated part");
    if (!fused || (!q_whole && (!q_plain || !q_folded)))
        return fail("skv_latent_finish", "a place for the queries is needed: the two parts apart, or whole heads");
    if (write_cache && (!latent_gamma || !cache || latent_offset < heads * (dim + rope_dim)))
        return fail("skv_latent_finish", "a cache write needs the cache, the latent's norm weight and the latent behind the queries");
    if (row_stride < (write_cache ? latent_offset + latent_dim + rope_dim : heads * (dim + rope_dim)))
        return fail("skv_latent_finish", "a row is shorter than its queries, latent and key part");
    const int sizes = dim | rope_dim | latent_dim | row_stride | latent_offset | (rotation ? rotated / 2 : 0);
    const uintptr_t places = (uintptr_t)fused | (uintptr_t)q_plain | (uintptr_t)q_folded | (uintptr_t)q_whole | (uintptr_t)cache |
                             (uintptr_t)rotation | (uintptr_t)latent_gamma;
    if (sizes % 4 == 0 && (places & 15) == 0) {
        // a token's queries in one block once the tokens fill the GPU
        const int quads = heads * (dim + rope_dim) / 4, most = (quads + LATENT_FINISH_THREADS - 1) / LATENT_FINISH_THREADS;
        const int slices = n_tokens >= 2 * sm_count() ? 1 : most < 64 ? most : 64;
        return launch_pdl("skv_latent_finish", latent_finish_wide_kernel<skv_t>, dim3(n_tokens, slices + (slices > 1 && write_cache)),
                          dim3(LATENT_FINISH_THREADS), 0, stream, fused, row_stride, (skv_t*)q_plain, (skv_t*)q_folded, (skv_t*)q_whole,
                          (skv_t*)cache, positions, token_seq, block_table, table_width, heads, dim, rope_dim, latent_dim, block_size,
                          rotation, rotation ? rotated : 0, table_len, latent_offset, latent_gamma, eps, write_cache, slices);
    }
    return launch_pdl("skv_latent_finish", latent_finish_kernel<skv_t>, dim3(n_tokens), dim3(LATENT_FINISH_THREADS), 0,
                      stream, fused, row_stride, (skv_t*)q_plain, (skv_t*)q_folded, (skv_t*)q_whole, (skv_t*)cache, positions, token_seq,
                      block_table, table_width, heads, dim, rope_dim, latent_dim, block_size, rotation,
                      rotation ? rotated : 0, table_len, latent_offset, latent_gamma, eps, write_cache);
}
