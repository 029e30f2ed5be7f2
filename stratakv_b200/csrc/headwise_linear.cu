// A projection with a matrix of its own for every head (or every equal part of the channels):
//
//   out[t, h, o] = sum_i w[h, o, i] * x[t, h, i]          w [heads, out_dim, in_dim] in the compute dtype
//
// x rows are x_stride apart and out rows out_stride apart, head h starting at h * in_dim and h * out_dim; either may
// be float or the compute dtype.  Sums are float and a float input, a gate of a recurrence for instance, is never
// rounded: the float32 build is FMA throughout, the bfloat16 build has a tensor-core form that keeps floats whole.
// Used for block-diagonal gates and for the two per-head products that fold a latent's up-projections into queries and
// outputs.
#include "common.cuh"

namespace skv {

constexpr int HW_TOKENS = 32, HW_OUTS = 64, HW_K = 32;

template <typename TIn, typename TOut, typename TW>
__global__ void __launch_bounds__(256)
headwise_linear_kernel(const TIn* __restrict__ x, int x_stride, const TW* __restrict__ w, TOut* __restrict__ out,
                       int out_stride, int n_tokens, int in_dim, int out_dim, int zero_pad, int out_head_stride) {
    __shared__ float xs[HW_TOKENS][HW_K + 1];
    __shared__ float ws[HW_OUTS][HW_K + 1];
    pdl_launch_dependents();
    pdl_wait();
    const int head = blockIdx.z, t0 = blockIdx.y * HW_TOKENS, o0 = blockIdx.x * HW_OUTS;
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;       // outputs tx, tx + 16, tx + 32, tx + 48; tokens ty, ty + 16
    const TIn* x_head = x + (size_t)head * in_dim;
    const TW* w_head = w + (size_t)head * out_dim * in_dim;
    float acc[2][4] = {};
    for (int k0 = 0; k0 < in_dim; k0 += HW_K) {
        for (int idx = threadIdx.x; idx < HW_TOKENS * HW_K; idx += 256) {
            const int row = idx / HW_K, k = idx % HW_K;
            const int t = t0 + row;
            xs[row][k] = t < n_tokens && k0 + k < in_dim ? to_float(x_head[(size_t)t * x_stride + k0 + k]) : 0.0f;
        }
        for (int idx = threadIdx.x; idx < HW_OUTS * HW_K; idx += 256) {
            const int row = idx / HW_K, k = idx % HW_K;
            const int o = o0 + row;
            ws[row][k] = o < out_dim && k0 + k < in_dim ? to_float(w_head[(size_t)o * in_dim + k0 + k]) : 0.0f;
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < HW_K; ++k) {
            const float a0 = xs[ty][k], a1 = xs[ty + 16][k];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const float b = ws[tx + 16 * j][k];
                acc[0][j] = fmaf(a0, b, acc[0][j]);
                acc[1][j] = fmaf(a1, b, acc[1][j]);
            }
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        const int t = t0 + ty + 16 * i;
        if (t >= n_tokens) continue;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int o = o0 + tx + 16 * j;
            if (o < out_dim) out[(size_t)t * out_stride + (size_t)head * out_head_stride + o] = from_float<TOut>(acc[i][j]);
        }
    }
    // columns that pad a row for the projection after it are zero
    if (zero_pad && head == (int)gridDim.z - 1 && blockIdx.x == 0) {
        const int first = (int)gridDim.z * out_dim, pad = out_stride - first;
        for (int idx = threadIdx.x; idx < HW_TOKENS * pad; idx += 256) {
            const int t = t0 + idx / pad;
            if (t < n_tokens) out[(size_t)t * out_stride + first + idx % pad] = from_float<TOut>(0.0f);
        }
    }
}

#if SKV_DTYPE == SKV_BF16
// The same on tensor cores (mma.sync m16n8k16), for weights whose rows are whole 16 bytes: a warp makes 16 tokens x 8 NT
// outputs of a head.  A lane reads eight neighbouring k of a row at a time, in the same order for both operands.  A float
// input stays float: it is split into three bfloat16 that add up to it (24 of 24 bits), against weights that are
// bfloat16 anyway, so every product is exact and the sums are float (mma_bf16_add: relative errors over an inner size of 256 of
// 0.8e-7 to 0.9e-7 of a float input and 0.7e-7 of a bfloat16 one, where the FMA kernel's are 2.5e-7 to 2.9e-7 and 1.1e-7 to 1.5e-7
// and sums left in the tensor core had up to 8.5e-7; that costs 0 to 10 % of a prompt's time and nothing of a few tokens').
// A step of few tokens is bound by latency (a matrix of a MB over all heads): NT 2 gives warps enough, and the first
// weights are under way before the wait.  A prompt is bound by the rows it reads and writes: NT 8 reads a float row once
// per 64 outputs.  32 heads 64 -> 256 at 8 and 3,764 tokens: 6.2 -> 1.6 us and 216 -> 49; 256 -> 64: 17.7 -> 3.1 us and
// 219 -> 37; float to float 64 -> 64: 5.1 -> 2.1 us and 57 -> 18.
constexpr int HM_WARPS = 4;

// Eight numbers of a row as operand pairs: parts[s][i] holds numbers 2i and 2i + 1 (of a float row its s-th bfloat16).
__device__ __forceinline__ void headwise_parts(const __nv_bfloat16* p, bool live, uint32_t (&parts)[1][4]) {
    const uint4 v = live ? *(const uint4*)p : make_uint4(0u, 0u, 0u, 0u);
    parts[0][0] = v.x; parts[0][1] = v.y; parts[0][2] = v.z; parts[0][3] = v.w;
}
__device__ __forceinline__ void headwise_parts(const float* p, bool live, uint32_t (&parts)[3][4]) {
    const float4 zero = make_float4(0.0f, 0.0f, 0.0f, 0.0f), lo = live ? *(const float4*)p : zero, hi = live ? *(const float4*)(p + 4) : zero;
    const float v[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        uint32_t pair[3];
        split3(v[2 * i], v[2 * i + 1], pair);
#pragma unroll
        for (int s = 0; s < 3; ++s) parts[s][i] = pair[s];
    }
}

__device__ __forceinline__ void headwise_store(float* p, float u, float v) { *(float2*)p = make_float2(u, v); }
__device__ __forceinline__ void headwise_store(__nv_bfloat16* p, float u, float v) { *(__nv_bfloat162*)p = __floats2bfloat162_rn(u, v); }

template <typename TIn, typename TOut, int NT>
__global__ void __launch_bounds__(HM_WARPS * 32)
headwise_mma_kernel(const TIn* __restrict__ x, int x_stride, const __nv_bfloat16* __restrict__ w, TOut* __restrict__ out,
                    int out_stride, int n_tokens, int in_dim, int out_dim, int zero_pad, int out_head_stride, int paired) {
    constexpr int PARTS = sizeof(TIn) == 4 ? 3 : 1;
    const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3, head = blockIdx.z;
    const int out_groups = (out_dim + 8 * NT - 1) / (8 * NT);
    const int work = blockIdx.x * HM_WARPS + (threadIdx.x >> 5);
    const int o0 = work % out_groups * 8 * NT, t0 = work / out_groups * 16;
    const __nv_bfloat16* w_rows[NT];
    uint4 weights[NT];
    auto load_weights = [&](int k) {
#pragma unroll
        for (int n = 0; n < NT; ++n) weights[n] = k < in_dim ? *(const uint4*)(w_rows[n] + k) : make_uint4(0u, 0u, 0u, 0u);
    };
#pragma unroll
    for (int n = 0; n < NT; ++n) w_rows[n] = w + ((size_t)head * out_dim + min(o0 + 8 * n + g, out_dim - 1)) * in_dim;
    load_weights(8 * t);
    pdl_launch_dependents();
    pdl_wait();
    if (t0 >= n_tokens) return;
    const TIn* rows[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) rows[h] = x + (size_t)min(t0 + 8 * h + g, n_tokens - 1) * x_stride + (size_t)head * in_dim;
    float acc[NT][4] = {};
    for (int k0 = 0; k0 < in_dim; k0 += 32) {
        const int k = k0 + 8 * t;
        uint32_t a[2][PARTS][4];
#pragma unroll
        for (int h = 0; h < 2; ++h) headwise_parts(rows[h] + k, k < in_dim, a[h]);
        if (k0 > 0) load_weights(k);
        uint32_t first[PARTS][4], second[PARTS][4];
#pragma unroll
        for (int s = 0; s < PARTS; ++s)
#pragma unroll
            for (int i = 0; i < 4; ++i) { first[s][i] = a[i & 1][s][i >> 1]; second[s][i] = a[i & 1][s][2 + (i >> 1)]; }
#pragma unroll
        for (int n = 0; n < NT; ++n) {
            mma_bf16_add<PARTS>(acc[n], first, weights[n].x, weights[n].y);
            mma_bf16_add<PARTS>(acc[n], second, weights[n].z, weights[n].w);
        }
    }
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const int token = t0 + 8 * h + g;
        if (token >= n_tokens) continue;
        TOut* row = out + (size_t)token * out_stride + (size_t)head * out_head_stride;
#pragma unroll
        for (int n = 0; n < NT; ++n) {
            const int o = o0 + 8 * n + 2 * t;
            if (paired && o + 1 < out_dim) {
                headwise_store(row + o, acc[n][2 * h], acc[n][2 * h + 1]);
            } else {
                if (o < out_dim) row[o] = from_float<TOut>(acc[n][2 * h]);
                if (o + 1 < out_dim) row[o + 1] = from_float<TOut>(acc[n][2 * h + 1]);
            }
        }
    }
    // columns that pad a row for the projection after it are zero
    if (zero_pad && head == (int)gridDim.z - 1 && o0 == 0) {
        const int first = (int)gridDim.z * out_dim, pad = out_stride - first;
        for (int i = lane; i < 16 * pad; i += 32)
            if (t0 + i / pad < n_tokens) out[(size_t)(t0 + i / pad) * out_stride + first + i % pad] = from_float<TOut>(0.0f);
    }
}

template <typename TIn, typename TOut, int NT>
static int launch_headwise_mma(const void* x, int x_stride, const void* w, void* out, int out_stride, int n_tokens,
                               int heads, int in_dim, int out_dim, int zero_pad, int out_head_stride, cudaStream_t stream) {
    const long long work = (long long)((out_dim + 8 * NT - 1) / (8 * NT)) * ((n_tokens + 15) / 16);
    const long long blocks = (work + HM_WARPS - 1) / HM_WARPS;
    if (blocks > 0x7fffffffLL) return fail("skv_headwise_linear", "too many tokens for one launch");
    const int paired = out_stride % 2 == 0 && out_head_stride % 2 == 0 && ((uintptr_t)out & (2 * sizeof(TOut) - 1)) == 0;
    return launch_pdl("skv_headwise_linear", headwise_mma_kernel<TIn, TOut, NT>, dim3((unsigned)blocks, 1, heads), dim3(HM_WARPS * 32), 0,
                      stream, (const TIn*)x, x_stride, (const __nv_bfloat16*)w, (TOut*)out, out_stride, n_tokens, in_dim, out_dim,
                      zero_pad, out_head_stride, paired);
}
#endif

template <typename TIn, typename TOut>
static int launch_headwise(const void* x, int x_stride, const void* w, void* out, int out_stride, int n_tokens,
                           int heads, int in_dim, int out_dim, int zero_pad, int out_head_stride, cudaStream_t stream) {
#if SKV_DTYPE == SKV_BF16
    // rows of whole 16 bytes on both sides; few tokens (a tile or four of them) take the form with more warps
    if (in_dim % 8 == 0 && (x_stride * sizeof(TIn)) % 16 == 0 && (((uintptr_t)x | (uintptr_t)w) & 15) == 0) {
        if (n_tokens <= 64 || out_dim <= 16)
            return launch_headwise_mma<TIn, TOut, 2>(x, x_stride, w, out, out_stride, n_tokens, heads, in_dim, out_dim, zero_pad, out_head_stride, stream);
        return launch_headwise_mma<TIn, TOut, 8>(x, x_stride, w, out, out_stride, n_tokens, heads, in_dim, out_dim, zero_pad, out_head_stride, stream);
    }
#endif
    const dim3 grid((out_dim + HW_OUTS - 1) / HW_OUTS, (n_tokens + HW_TOKENS - 1) / HW_TOKENS, heads);
    return launch_pdl("skv_headwise_linear", headwise_linear_kernel<TIn, TOut, skv_t>, grid, dim3(256), 0, stream,
                      (const TIn*)x, x_stride, (const skv_t*)w, (TOut*)out, out_stride, n_tokens, in_dim, out_dim, zero_pad,
                      out_head_stride);
}

}  // namespace skv

using namespace skv;

// out_head_stride: head h of an out row starts at h * out_head_stride (0: out_dim, the heads side by side).
// x_is_float / out_is_float: 1 for float, 0 for the compute dtype.  zero_pad: the columns of an out row beyond its
// heads are set to zero.
SKV_EXPORT int skv_headwise_linear(const void* x, int x_is_float, int x_stride, const void* w, void* out,
                                   int out_is_float, int out_stride, int n_tokens, int heads, int in_dim, int out_dim,
                                   int zero_pad, int out_head_stride, cudaStream_t stream) {
    if (n_tokens <= 0) return 0;
    if (heads <= 0 || in_dim <= 0 || out_dim <= 0) return fail("skv_headwise_linear", "sizes must be positive");
    if (heads > 65535 || (n_tokens + HW_TOKENS - 1) / HW_TOKENS > 65535)
        return fail("skv_headwise_linear", "too many heads or tokens for one launch");
    if (out_head_stride <= 0) out_head_stride = out_dim;
    if (x_stride < heads * in_dim || out_head_stride < out_dim || out_stride < (heads - 1) * out_head_stride + out_dim)
        return fail("skv_headwise_linear", "a row is shorter than its heads");
    if (zero_pad && out_head_stride != out_dim)
        return fail("skv_headwise_linear", "zero_pad goes with heads that lie side by side");
    if (x_is_float && out_is_float)
        return launch_headwise<float, float>(x, x_stride, w, out, out_stride, n_tokens, heads, in_dim, out_dim, zero_pad, out_head_stride, stream);
    if (x_is_float)
        return launch_headwise<float, skv_t>(x, x_stride, w, out, out_stride, n_tokens, heads, in_dim, out_dim, zero_pad, out_head_stride, stream);
    if (out_is_float)
        return launch_headwise<skv_t, float>(x, x_stride, w, out, out_stride, n_tokens, heads, in_dim, out_dim, zero_pad, out_head_stride, stream);
    return launch_headwise<skv_t, skv_t>(x, x_stride, w, out, out_stride, n_tokens, heads, in_dim, out_dim, zero_pad, out_head_stride, stream);
}
