// Kernels on the float residual stream for layers that norm a sublayer's output before it is added, and for a
// per-layer input that depends on the token:
//
//   rmsnorm_add:  x[r, :] += y[r, :] / sqrt(mean(y[r, :]^2) + eps) * gamma          (the norm after a sublayer)
//   token_side:   e = table[token, offset : offset + dim];  g = gelu_tanh(gate_w . x) * e;  y = proj_w . g;
//                 x += y / sqrt(mean(y^2) + eps) * norm_w                            (dim is small: tens)
//
// Both can hand the next reader its input in the same pass: with next_out, the new row of the stream is normed
// with next_gamma and next_eps and written in the compute dtype, so the norm in front of the next sublayer needs no
// kernel of its own; rmsnorm_add without next_gamma writes the new row as it is, for sublayers that read the stream itself.  Everything is float but the tables and weights, which are read in the compute dtype.
#include "common.cuh"

namespace skv {

template <typename T>
__global__ void rmsnorm_add_kernel(const float* __restrict__ y, const float* __restrict__ gamma, float eps,
                                   float* __restrict__ x, const float* __restrict__ next_gamma, float next_eps,
                                   T* __restrict__ next_out, int hidden) {
    __shared__ float scratch[33];
    pdl_launch_dependents();
    pdl_wait();
    const size_t r = blockIdx.x;
    const float* y_row = y + r * hidden;
    float* x_row = x + r * hidden;
    float partial = 0.0f;
    for (int c = threadIdx.x; c < hidden; c += blockDim.x) {
        const float v = y_row[c];
        partial = fmaf(v, v, partial);
    }
    const float inverse_rms = 1.0f / sqrtf(block_sum(partial, scratch) / (float)hidden + eps);
    float squares = 0.0f;
    for (int c = threadIdx.x; c < hidden; c += blockDim.x) {
        const float v = x_row[c] + y_row[c] * inverse_rms * gamma[c];
        x_row[c] = v;
        squares = fmaf(v, v, squares);
    }
    if (!next_out) return;
    T* out_row = next_out + r * hidden;
    if (!next_gamma) {
        for (int c = threadIdx.x; c < hidden; c += blockDim.x) out_row[c] = from_float<T>(x_row[c]);
        return;
    }
    const float next_inverse = 1.0f / sqrtf(block_sum(squares, scratch) / (float)hidden + next_eps);
    for (int c = threadIdx.x; c < hidden; c += blockDim.x)     // (each thread reads back what it wrote itself)
        out_row[c] = from_float<T>(x_row[c] * next_inverse * next_gamma[c]);
}

// The same with the row held in registers (hidden a multiple of 4, at most 4 * VEC * blockDim, 16-byte aligned rows):
// a thread keeps VEC float4 of the branch and of the stream, so memory is read once and written once.
template <typename T, int VEC>
__global__ void rmsnorm_add_rows_kernel(const float* __restrict__ y, const float* __restrict__ gamma, float eps,
                                        float* __restrict__ x, const float* __restrict__ next_gamma, float next_eps,
                                        T* __restrict__ next_out, int hidden) {
    __shared__ float scratch[33];
    pdl_launch_dependents();
    pdl_wait();
    const size_t r = blockIdx.x;
    const float4* y_row = (const float4*)(y + r * hidden);
    float4* x_row = (float4*)(x + r * hidden);
    const int quads = hidden >> 2;
    float4 branch[VEC], stream[VEC];
    float partial = 0.0f;
#pragma unroll
    for (int u = 0; u < VEC; ++u) {
        const int i = threadIdx.x + u * blockDim.x;
        if (i < quads) {
            branch[u] = y_row[i];
            stream[u] = x_row[i];
            partial += branch[u].x * branch[u].x + branch[u].y * branch[u].y + branch[u].z * branch[u].z + branch[u].w * branch[u].w;
        }
    }
    const float inverse_rms = 1.0f / sqrtf(block_sum(partial, scratch) / (float)hidden + eps);
    float squares = 0.0f;
#pragma unroll
    for (int u = 0; u < VEC; ++u) {
        const int i = threadIdx.x + u * blockDim.x;
        if (i < quads) {
            const float4 g = ((const float4*)gamma)[i];
            stream[u].x += branch[u].x * inverse_rms * g.x; stream[u].y += branch[u].y * inverse_rms * g.y;
            stream[u].z += branch[u].z * inverse_rms * g.z; stream[u].w += branch[u].w * inverse_rms * g.w;
            x_row[i] = stream[u];
            squares += stream[u].x * stream[u].x + stream[u].y * stream[u].y + stream[u].z * stream[u].z + stream[u].w * stream[u].w;
        }
    }
    if (!next_out) return;
    T* out_row = next_out + r * hidden;
    const float next_inverse = next_gamma ? 1.0f / sqrtf(block_sum(squares, scratch) / (float)hidden + next_eps) : 1.0f;
#pragma unroll
    for (int u = 0; u < VEC; ++u) {
        const int i = threadIdx.x + u * blockDim.x;
        if (i < quads) {
            const float4 g = next_gamma ? ((const float4*)next_gamma)[i] : make_float4(1.0f, 1.0f, 1.0f, 1.0f);
            const float4 v = make_float4(stream[u].x * next_inverse * g.x, stream[u].y * next_inverse * g.y,
                                         stream[u].z * next_inverse * g.z, stream[u].w * next_inverse * g.w);
            if (sizeof(T) == 4) {
                *(float4*)(out_row + 4 * i) = v;
            } else {
                const __nv_bfloat162 lo = __floats2bfloat162_rn(v.x, v.y), hi = __floats2bfloat162_rn(v.z, v.w);
                *(uint2*)(out_row + 4 * i) = make_uint2(*(const uint32_t*)&lo, *(const uint32_t*)&hi);
            }
        }
    }
}

// Four neighbouring weights of a row as floats (the row 8-byte aligned at `p` for bfloat16, 16-byte for float).
__device__ __forceinline__ void load4(const float* p, float (&out)[4]) {
    const float4 v = *(const float4*)p;
    out[0] = v.x; out[1] = v.y; out[2] = v.z; out[3] = v.w;
}
__device__ __forceinline__ void load4(const __nv_bfloat16* p, float (&out)[4]) {
    const uint2 raw = *(const uint2*)p;
    const float2 lo = __bfloat1622float2(*(const __nv_bfloat162*)&raw.x), hi = __bfloat1622float2(*(const __nv_bfloat162*)&raw.y);
    out[0] = lo.x; out[1] = lo.y; out[2] = hi.x; out[3] = hi.y;
}

// A block takes TOK tokens, so that it reads the two weights once for all of them (one token a block where tokens are
// few, so that there are blocks enough).  `proj_t` is the projection transposed, [dim][hidden], which lets
// neighbouring threads read neighbouring columns.  VEC: hidden is a multiple of 4 and every row 16-byte aligned; a
// lane then takes four neighbouring columns at a time.  A warp works on four of the dim gate rows at once.
template <typename T, int TOK, bool VEC>
__global__ void __launch_bounds__(TOK == 1 ? 512 : 256) token_side_kernel(float* __restrict__ x, const int* __restrict__ ids, const T* __restrict__ table,
                                  int table_stride, int offset, int dim, int vocab, const T* __restrict__ gate_w,
                                  const T* __restrict__ proj_t, const float* __restrict__ norm_w, float eps,
                                  const float* __restrict__ next_gamma, float next_eps, T* __restrict__ next_out,
                                  int n_tokens, int hidden, const float* __restrict__ branch,
                                  const float* __restrict__ post_gamma, float post_eps) {
    extern __shared__ __align__(16) float side_shared[];       // [TOK][dim] gated values, [TOK][hidden] projected
    __shared__ float scratch[33];
    pdl_launch_dependents();
    pdl_wait();
    float* gated = side_shared;
    float* projected = side_shared + TOK * ((dim + 3) & ~3);
    const int t0 = blockIdx.x * TOK;
    const int count = min(TOK, n_tokens - t0);
    const float* rows[TOK];
#pragma unroll
    for (int k = 0; k < TOK; ++k) rows[k] = x + (size_t)(t0 + min(k, count - 1)) * hidden;
    if (branch) {
        // first the sublayer in front: x += rmsnorm(branch) * post_gamma on this block's rows (rmsnorm_add's work)
#pragma unroll
        for (int k = 0; k < TOK; ++k) {
            const float* y_row = branch + (size_t)(t0 + min(k, count - 1)) * hidden;
            float sum = 0.0f;
            for (int c = threadIdx.x; c < hidden; c += blockDim.x) sum = fmaf(y_row[c], y_row[c], sum);
            const float inverse = 1.0f / sqrtf(block_sum(sum, scratch) / (float)hidden + post_eps);
            if (k < count) {
                float* x_row = x + (size_t)(t0 + k) * hidden;
                for (int c = threadIdx.x; c < hidden; c += blockDim.x) x_row[c] += y_row[c] * inverse * post_gamma[c];
            }
        }
        __syncthreads();                                       // (the rows are read by other threads from here on)
    }
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, warps = blockDim.x >> 5;
    if (VEC) {
        // the block's rows of the stream go to shared memory once (the place of the projected values, which come
        // later), with every thread's loads in flight together; the gate rows then meet them there
        const int quads = hidden >> 2;
        for (int i = threadIdx.x; i < TOK * quads; i += blockDim.x) {
            const int k = i / quads, q4 = i - k * quads;
            ((float4*)projected)[i] = *(const float4*)(x + (size_t)(t0 + min(k, count - 1)) * hidden + 4 * q4);
        }
        __syncthreads();
    }
    for (int j0 = 4 * warp; j0 < dim; j0 += 4 * warps) {
        float dot[4][TOK] = {};
        const T* w_rows[4];
#pragma unroll
        for (int jj = 0; jj < 4; ++jj) w_rows[jj] = gate_w + (size_t)min(j0 + jj, dim - 1) * hidden;
        if (VEC) {
#pragma unroll 2
            for (int c = 4 * lane; c < hidden; c += 128) {
                float w[4][4];
#pragma unroll
                for (int jj = 0; jj < 4; ++jj) load4(w_rows[jj] + c, w[jj]);
#pragma unroll
                for (int k = 0; k < TOK; ++k) {
                    const float4 xs = *(const float4*)(projected + (size_t)k * hidden + c);
#pragma unroll
                    for (int jj = 0; jj < 4; ++jj)
                        dot[jj][k] += w[jj][0] * xs.x + w[jj][1] * xs.y + w[jj][2] * xs.z + w[jj][3] * xs.w;
                }
            }
        } else {
            for (int c = lane; c < hidden; c += 32) {
#pragma unroll
                for (int jj = 0; jj < 4; ++jj) {
                    const float w = to_float(w_rows[jj][c]);
#pragma unroll
                    for (int k = 0; k < TOK; ++k) dot[jj][k] = fmaf(w, rows[k][c], dot[jj][k]);
                }
            }
        }
#pragma unroll
        for (int jj = 0; jj < 4; ++jj) {
#pragma unroll
            for (int k = 0; k < TOK; ++k) {
                const float total = warp_sum(dot[jj][k]);
                if (lane == 0 && j0 + jj < dim) {
                    const int id = ids[t0 + min(k, count - 1)];
                    // (the embedding has flagged an id outside the table)
                    const bool known = id >= 0 && id < vocab;
                    gated[k * dim + j0 + jj] =
                        known ? gelu_tanh(total) * to_float(table[(size_t)id * table_stride + offset + j0 + jj]) : 0.0f;
                }
            }
        }
    }
    __syncthreads();
    float partial[TOK] = {};
    // four columns a thread at a time: a gated value is read from shared memory once for the four
    for (int c0 = threadIdx.x; c0 < hidden; c0 += 4 * blockDim.x) {
        float sum[4][TOK] = {};
        int cols[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) cols[i] = min(c0 + i * (int)blockDim.x, hidden - 1);
#pragma unroll 2
        for (int j = 0; j < dim; ++j) {
            float g[TOK];
#pragma unroll
            for (int k = 0; k < TOK; ++k) g[k] = gated[k * dim + j];
            const T* w_row = proj_t + (size_t)j * hidden;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const float w = to_float(w_row[cols[i]]);
#pragma unroll
                for (int k = 0; k < TOK; ++k) sum[i][k] = fmaf(w, g[k], sum[i][k]);
            }
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int c = c0 + i * (int)blockDim.x;
            if (c >= hidden) continue;
#pragma unroll
            for (int k = 0; k < TOK; ++k) {
                projected[(size_t)k * hidden + c] = sum[i][k];
                partial[k] = fmaf(sum[i][k], sum[i][k], partial[k]);
            }
        }
    }
    float inverse_rms[TOK];
#pragma unroll
    for (int k = 0; k < TOK; ++k) inverse_rms[k] = 1.0f / sqrtf(block_sum(partial[k], scratch) / (float)hidden + eps);
    float squares[TOK] = {};
#pragma unroll
    for (int k = 0; k < TOK; ++k) {
        if (k >= count) continue;
        float* x_row = x + (size_t)(t0 + k) * hidden;
        for (int c = threadIdx.x; c < hidden; c += blockDim.x) {
            const float v = x_row[c] + projected[(size_t)k * hidden + c] * inverse_rms[k] * norm_w[c];
            x_row[c] = v;
            squares[k] = fmaf(v, v, squares[k]);
        }
    }
    if (!next_out) return;
#pragma unroll
    for (int k = 0; k < TOK; ++k) {
        const float next_inverse = 1.0f / sqrtf(block_sum(squares[k], scratch) / (float)hidden + next_eps);
        if (k >= count) continue;
        const float* x_row = x + (size_t)(t0 + k) * hidden;
        T* out_row = next_out + (size_t)(t0 + k) * hidden;
        for (int c = threadIdx.x; c < hidden; c += blockDim.x)     // (each thread reads back what it wrote itself)
            out_row[c] = from_float<T>(x_row[c] * next_inverse * next_gamma[c]);
    }
}

template <int TOK, bool VEC>
static int launch_token_side(float* x, const int* ids, const void* table, int table_stride, int offset, int dim,
                             int vocab, const void* gate_w, const void* proj_t, const float* norm_w, float eps,
                             const float* next_gamma, float next_eps, void* next_out, int n_tokens, int hidden,
                             const float* branch, const float* post_gamma, float post_eps, int threads,
                             cudaStream_t stream) {
    const size_t smem = (size_t)TOK * (((dim + 3) & ~3) + hidden) * sizeof(float);
    auto kernel = token_side_kernel<skv_t, TOK, VEC>;
    if (smem > 48 * 1024) {
        static bool raised = false;
        if (!raised) {
            if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024) != cudaSuccess)
                return fail("skv_token_side", "cannot raise the shared-memory limit");
            raised = true;
        }
    }
    return launch_pdl("skv_token_side", kernel, dim3((n_tokens + TOK - 1) / TOK), dim3(threads), smem, stream, x, ids,
                      (const skv_t*)table, table_stride, offset, dim, vocab, (const skv_t*)gate_w, (const skv_t*)proj_t,
                      norm_w, eps, next_gamma, next_eps, (skv_t*)next_out, n_tokens, hidden, branch, post_gamma, post_eps);
}

#if SKV_DTYPE == SKV_BF16
// The token input on tensor cores.  Both products are small (dim x hidden and back) but every token needs all of both
// weights, which is what bounds them: a cluster takes 16 * MT tokens and shares the columns of the stream, eight warps
// a block and COLS columns a warp, so the weights are read once per 16 or 32 tokens and a token's chain of loads is short.
//   gate: a warp multiplies its own columns (its part of the inner size); sums over warps, then over the cluster;
//   projection: a warp makes its own columns, which stay in registers while the mean of squares goes round.
// The stream and the gated values are float32 and stay so: each is split into three bfloat16 whose sum is the float to
// its last bit (24 of 24), against weights that are bfloat16 anyway, so the products are exact and the sums float
// (mma_bf16_add: what is added errs by 1.3e-7 to 1.5e-7 of itself, 1.8e-7 to 2.2e-7 in the block per token above; sums left in the
// tensor core erred by 3.1e-7 with many tokens, at 2 to 8 % less time).
// Few tokens (MT 1): the smallest COLS whose cluster is at most 8 blocks, and the weights are asked into L2 ahead of the
// wait.  Width 64 on 2,048 at 8 / 300 / 3,874 tokens: 20 / 79 / 187 us before, 10 / 35 / 71; on 4,096: 37 / 136 / 581, 14 / 36 / 147.
constexpr int SIDE_WARPS = 8;

__device__ __forceinline__ void side_cluster_sync() {
    __syncwarp();
    asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

__device__ __forceinline__ float side_remote(const float* p, int rank) {
    uint32_t there;
    float v;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(there) : "r"(smem_u32(p)), "r"(rank));
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(there) : "memory");
    return v;
}

template <int DIM, int COLS, int MT, bool ROOMY>
__global__ void __launch_bounds__(SIDE_WARPS * 32, ROOMY && (MT == 2 || DIM * COLS >= 32 * 64) ? 1 : 2)
token_side_mma_kernel(float* __restrict__ x, const int* __restrict__ ids, const __nv_bfloat16* __restrict__ table,
                      int table_stride, int offset, int vocab, const __nv_bfloat16* __restrict__ gate_w,
                      const __nv_bfloat16* __restrict__ proj_t, const float* __restrict__ norm_w, float eps,
                      const float* __restrict__ next_gamma, float next_eps, __nv_bfloat16* __restrict__ next_out,
                      int n_tokens, int hidden, int ranks) {
    constexpr int R = 16 * MT, CW = COLS < 64 ? COLS : 64, CHUNKS = COLS / CW, TILES = CW / 8, PITCH = DIM + 8;
    extern __shared__ __align__(16) float side_smem[];
    float* part = side_smem;                                          // [warps][R][DIM]
    float* own = part + SIDE_WARPS * R * DIM;                         // [R][DIM], read by the cluster
    float* squares = own + R * DIM;                                   // [warps][R]
    float* own_squares = squares + SIDE_WARPS * R;                    // [2][R], read by the cluster
    float* factor = own_squares + 2 * R;                              // [R]
    __nv_bfloat16* gated = (__nv_bfloat16*)(factor + R);              // [3][R][PITCH]
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
    const int rank = blockIdx.x % ranks, t0 = blockIdx.x / ranks * R;
    const int block_col = rank * SIDE_WARPS * COLS, col0 = block_col + warp * COLS;
    // Few tokens: the chain of loads is all there is, so that the weights and the norms' weights, which no kernel in front writes,
    // are in registers ahead of the wait.  The ids are not: a kernel in front may be the one that chooses them.  They are asked for first
    // behind the wait, and their table entries as soon as the first products have been issued, two barriers ahead of their use.
    constexpr bool EARLY = ROOMY && MT == 1 && COLS <= 64;
    constexpr int EACH = R * DIM / (SIDE_WARPS * 32);                 // gated values a thread makes
    static_assert(R * DIM % (SIDE_WARPS * 32) == 0, "gated values a thread");
    int id[EACH];
    float entry[EACH];
    auto known = [&](int n) { return id[n] >= 0 && id[n] < vocab; };  // (the embedding has flagged an id outside the table)
    auto load_ids = [&]() {
#pragma unroll
        for (int n = 0; n < EACH; ++n) id[n] = ids[min(t0 + (tid + n * SIDE_WARPS * 32) / DIM, n_tokens - 1)];
    };
    auto load_entries = [&]() {
#pragma unroll
        for (int n = 0; n < EACH; ++n)
            entry[n] = known(n) ? __bfloat162float(table[(size_t)id[n] * table_stride + offset + (tid + n * SIDE_WARPS * 32) % DIM]) : 0.0f;
    };
    auto load_gate = [&](int c, uint4 (&w)[DIM / 8]) {
#pragma unroll
        for (int n = 0; n < DIM / 8; ++n) w[n] = *(const uint4*)(gate_w + (size_t)(8 * n + g) * hidden + col0 + c + 8 * t);
    };
    auto load_proj = [&](int c, int k, uint32_t (&w)[4][TILES / 2]) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const __nv_bfloat16* at = proj_t + (size_t)(k + 2 * t + (i & 1) + 8 * (i >> 1)) * hidden + col0 + c * CW + TILES * g;
            if (TILES == 8) { const uint4 v = *(const uint4*)at; w[i][0] = v.x; w[i][1] = v.y; w[i][TILES / 2 - 2] = v.z; w[i][TILES / 2 - 1] = v.w; }
            else { const uint2 v = *(const uint2*)at; w[i][0] = v.x; w[i][1] = v.y; }
        }
    };
    uint4 gate_early[EARLY ? COLS / 32 : 1][DIM / 8];
    uint32_t proj_early[EARLY ? DIM / 16 : 1][4][TILES / 2];
    float4 norm_early[EARLY ? TILES / 2 : 1], next_early[EARLY ? TILES / 2 : 1];
    if (EARLY && col0 < hidden) {
#pragma unroll
        for (int c = 0; c < COLS; c += 32) load_gate(c, gate_early[c / 32]);
#pragma unroll
        for (int k = 0; k < DIM; k += 16) load_proj(0, k, proj_early[k / 16]);
#pragma unroll
        for (int i = 0; i < TILES / 2; ++i) {
            norm_early[i] = *(const float4*)(norm_w + col0 + 2 * TILES * t + 4 * i);
            if (next_out) next_early[i] = *(const float4*)(next_gamma + col0 + 2 * TILES * t + 4 * i);
        }
    } else if (!EARLY && MT == 1) {
        constexpr int LINES = SIDE_WARPS * COLS * 2 / 128;             // 128-byte lines of a weight row in this block's columns
        for (int i = tid; i < 2 * DIM * LINES; i += SIDE_WARPS * 32) {
            const int c = block_col + (i % LINES) * 64, row = (i / LINES) % DIM;
            const __nv_bfloat16* at = (i < DIM * LINES ? gate_w : proj_t) + (size_t)row * hidden + c;
            if (c < hidden) asm volatile("prefetch.global.L2 [%0];" :: "l"(at));
        }
    }
    pdl_launch_dependents();
    pdl_wait();
    if (EARLY) load_ids();
    const float* rows[MT][2];
#pragma unroll
    for (int m = 0; m < MT; ++m)
#pragma unroll
        for (int h = 0; h < 2; ++h) rows[m][h] = x + (size_t)min(t0 + 16 * m + 8 * h + g, n_tokens - 1) * hidden;

    // gate_w . x over this warp's columns: 32 at a time, eight neighbours a lane (the order of k inside the two products
    // of 16 is the same for both operands)
    {
        float acc[MT][DIM / 8][4] = {};
#pragma unroll (EARLY ? COLS / 32 : MT == 1 ? 2 : 1)
        for (int c = 0; c < COLS; c += 32) {
            const int k = col0 + c + 8 * t;
            if (col0 + c >= hidden) break;
            uint4 w[DIM / 8];
            if (!EARLY) load_gate(c, w);
            uint32_t a[MT][2][3][4];
#pragma unroll
            for (int m = 0; m < MT; ++m)
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const float4 u = *(const float4*)(rows[m][h] + k), v = *(const float4*)(rows[m][h] + k + 4);
                    uint32_t p[4][3];
                    split3(u.x, u.y, p[0]); split3(u.z, u.w, p[1]);
                    split3(v.x, v.y, p[2]); split3(v.z, v.w, p[3]);
#pragma unroll
                    for (int s = 0; s < 3; ++s) {
                        a[m][0][s][h] = p[0][s]; a[m][0][s][2 + h] = p[1][s];
                        a[m][1][s][h] = p[2][s]; a[m][1][s][2 + h] = p[3][s];
                    }
                }
#pragma unroll
            for (int n = 0; n < DIM / 8; ++n)
#pragma unroll
                for (int m = 0; m < MT; ++m) {
                    const uint4 of = EARLY ? gate_early[c / 32 % (EARLY ? COLS / 32 : 1)][n] : w[n];
                    mma_bf16_add<3>(acc[m][n], a[m][0], of.x, of.y);
                    mma_bf16_add<3>(acc[m][n], a[m][1], of.z, of.w);
                }
        }
#pragma unroll
        for (int m = 0; m < MT; ++m)
#pragma unroll
            for (int n = 0; n < DIM / 8; ++n) {
                float* at = part + ((size_t)warp * R + 16 * m + g) * DIM + 8 * n + 2 * t;
                *(float2*)at = make_float2(acc[m][n][0], acc[m][n][1]);
                *(float2*)(at + 8 * DIM) = make_float2(acc[m][n][2], acc[m][n][3]);
            }
    }
    if (EARLY) load_entries();
    __syncthreads();
    for (int i = tid; i < R * DIM; i += SIDE_WARPS * 32) {
        float sum = part[i];
#pragma unroll
        for (int w = 1; w < SIDE_WARPS; ++w) sum += part[w * R * DIM + i];
        own[i] = sum;
    }
    if (!EARLY) {
        load_ids();
        load_entries();
    }
    side_cluster_sync();
#pragma unroll
    for (int n = 0; n < EACH; ++n) {
        const int i = tid + n * SIDE_WARPS * 32;
        float sum = 0.0f;
        for (int r = 0; r < ranks; ++r) sum += side_remote(own + i, r);
        uint32_t parts[3];
        split3(known(n) ? gelu_tanh(sum) * entry[n] : 0.0f, 0.0f, parts);
#pragma unroll
        for (int s = 0; s < 3; ++s) gated[(s * R + i / DIM) * PITCH + i % DIM] = __ushort_as_bfloat16((unsigned short)parts[s]);
    }
    __syncthreads();

    // proj . gated for this warp's columns: column n of tile j is TILES * n + j of a chunk of CW, so that a lane's loads
    // of the four rows it needs and its results lie side by side
    float y[CHUNKS][MT][TILES][4] = {};
    float sums[MT][2] = {};
#pragma unroll
    for (int c = 0; c < CHUNKS; ++c) {
        if (col0 + c * CW >= hidden) continue;
#pragma unroll
        for (int k = 0; k < DIM; k += 16) {
            uint32_t loaded[4][TILES / 2];
            if (!EARLY) load_proj(c, k, loaded);
            const uint32_t (&w)[4][TILES / 2] = EARLY ? proj_early[k / 16 % (EARLY ? DIM / 16 : 1)] : loaded;
#pragma unroll
            for (int m = 0; m < MT; ++m) {
                uint32_t a[3][4];
#pragma unroll
                for (int s = 0; s < 3; ++s) {
                    const __nv_bfloat16* at = gated + (s * R + 16 * m + g) * PITCH + k + 2 * t;
                    a[s][0] = *(const uint32_t*)at; a[s][1] = *(const uint32_t*)(at + 8 * PITCH);
                    a[s][2] = *(const uint32_t*)(at + 8); a[s][3] = *(const uint32_t*)(at + 8 * PITCH + 8);
                }
#pragma unroll
                for (int j = 0; j < TILES; ++j) {
                    const uint32_t pick = j & 1 ? 0x7632 : 0x5410;
                    mma_bf16_add<3>(y[c][m][j], a, __byte_perm(w[0][j >> 1], w[1][j >> 1], pick), __byte_perm(w[2][j >> 1], w[3][j >> 1], pick));
                }
            }
        }
#pragma unroll
        for (int m = 0; m < MT; ++m)
#pragma unroll
            for (int j = 0; j < TILES; ++j)
#pragma unroll
                for (int h = 0; h < 2; ++h)
                    sums[m][h] += y[c][m][j][2 * h] * y[c][m][j][2 * h] + y[c][m][j][2 * h + 1] * y[c][m][j][2 * h + 1];
    }
    // the rows' factor 1 / sqrt(mean of squares + eps) from this lane's sums: over the quad, the warps, the cluster
    auto make_factor = [&](int which, float eps_of) {
#pragma unroll
        for (int m = 0; m < MT; ++m)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                float v = sums[m][h];
                v += __shfl_xor_sync(0xffffffffu, v, 1);
                v += __shfl_xor_sync(0xffffffffu, v, 2);
                if (t == 0) squares[warp * R + 16 * m + 8 * h + g] = v;
            }
        __syncthreads();
        if (tid < R) {
            float v = 0.0f;
            for (int w = 0; w < SIDE_WARPS; ++w) v += squares[w * R + tid];
            own_squares[which * R + tid] = v;
        }
        side_cluster_sync();
        if (tid < R) {
            float v = 0.0f;
            for (int r = 0; r < ranks; ++r) v += side_remote(own_squares + which * R + tid, r);
            factor[tid] = 1.0f / sqrtf(v / (float)hidden + eps_of);
        }
        __syncthreads();
    };
    float4 old[EARLY ? 2 : 1][EARLY ? TILES / 2 : 1];
    if (EARLY && col0 < hidden) {
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int i = 0; i < TILES / 2; ++i) old[h][i] = *(const float4*)(rows[0][h] + col0 + 2 * TILES * t + 4 * i);
    }
    make_factor(0, eps);
#pragma unroll
    for (int m = 0; m < MT; ++m)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int row = 16 * m + 8 * h + g;
            const float inverse = factor[row];
            sums[m][h] = 0.0f;
            if (t0 + row >= n_tokens) continue;
#pragma unroll
            for (int c = 0; c < CHUNKS; ++c) {
                if (col0 + c * CW >= hidden) continue;
                const int col = col0 + c * CW + 2 * TILES * t;
                float* at = x + (size_t)(t0 + row) * hidden + col;
#pragma unroll
                for (int i = 0; i < 2 * TILES; i += 4) {
                    float4 v = EARLY ? old[EARLY ? h : 0][EARLY ? i / 4 : 0] : *(const float4*)(at + i);
                    const float4 n = EARLY ? norm_early[EARLY ? i / 4 : 0] : *(const float4*)(norm_w + col + i);
                    const int half = i / TILES, j = i % TILES;
                    v.x += y[c][m][j][2 * h + half] * inverse * n.x; v.y += y[c][m][j + 1][2 * h + half] * inverse * n.y;
                    v.z += y[c][m][j + 2][2 * h + half] * inverse * n.z; v.w += y[c][m][j + 3][2 * h + half] * inverse * n.w;
                    *(float4*)(at + i) = v;
                    y[c][m][j][2 * h + half] = v.x; y[c][m][j + 1][2 * h + half] = v.y;
                    y[c][m][j + 2][2 * h + half] = v.z; y[c][m][j + 3][2 * h + half] = v.w;
                    sums[m][h] += v.x * v.x + v.y * v.y + v.z * v.z + v.w * v.w;
                }
            }
        }
    if (next_out) {
        __syncthreads();                                              // (the factors have been read)
        make_factor(1, next_eps);
#pragma unroll
        for (int m = 0; m < MT; ++m)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int row = 16 * m + 8 * h + g;
                if (t0 + row >= n_tokens) continue;
                const float inverse = factor[row];
#pragma unroll
                for (int c = 0; c < CHUNKS; ++c) {
                    if (col0 + c * CW >= hidden) continue;
                    const int col = col0 + c * CW + 2 * TILES * t;
                    __nv_bfloat16* at = next_out + (size_t)(t0 + row) * hidden + col;
#pragma unroll
                    for (int i = 0; i < 2 * TILES; i += 8) {
                        uint32_t packed[4];
#pragma unroll
                        for (int q = 0; q < 4; ++q) {
                            const int e = i + 2 * q, half = e / TILES, j = e % TILES;
                            const float4 four = next_early[EARLY ? e / 4 : 0];
                            const float2 n = EARLY ? (e & 2 ? make_float2(four.z, four.w) : make_float2(four.x, four.y)) : *(const float2*)(next_gamma + col + e);
                            const __nv_bfloat162 v = __floats2bfloat162_rn(y[c][m][j][2 * h + half] * inverse * n.x,
                                                                           y[c][m][j + 1][2 * h + half] * inverse * n.y);
                            packed[q] = *(const uint32_t*)&v;
                        }
                        *(uint4*)(at + i) = make_uint4(packed[0], packed[1], packed[2], packed[3]);
                    }
                }
            }
    }
    side_cluster_sync();                                              // no block leaves while another reads its sums
}

template <int DIM, int COLS, int MT, bool ROOMY>
static int launch_token_side_mma(float* x, const int* ids, const void* table, int table_stride, int offset, int vocab,
                                 const void* gate_w, const void* proj_t, const float* norm_w, float eps,
                                 const float* next_gamma, float next_eps, void* next_out, int n_tokens, int hidden,
                                 cudaStream_t stream) {
    constexpr int R = 16 * MT;
    constexpr size_t smem = (size_t)((SIDE_WARPS + 1) * R * DIM + (SIDE_WARPS + 3) * R) * 4 + (size_t)3 * R * (DIM + 8) * 2;
    auto kernel = token_side_mma_kernel<DIM, COLS, MT, ROOMY>;
    if (int code = reserve_shared_once<token_side_mma_kernel<DIM, COLS, MT, ROOMY>>("skv_token_side", smem)) return code;
    const int ranks = (hidden + SIDE_WARPS * COLS - 1) / (SIDE_WARPS * COLS);
    cudaLaunchConfig_t config = {};
    config.gridDim = dim3((unsigned)(ranks * ((n_tokens + R - 1) / R)));
    config.blockDim = dim3(SIDE_WARPS * 32);
    config.dynamicSmemBytes = smem;
    config.stream = stream;
    cudaLaunchAttribute attributes[2];
    attributes[0].id = cudaLaunchAttributeClusterDimension;
    attributes[0].val.clusterDim.x = ranks;
    attributes[0].val.clusterDim.y = 1;
    attributes[0].val.clusterDim.z = 1;
    attributes[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attributes[1].val.programmaticStreamSerializationAllowed = 1;
    config.attrs = attributes;
    config.numAttrs = pdl_enabled() ? 2 : 1;
    const cudaError_t status = cudaLaunchKernelEx(&config, kernel, x, ids, (const __nv_bfloat16*)table, table_stride, offset, vocab,
                                                  (const __nv_bfloat16*)gate_w, (const __nv_bfloat16*)proj_t, norm_w, eps, next_gamma,
                                                  next_eps, (__nv_bfloat16*)next_out, n_tokens, hidden, ranks);
    if (status != cudaSuccess) return fail("skv_token_side", cudaGetErrorString(status));
    return 0;
}

// At most 256 tokens.  With as many registers as they ask for (they hold weights ahead of the wait) the forms below take up to 128, and two
// blocks share an SM, or up to 255 and have it to themselves.  The latter are the faster ones while all clusters run at once, which fifteen of eight
// blocks do and sixteen don't (a partition of the GPU leaves some of its SMs over): 240 tokens with / with at most 128 registers, width 64 on
// 2,048 10.4 / 14.1 us, 32 on 8,192 17.9 / 23.5; 256 tokens 19.5 / 13.6 and 34.6 / 24.4.  (Width 64 on more than 4,096 takes more than 128 without such weights.)
template <int DIM, int COLS>
static int launch_token_side_few(float* x, const int* ids, const void* table, int table_stride, int offset, int vocab,
                                 const void* gate_w, const void* proj_t, const float* norm_w, float eps,
                                 const float* next_gamma, float next_eps, void* next_out, int n_tokens, int hidden,
                                 cudaStream_t stream) {
    const int ranks = (hidden + SIDE_WARPS * COLS - 1) / (SIDE_WARPS * COLS), clusters = (n_tokens + 15) / 16;
    if constexpr (DIM * COLS >= 32 * 64 && DIM * COLS < 64 * 128)
        if (ranks * clusters > sm_count() - sm_count() / 6)
            return launch_token_side_mma<DIM, COLS, 1, false>(x, ids, table, table_stride, offset, vocab, gate_w, proj_t, norm_w, eps,
                                                              next_gamma, next_eps, next_out, n_tokens, hidden, stream);
    return launch_token_side_mma<DIM, COLS, 1, true>(x, ids, table, table_stride, offset, vocab, gate_w, proj_t, norm_w, eps, next_gamma,
                                                     next_eps, next_out, n_tokens, hidden, stream);
}
#endif

}  // namespace skv

using namespace skv;

static int stream_threads(int hidden) { return hidden >= 2048 ? 512 : (hidden >= 512 ? 256 : 128); }

// x [n_rows, hidden] float += rmsnorm(y [n_rows, hidden] float) * gamma.  next_gamma and next_out (compute dtype,
// [n_rows, hidden]) both given: next_out = rmsnorm(new x) * next_gamma as well.
SKV_EXPORT int skv_rmsnorm_add(const float* y, const float* gamma, float eps, float* x, const float* next_gamma,
                               float next_eps, void* next_out, int n_rows, int hidden, cudaStream_t stream) {
    if (n_rows <= 0) return 0;
    if (hidden <= 0) return fail("skv_rmsnorm_add", "hidden must be positive");
    if (next_gamma && !next_out) return fail("skv_rmsnorm_add", "the next norm needs a place for its result");
    const int threads = stream_threads(hidden);
    const bool aligned = hidden % 4 == 0 &&
                         (((uintptr_t)y | (uintptr_t)x | (uintptr_t)gamma | (uintptr_t)next_gamma | (uintptr_t)next_out) & 15) == 0;
    if (aligned && hidden <= 4 * 4 * threads)
        return launch_pdl("skv_rmsnorm_add", rmsnorm_add_rows_kernel<skv_t, 4>, dim3(n_rows), dim3(threads), 0, stream, y,
                          gamma, eps, x, next_gamma, next_eps, (skv_t*)next_out, hidden);
    return launch_pdl("skv_rmsnorm_add", rmsnorm_add_kernel<skv_t>, dim3(n_rows), dim3(threads), 0,
                      stream, y, gamma, eps, x, next_gamma, next_eps, (skv_t*)next_out, hidden);
}

// table [vocab, table_stride], of whose rows the columns offset .. offset + dim - 1 are this layer's; gate_w
// [dim, hidden]; proj_t [dim, hidden], the projection transposed; norm_w float [hidden].  branch and post_gamma
// (both or neither): x += rmsnorm(branch [n_tokens, hidden] float) * post_gamma comes first, in the same pass.
SKV_EXPORT int skv_token_side(float* x, const int* ids, const void* table, int table_stride, int offset, int dim,
                              int vocab, const void* gate_w, const void* proj_t, const float* norm_w, float eps,
                              const float* next_gamma, float next_eps, void* next_out, int n_tokens, int hidden,
                              const float* branch, const float* post_gamma, float post_eps, cudaStream_t stream) {
    if (n_tokens <= 0) return 0;
    if (hidden <= 0 || dim <= 0 || vocab <= 0) return fail("skv_token_side", "sizes must be positive");
    if ((branch == nullptr) != (post_gamma == nullptr))
        return fail("skv_token_side", "a branch needs the weight of the norm it passes on its way into the stream");
    if (offset < 0 || offset + dim > table_stride) return fail("skv_token_side", "the layer's columns lie outside the table");
    if ((next_gamma == nullptr) != (next_out == nullptr))
        return fail("skv_token_side", "the next norm needs its weight and a place for its result");
    if ((size_t)(((dim + 3) & ~3) + hidden) * sizeof(float) > 200 * 1024)
        return fail("skv_token_side", "the stream is too wide for one block's shared memory");
#if SKV_DTYPE == SKV_BF16
    // the tensor-core form: a gated width it is built for, columns in whole chunks of 64 for at most 8 blocks a cluster,
    // 16-byte rows, nothing to add first
    if (!branch && (dim == 16 || dim == 32 || dim == 64) && hidden % 64 == 0 && hidden <= 8 * SIDE_WARPS * 128 &&
        (((uintptr_t)x | (uintptr_t)gate_w | (uintptr_t)proj_t | (uintptr_t)norm_w | (uintptr_t)next_gamma | (uintptr_t)next_out) & 15) == 0) {
#define SKV_SIDE_ARGS x, ids, table, table_stride, offset, vocab, gate_w, proj_t, norm_w, eps, next_gamma, next_eps, next_out, n_tokens, hidden, stream
#define SKV_SIDE_DIM(DIM) (n_tokens > 256 ? launch_token_side_mma<DIM, 128, 2, true>(SKV_SIDE_ARGS) :                       \
                           hidden <= 8 * SIDE_WARPS * 32 ? launch_token_side_few<DIM, 32>(SKV_SIDE_ARGS) :                  \
                           hidden <= 8 * SIDE_WARPS * 64 ? launch_token_side_few<DIM, 64>(SKV_SIDE_ARGS) : launch_token_side_few<DIM, 128>(SKV_SIDE_ARGS))
        return dim == 64 ? SKV_SIDE_DIM(64) : dim == 32 ? SKV_SIDE_DIM(32) : SKV_SIDE_DIM(16);
#undef SKV_SIDE_DIM
#undef SKV_SIDE_ARGS
    }
#endif
    const bool vec = hidden % 4 == 0 && (((uintptr_t)x | (uintptr_t)gate_w) & 15) == 0 && sizeof(skv_t) * hidden % 8 == 0;
    // eight tokens a block where their projected rows fit its shared memory, else four, else one; one token a block
    // where tokens are few, so that the step has blocks enough
    const size_t per_token = (size_t)(((dim + 3) & ~3) + hidden) * sizeof(float);
    const int tok = n_tokens <= 256 ? 1 : (8 * per_token <= 160 * 1024 ? 8 : (4 * per_token <= 200 * 1024 ? 4 : 1));
    const int threads = tok == 1 && hidden >= 1024 ? 512 : 256;      // (the many-token forms keep 100 to 200 registers a thread)
#define SKV_SIDE(TOK, VEC) launch_token_side<TOK, VEC>(x, ids, table, table_stride, offset, dim, vocab, gate_w, proj_t, norm_w, \
                                                      eps, next_gamma, next_eps, next_out, n_tokens, hidden, branch, post_gamma, \
                                                      post_eps, threads, stream)
    if (tok == 8) return vec ? SKV_SIDE(8, true) : SKV_SIDE(8, false);
    if (tok == 4) return vec ? SKV_SIDE(4, true) : SKV_SIDE(4, false);
    return vec ? SKV_SIDE(1, true) : SKV_SIDE(1, false);
#undef SKV_SIDE
}
