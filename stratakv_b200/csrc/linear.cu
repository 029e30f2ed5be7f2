// Linear layers: out = A[M,K] . W[N,K]^T with a fused epilogue.
//
// W keeps the checkpoint's [out, in] rows (K contiguous), as the reference's
// GPU path does (src/generation/generator.cpp:311-319).  These kernels replace
// its warp-per-output GEMV and 32x32 tile GEMM (src/cuda/gemm_cuda.cu:445-608)
// and the separate add and SwiGLU kernels that follow them (:221-231, 276-284).
//
// Epilogues (`mode`):
//   0 STORE      out[M,N] in the compute dtype
//   1 STORE_F32  out[M,N] float
//   2 ADD_F32    out[M,N] float += result          (residual sum in float)
//   3 GATED      W rows come in tiles of 16: rows 0-7 of a tile are gate rows
//                8t..8t+7, rows 8-15 the matching up rows; out[M,N/2] =
//                act(gate) * up in the compute dtype
//
// float build: true 32-bit FMA kernels (no tensor cores, no TF32), one that streams the weights for a few tokens and
// a tiled one.
// bfloat16 build: weight-streaming kernels for few tokens that take 16 weight rows
// at a time and feed tokens in groups of 8 through mma.sync m16n8k16 with float
// accumulation.  Each lane loads 16 bytes (8 consecutive k) of a weight row and of
// a token row and issues two MMAs on them; the k order inside an MMA is permuted
// the same way for both operands, which leaves the dot products unchanged.
#include "common.cuh"

namespace skv {

enum { MODE_STORE = 0, MODE_STORE_F32 = 1, MODE_ADD_F32 = 2, MODE_GATED = 3 };
// What callers name besides: out = act(a . w^T) in the compute dtype.  Inside the library it is MODE_STORE
// with ACT_ON_STORE added to the activation's code.
constexpr int MODE_STORE_ACT = 5;

__device__ __forceinline__ float activate(float g, act_t act) {
    if (act == ACT_GELU_TANH) return gelu_tanh(g);
    if (act == ACT_RELU2) return relu_squared(g);
    // silu(g) = g * sigmoid(g); the two-branch sigmoid of the reference's CPU
    // block (src/models/transformer_block.cpp:315-323) avoids overflow of exp.
    const float sig = g >= 0.0f ? 1.0f / (1.0f + expf(-g)) : expf(g) / (1.0f + expf(g));
    return g * sig;
}

// What a gated projection stores for a gate value and its up value.
__device__ __forceinline__ float gated_product(float gate, float up, act_t act) {
    if ((act & 0xff) == ACT_SWIGLU_CLAMP) return clamped_swiglu(gate, up, act_param(act));
    return activate(gate, act) * up;
}

template <typename T>
__device__ __forceinline__ void epilogue_store(void* out, int mode, int M, int N, int m, int n, float v, act_t act) {
    if (m >= M || n >= N) return;
    const size_t at = (size_t)m * N + n;
    if (mode == MODE_STORE) ((T*)out)[at] = from_float<T>(stored_value(v, act));
    else if (mode == MODE_STORE_F32) ((float*)out)[at] = v;
    else ((float*)out)[at] += v;
}

#if SKV_DTYPE == SKV_F32
// ---------------------------------------------------------------------------
// Steps of at most 16 tokens: the weights stream by once.  A block serves one group of 16 weight rows (of a gated
// matrix: 8 gate rows and their up rows).  Four row groups of four rows ({2j, 2j+1, 2j+8, 2j+9}, so that a gate row and
// its up row meet in one warp) times KS parts of K are its warps; a lane reads 16 bytes of each of its four rows and
// 16 bytes of every token, and the parts meet in shared memory in a fixed order.  The weights travel two rounds ahead in
// registers, the tokens two rounds ahead into shared memory (loads of the tokens through L1 queue behind the weights'
// misses).  Bound by HBM: the weights are the only traffic that counts.  KS fills the GPU where N is small: 2048 rows are
// 128 blocks.  Measured (weights larger than L2) at 1 / 3 / 8 / 16 tokens: 11264 x 2048 15.8 / 19.6 / 27 / 48 us (5.9 to 1.9
// TB/s), 2048 x 5632 10.5 / 12.5 / 15.5 / 24 us.  A 64 x 64 tile did this before, one token or sixteen alike: 335 and 640 us.
constexpr int FEW_MAX = 16;

// The four numbers at k..k+3 of a row of K numbers: one 16-byte load, or (WIDE off: any K, any alignment) one by one.
template <bool WIDE>
__device__ __forceinline__ float4 load_four(const float* row, int k, int K, bool live) {
    if (!live) return make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    if (WIDE) return k < K ? *(const float4*)(row + k) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    return make_float4(k < K ? row[k] : 0.0f, k + 1 < K ? row[k + 1] : 0.0f, k + 2 < K ? row[k + 2] : 0.0f,
                       k + 3 < K ? row[k + 3] : 0.0f);
}

template <int MT, int KS, bool WIDE>
__global__ void __launch_bounds__(128 * KS)
linear_f32_few_kernel(const float* __restrict__ A, const float* __restrict__ W, void* __restrict__ out,
                      int M, int N, int K, int mode, act_t act) {
    constexpr int STAGES = 3;
    extern __shared__ __align__(16) float few_smem[];
    float (*tokens)[MT][128] = (float (*)[MT][128])(few_smem + (size_t)(threadIdx.x >> 7) * STAGES * MT * 128);   // this part's [stage][token][128 k]
    __shared__ float sums[KS][16][MT];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int group = warp & 3, part = warp >> 2;
    const int n0 = blockIdx.x * 16;
    const int local[4] = {2 * group, 2 * group + 1, 2 * group + 8, 2 * group + 9};
    const int per_part = ((K + KS * 128 - 1) / (KS * 128)) * 128;
    const int k_begin = part * per_part + 4 * lane, k_end = min(K, (part + 1) * per_part);
    const float* rows[4];
    bool live[4];
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        live[r] = n0 + local[r] < N;
        rows[r] = W + (size_t)(live[r] ? n0 + local[r] : 0) * K;
    }
    float4 w[2][4];
    // the weights do not depend on the kernel in front: their first loads are under way before it has finished
#pragma unroll
    for (int s = 0; s < 2; ++s)
#pragma unroll
        for (int r = 0; r < 4; ++r) w[s][r] = load_four<WIDE>(rows[r], k_begin + 128 * s, k_end, live[r]);
    pdl_launch_dependents();
    pdl_wait();
    auto fetch_tokens = [&](int stage, int k) {                    // the part's warps take every fourth token each
#pragma unroll
        for (int m = group; m < MT; m += 4) {
            const float* row = A + (size_t)min(m, M - 1) * K;
            if (WIDE) {
                const int bytes = k < k_end ? 16 : 0;              // (zeros beyond the part's end)
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" :: "r"(smem_u32(&tokens[stage][m][4 * lane])),
                             "l"(row + (k < k_end ? k : 0)), "r"(bytes) : "memory");
            } else {
                *(float4*)&tokens[stage][m][4 * lane] = load_four<false>(row, k, k_end, true);
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    fetch_tokens(0, k_begin);
    fetch_tokens(1, k_begin + 128);
    float acc[4][MT] = {};
    int stage = 0, k = k_begin;
    // one round: the numbers of round i are used, those of round i + 2 are asked for
    auto round = [&](float4 (&wk)[4]) {
        asm volatile("cp.async.wait_group 1;" ::: "memory");
        asm volatile("bar.sync %0, 128;" :: "r"(part + 1) : "memory");    // the part's warps: everybody's copies are in, and the
        fetch_tokens(stage >= 1 ? stage - 1 : STAGES - 1, k + 256);      // stage of the round before is free again
#pragma unroll
        for (int m = 0; m < MT; ++m) {
            const float4 a = *(const float4*)&tokens[stage][m][4 * lane];
#pragma unroll
            for (int r = 0; r < 4; ++r)
                acc[r][m] = fmaf(a.w, wk[r].w, fmaf(a.z, wk[r].z, fmaf(a.y, wk[r].y, fmaf(a.x, wk[r].x, acc[r][m]))));
        }
#pragma unroll
        for (int r = 0; r < 4; ++r) wk[r] = load_four<WIDE>(rows[r], k + 256, k_end, live[r]);
        stage = stage == STAGES - 1 ? 0 : stage + 1;
        k += 128;
    };
    while (k - 4 * lane < k_end) {                                 // (a round beyond the end adds zeros)
        round(w[0]);
        round(w[1]);
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int m = 0; m < MT; ++m) {
            const float v = warp_sum(acc[r][m]);
            if (lane == 0) sums[part][local[r]][m] = v;
        }
    __syncthreads();
    for (int i = threadIdx.x; i < 16 * MT; i += 128 * KS) {
        const int n = i & 15, m = i >> 4;
        float v = sums[0][n][m];
#pragma unroll
        for (int p = 1; p < KS; ++p) v += sums[p][n][m];
        if (mode == MODE_GATED) {
            if (n >= 8 || m >= M) continue;
            float up = sums[0][n + 8][m];
#pragma unroll
            for (int p = 1; p < KS; ++p) up += sums[p][n + 8][m];
            const int half_n = N >> 1, o = (n0 >> 1) + n;
            if (o < half_n) ((float*)out)[(size_t)m * half_n + o] = gated_product(v, up, act);
        } else {
            epilogue_store<float>(out, mode, M, N, m, n0 + n, v, act);
        }
    }
}

// ---------------------------------------------------------------------------
// More tokens: BM x 128 output tiles, 2 BM threads with 8 x 8 outputs each, K in steps of 16 through two shared buffers
// (the next step's numbers travel to registers while this one's are multiplied).  Bound by the FMA pipe.  Where the
// tiles alone leave SMs idle, a cluster of up to 8 blocks shares K; each block then adds up a slice of the tile's rows
// over the blocks' shared memory, in rank order.  The 64 x 64 tile with 4 x 4 outputs a thread that this replaces read
// shared memory twice as often per product.  639 tokens: x 11264 x 2048 1,307 -> 658 us (45 TFLOP/s of the pipe's 74),
// x 2048 x 5632 1,172 -> 383 us; 2,000 tokens x 11264 x 2048 4,088 -> 2,030 us; 60 tokens x 2048 x 2048 257 -> 41 us.
// In shared memory a row of 16 k is stored k-major; A's row index is XORed with k's upper bits (a warp's stores then
// hit 32 banks), W's columns are kept as 64 "gate" columns (n mod 16 < 8) and their 64 "up" columns (n + 8), so that a
// thread holds both of a gated pair.
constexpr int FBN = 128, FBK = 16;

template <int BM, bool WIDE>
__global__ void __launch_bounds__(2 * BM, BM == 128 ? 2 : 1)
linear_f32_tile_kernel(const float* __restrict__ A, const float* __restrict__ W, void* __restrict__ out,
                       int M, int N, int K, int mode, act_t act) {
    constexpr int THREADS = 2 * BM, A_LOADS = 2, W_LOADS = FBN * FBK / 4 / THREADS;
    extern __shared__ __align__(16) float smem[];
    float (*As)[FBK][BM] = (float (*)[FBK][BM])smem;
    float (*Ws)[FBK][FBN] = (float (*)[FBK][FBN])(smem + 2 * FBK * BM);
    pdl_launch_dependents();
    pdl_wait();
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int tx = lane & 7, ty = lane >> 3, wn = warp & 1, wm = warp >> 1;
    const int splits = gridDim.z, split = blockIdx.z;
    const int m0 = blockIdx.y * BM, n0 = blockIdx.x * FBN;
    const int steps = (K + FBK - 1) / FBK;
    const int first = (int)((long long)steps * split / splits), last = (int)((long long)steps * (split + 1) / splits);

    float4 a_next[A_LOADS], w_next[W_LOADS];
    auto fetch = [&](int step) {
        const int k = step * FBK + 4 * (tid & 3);
#pragma unroll
        for (int i = 0; i < A_LOADS; ++i) {
            const int row = m0 + (tid + i * THREADS) / 4;
            a_next[i] = load_four<WIDE>(A + (size_t)min(row, M - 1) * K, k, K, row < M);
        }
#pragma unroll
        for (int i = 0; i < W_LOADS; ++i) {
            const int row = n0 + (tid + i * THREADS) / 4;
            w_next[i] = load_four<WIDE>(W + (size_t)min(row, N - 1) * K, k, K, row < N);
        }
    };
    auto keep = [&](int buffer) {
        const int kq = tid & 3;
#pragma unroll
        for (int i = 0; i < A_LOADS; ++i) {
            const int row = ((tid + i * THREADS) / 4) ^ (kq << 3);
            const float4 v = a_next[i];
            As[buffer][4 * kq][row] = v.x; As[buffer][4 * kq + 1][row] = v.y;
            As[buffer][4 * kq + 2][row] = v.z; As[buffer][4 * kq + 3][row] = v.w;
        }
#pragma unroll
        for (int i = 0; i < W_LOADS; ++i) {
            const int row = (tid + i * THREADS) / 4;
            const int at = (((row & 8) << 3) | ((row >> 4) << 3) | (row & 7)) ^ (kq << 3);
            const float4 v = w_next[i];
            Ws[buffer][4 * kq][at] = v.x; Ws[buffer][4 * kq + 1][at] = v.y;
            Ws[buffer][4 * kq + 2][at] = v.z; Ws[buffer][4 * kq + 3][at] = v.w;
        }
    };
    unsigned long long pairs[8][4] = {};                  // two neighbouring columns each: one instruction multiplies both
    if (first < last) {
        fetch(first);
        keep(0);
    }
    __syncthreads();
    for (int step = first; step < last; ++step) {
        const int buffer = (step - first) & 1;
        if (step + 1 < last) fetch(step + 1);
#pragma unroll
        for (int k = 0; k < FBK; ++k) {
            const int turn = (k >> 2) << 3;
            float a[8];
            *(float4*)a = *(const float4*)&As[buffer][k][(wm * 32 + ty * 4) ^ turn];
            *(float4*)(a + 4) = *(const float4*)&As[buffer][k][(wm * 32 + 16 + ty * 4) ^ turn];
            const ulonglong2 w_gate = *(const ulonglong2*)&Ws[buffer][k][(wn * 32 + tx * 4) ^ turn];
            const ulonglong2 w_up = *(const ulonglong2*)&Ws[buffer][k][(64 + wn * 32 + tx * 4) ^ turn];
            const unsigned long long w[4] = {w_gate.x, w_gate.y, w_up.x, w_up.y};
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                unsigned long long both;
                asm("mov.b64 %0, {%1, %1};" : "=l"(both) : "f"(a[i]));
#pragma unroll
                for (int j = 0; j < 4; ++j) asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(pairs[i][j]) : "l"(both), "l"(w[j]));
            }
        }
        if (step + 1 < last) keep(buffer ^ 1);
        __syncthreads();
    }
    float acc[8][8];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) asm("mov.b64 {%0, %1}, %2;" : "=f"(acc[i][2 * j]), "=f"(acc[i][2 * j + 1]) : "l"(pairs[i][j]));
    // column n0 + column(j), column(j + 4) = column(j) + 8
    const int column = ((wn * 32 + tx * 4) >> 3) * 16 + ((tx * 4) & 7);
    const int half_n = N >> 1;
    if (splits == 1) {
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int m = m0 + wm * 32 + ty * 4 + (i & 3) + (i >> 2) * 16;
            if (m >= M) continue;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int n = n0 + column + j;
                if (mode == MODE_GATED) {
                    if (n < N) ((float*)out)[(size_t)m * half_n + (n >> 4) * 8 + (n & 7)] = gated_product(acc[i][j], acc[i][j + 4], act);
                } else {
                    epilogue_store<float>(out, mode, M, N, m, n, acc[i][j], act);
                    epilogue_store<float>(out, mode, M, N, m, n + 8, acc[i][j + 4], act);
                }
            }
        }
        return;
    }
    // every block of the cluster leaves its sums in its own shared memory and adds up its share of the rows
    float (*tile)[FBN] = (float (*)[FBN])smem;             // (the last step's barrier is behind us: the buffers are free)
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int row = wm * 32 + ty * 4 + (i & 3) + (i >> 2) * 16;
#pragma unroll
        for (int j = 0; j < 8; ++j) tile[row][column + (j & 3) + (j >> 2) * 8] = acc[i][j];
    }
    asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
    const int rows_each = (BM + splits - 1) / splits;
    const uint32_t here = smem_u32(smem);
    for (int at = tid; at < rows_each * FBN; at += THREADS) {
        const int row = split * rows_each + at / FBN, c = at % FBN, m = m0 + row, n = n0 + c;
        if (row >= BM || m >= M || n >= N || (mode == MODE_GATED && (c & 8))) continue;
        float v = 0.0f, up = 0.0f;
        for (int rank = 0; rank < splits; ++rank) {
            uint32_t there;
            float part;
            asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(there) : "r"(here + (row * FBN + c) * 4), "r"(rank));
            asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(part) : "r"(there));
            v += part;
            if (mode == MODE_GATED) {
                asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(part) : "r"(there + 32));
                up += part;
            }
        }
        if (mode == MODE_GATED) ((float*)out)[(size_t)m * half_n + (n >> 4) * 8 + (n & 7)] = gated_product(v, up, act);
        else epilogue_store<float>(out, mode, M, N, m, n, v, act);
    }
    __syncwarp();
    // no block leaves while another still reads its sums
    asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

struct NormArgs { const float* row_scale; const float* partials_in; int n_partials_in, stride_in; float eps_in;
                  const int* rows; float* partials; int partial_stride; unsigned int* counter;
                  const float* gamma_next; float eps_next; void* scaled_out; float* row_scale_out; };

template <bool WIDE, int MT>
static int launch_few_of(const void* a, const void* w, void* out, int M, int N, int K, int mode, act_t act, cudaStream_t stream) {
    const dim3 grid((N + 15) / 16);
    constexpr int stages_of_part = 3 * MT * 128 * 4;
    // four parts of K where every block has an SM to itself (16 warps, most of its registers), else two
    if ((int)grid.x <= sm_count()) {
        if (int code = reserve_shared_once<linear_f32_few_kernel<MT, 4, WIDE>>("skv_linear(float)", 4 * stages_of_part)) return code;
        return launch_pdl("skv_linear(float)", linear_f32_few_kernel<MT, 4, WIDE>, grid, dim3(512), 4 * stages_of_part, stream, (const float*)a, (const float*)w, out, M, N, K, mode, act);
    }
    if (int code = reserve_shared_once<linear_f32_few_kernel<MT, 2, WIDE>>("skv_linear(float)", 2 * stages_of_part)) return code;
    return launch_pdl("skv_linear(float)", linear_f32_few_kernel<MT, 2, WIDE>, grid, dim3(256), 2 * stages_of_part, stream, (const float*)a, (const float*)w, out, M, N, K, mode, act);
}

template <bool WIDE>
static int launch_few(const void* a, const void* w, void* out, int M, int N, int K, int mode, act_t act, cudaStream_t stream) {
    if (M == 1) return launch_few_of<WIDE, 1>(a, w, out, M, N, K, mode, act, stream);
    if (M == 2) return launch_few_of<WIDE, 2>(a, w, out, M, N, K, mode, act, stream);
    if (M <= 4) return launch_few_of<WIDE, 4>(a, w, out, M, N, K, mode, act, stream);
    if (M <= 8) return launch_few_of<WIDE, 8>(a, w, out, M, N, K, mode, act, stream);
    return launch_few_of<WIDE, 16>(a, w, out, M, N, K, mode, act, stream);
}

template <int BM, bool WIDE>
static int launch_tile_of(const void* a, const void* w, void* out, int M, int N, int K, int mode, act_t act, cudaStream_t stream) {
    constexpr size_t buffers = (size_t)2 * FBK * (BM + FBN) * 4, tile = (size_t)BM * FBN * 4;
    const size_t smem = buffers > tile ? buffers : tile;
    if (int code = reserve_shared_once<linear_f32_tile_kernel<BM, WIDE>>("skv_linear(float)", smem)) return code;
    const int tiles = ((N + FBN - 1) / FBN) * ((M + BM - 1) / BM);
    // K is shared by as many blocks as keep the fullest SM's share smallest: its blocks run one after the other as far as
    // the FMA pipe goes, each for its part of K and about 200 k more to start and to add up.  A lone block leaves a third
    // of the pipe idle.  639 x 2048 x 5632 is 80 tiles on 148 SMs: 605 us as
    // two parts of K (160 blocks: some SMs have two), 383 us as five (400 blocks: three on the fullest).
    int splits = 1;
    float best = 0.0f;
    for (int s = 1; s <= 8 && (s == 1 || K >= 128 * s); ++s) {
        const int rounds = (tiles * s + sm_count() - 1) / sm_count();
        const float cost = (float)rounds * ((float)K / s + (s > 1 ? 200.0f : 100.0f)) * (rounds * BM < 256 ? 1.4f : 1.0f);
        if (s == 1 || cost < best) { best = cost; splits = s; }
    }
    cudaLaunchConfig_t config = {};
    config.gridDim = dim3((N + FBN - 1) / FBN, (M + BM - 1) / BM, splits);
    config.blockDim = dim3(2 * BM);
    config.dynamicSmemBytes = smem;
    config.stream = stream;
    cudaLaunchAttribute attributes[2];
    attributes[0].id = cudaLaunchAttributeClusterDimension;
    attributes[0].val.clusterDim.x = 1;
    attributes[0].val.clusterDim.y = 1;
    attributes[0].val.clusterDim.z = splits;
    attributes[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attributes[1].val.programmaticStreamSerializationAllowed = 1;
    config.attrs = attributes;
    config.numAttrs = pdl_enabled() ? 2 : 1;
    const cudaError_t status = cudaLaunchKernelEx(&config, linear_f32_tile_kernel<BM, WIDE>, (const float*)a, (const float*)w, out, M, N, K, mode, act);
    if (status != cudaSuccess) return fail("skv_linear(float)", cudaGetErrorString(status));
    return 0;
}

template <bool WIDE>
static int launch_tile(const void* a, const void* w, void* out, int M, int N, int K, int mode, act_t act, cudaStream_t stream) {
    if (M <= 32) return launch_tile_of<32, WIDE>(a, w, out, M, N, K, mode, act, stream);
    if (M <= 64 || (M + 63) / 64 % 2 == 1 && M <= 320) return launch_tile_of<64, WIDE>(a, w, out, M, N, K, mode, act, stream);
    return launch_tile_of<128, WIDE>(a, w, out, M, N, K, mode, act, stream);
}

static int launch_linear(const void* a, const void* w, void* out, int M, int N, int K, int mode, act_t act,
                         int* flag, const NormArgs& norm, cudaStream_t stream) {
    (void)flag;
    if (norm.row_scale || norm.partials_in || norm.partials) return fail("skv_linear(float)", "the norm-fused form exists in the bfloat16 build only");
    const bool wide = K % 4 == 0 && !(((uintptr_t)a | (uintptr_t)w) & 15);
    if (M <= FEW_MAX)
        return wide ? launch_few<true>(a, w, out, M, N, K, mode, act, stream) : launch_few<false>(a, w, out, M, N, K, mode, act, stream);
    return wide ? launch_tile<true>(a, w, out, M, N, K, mode, act, stream) : launch_tile<false>(a, w, out, M, N, K, mode, act, stream);
}

#else  // bfloat16
// ---------------------------------------------------------------------------
// RMSNorm folded into the projections around it.  The kernel that updates the float residual stream
// (residual-add mode) also leaves, per token, the updated row times the NEXT norm's weight in bfloat16
// and the factor 1 / sqrt(mean(row^2) + eps); the projection after that norm takes those activations
// and multiplies its result by the factor, which is one number per token and so commutes with the
// product.  Everything about the norm stays in float; the activations are rounded to bfloat16 once, as
// they are when the norm runs as a kernel of its own.
// A row's sum of squares is made in a fixed order whatever the timing: every block of the producer leaves
// the sum over its 16 columns.  With few tokens the consumer adds them up itself: it copies the partial sums
// of its tokens to shared memory while its main loop runs, so the producer ends without further ado.  With
// many tokens that would be a lot of traffic for every consumer block, and the producer's block that
// finishes last (a counter tells it) adds them up once and leaves the factor.
struct NormArgs {
    // consumer side: the factor itself, or the partial sums to make it from (both null: plain projection)
    const float* row_scale;        // [rows] factor of each row of X
    const float* partials_in;      // [rows, stride_in]: n_partials_in partial sums of squares per row
    int n_partials_in, stride_in;
    float eps_in;
    const int* rows;               // token m reads row rows[m] of X and of the above (null: row m)
    // producer side, residual-add mode (null partials: not wanted)
    float* partials;               // [M, partial_stride], partial_stride >= blocks of the grid
    int partial_stride;
    const float* gamma_next;       // [N] weight of the norm that reads the stream next
    __nv_bfloat16* scaled_out;     // [M, N] = bfloat16(updated out * gamma_next)
    unsigned int* counter;         // null: the consumer sums the partials; else zero before the launch and after it
    float eps_next;
    float* row_scale_out;          // with counter: [M] = 1 / sqrt(mean(updated out[m, :]^2) + eps_next)
};

// The three steps that the kernels below share.  First, what a folded norm's factors will be made from is sent for.
template <int COLS>
__device__ __forceinline__ void skinny_send_for_norm(float* staged, const NormArgs& norm, int M) {
    if (norm.partials_in) {
        // the partial sums are wanted after the main loop: they travel to shared memory meanwhile, 16 bytes
        // at a time where the rows allow it (the row in shared memory is `pitch` floats)
        const bool wide = (norm.stride_in & 3) == 0 && ((uintptr_t)norm.partials_in & 15) == 0;
        const int pitch = (norm.n_partials_in + 3) & ~3;
        const int pieces = wide ? pitch >> 2 : norm.n_partials_in;
        for (int i = threadIdx.x; i < COLS * pieces; i += blockDim.x) {
            const int m = i / pieces, piece = i - m * pieces;
            if (m < M) {
                const float* row = norm.partials_in + (size_t)(norm.rows ? norm.rows[m] : m) * norm.stride_in;
                if (wide)
                    asm volatile("cp.async.ca.shared.global [%0], [%1], 16;\n" ::"r"(smem_u32(staged + m * pitch + 4 * piece)),
                                 "l"(row + 4 * piece) : "memory");
                else
                    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(smem_u32(staged + m * pitch + piece)),
                                 "l"(row + piece) : "memory");
            }
        }
        asm volatile("cp.async.commit_group;\n" ::: "memory");
    } else if (norm.row_scale && !norm.rows && threadIdx.x * 32 < M) {
        // the factors are wanted after the main loop: bring their lines close meanwhile
        asm volatile("prefetch.global.L1 [%0];" ::"l"(norm.row_scale + threadIdx.x * 32));
    }
}

// Then, after the main loop, the factors of the block's tokens.
template <int COLS>
__device__ __forceinline__ void skinny_norm_factors(float* factor, const float* staged, const NormArgs& norm, int K, int warps, int warp, int lane) {
    if (norm.partials_in) {
        asm volatile("cp.async.wait_all;\n" ::: "memory");
        __syncthreads();
        for (int m = warp; m < COLS; m += warps) {          // one token per warp at a time, lanes in a fixed order
            float total = 0.0f;
            const int pitch = (norm.n_partials_in + 3) & ~3;
            for (int p = lane; p < norm.n_partials_in; p += 32) total += staged[m * pitch + p];
            total = warp_sum(total);
            if (lane == 0) factor[m] = 1.0f / sqrtf(total / (float)K + norm.eps_in);
        }
    }
}

// The block that gets here last adds the partial sums of squares up and leaves the rows' factors.
__device__ __forceinline__ void skinny_finish_partials(const NormArgs& norm, int M, int N, int partials, int warps, int warp, int lane) {
    __shared__ bool last;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) last = atomicAdd(norm.counter, 1u) == gridDim.x - 1;
    __syncthreads();
    if (last) {
        __threadfence();
        for (int m = warp; m < M; m += warps) {
            const float* partial = norm.partials + (size_t)m * norm.partial_stride;
            float total = 0.0f;
            for (int p = lane; p < partials; p += 32) total += __ldcg(partial + p);
            total = warp_sum(total);
            if (lane == 0) norm.row_scale_out[m] = 1.0f / sqrtf(total / (float)N + norm.eps_next);
        }
        if (threadIdx.x == 0) *norm.counter = 0u;
    }
}

// Last, the warps' partial tiles are added up and the result stored, rows n0 .. n0 + 15 of the weight.
template <int TG>
__device__ __forceinline__ void skinny_store(float* red, const float* factor, const float (&acc)[TG][4], void* __restrict__ out, int M,
                                             int N, int n0, int mode, act_t act, const NormArgs& norm, int warps, int warp, int lane) {
    constexpr int COLS = 8 * TG, PITCH = COLS + 1;
    const int g = lane >> 2, tig = lane & 3;
    float* mine = red + (size_t)warp * 16 * PITCH;
#pragma unroll
    for (int t = 0; t < TG; ++t) {
        mine[g * PITCH + t * 8 + 2 * tig] = acc[t][0];
        mine[g * PITCH + t * 8 + 2 * tig + 1] = acc[t][1];
        mine[(g + 8) * PITCH + t * 8 + 2 * tig] = acc[t][2];
        mine[(g + 8) * PITCH + t * 8 + 2 * tig + 1] = acc[t][3];
    }
    __syncthreads();
    for (int idx = threadIdx.x; idx < 16 * COLS; idx += blockDim.x) {
        const int r = idx & 15, m = idx >> 4;
        float sum = 0.0f;
        for (int w = 0; w < warps; ++w) sum += red[((size_t)w * 16 + r) * PITCH + m];
        if (norm.partials_in) sum *= factor[m];
        else if (norm.row_scale && m < M) sum *= norm.row_scale[norm.rows ? norm.rows[m] : m];
        red[(size_t)r * PITCH + m] = sum;          // warp 0's tile becomes the total
        // (each (r, m) is read and written by this thread only)
    }
    __syncthreads();
    if (mode == MODE_GATED) {
        const int half_n = N >> 1;
        for (int idx = threadIdx.x; idx < 8 * COLS; idx += blockDim.x) {
            const int r = idx & 7, m = idx >> 3;
            const int o = (n0 >> 1) + r;
            if (m < M && o < half_n) {
                const float gate = red[(size_t)r * PITCH + m], up = red[(size_t)(r + 8) * PITCH + m];
                ((__nv_bfloat16*)out)[(size_t)m * half_n + o] = __float2bfloat16_rn(gated_product(gate, up, act));
            }
        }
    } else if (mode == MODE_ADD_F32 && norm.partials) {
        // residual sum; the updated row times the next norm's weight; its sum of squares over this block's columns
        for (int idx = threadIdx.x; idx < 16 * COLS; idx += blockDim.x) {        // whole warps stay together
            const int r = idx & 15, m = idx >> 4;
            float updated = 0.0f;
            if (m < M && n0 + r < N) {
                float* at = (float*)out + (size_t)m * N + n0 + r;
                updated = *at + red[(size_t)r * PITCH + m];
                *at = updated;
                norm.scaled_out[(size_t)m * N + n0 + r] = __float2bfloat16_rn(updated * norm.gamma_next[n0 + r]);
            }
            float square = updated * updated;
#pragma unroll
            for (int offset = 8; offset > 0; offset >>= 1) square += __shfl_xor_sync(0xffffffffu, square, offset);
            if (r == 0 && m < M) norm.partials[(size_t)m * norm.partial_stride + blockIdx.x] = square;
        }
        if (norm.counter) skinny_finish_partials(norm, M, N, gridDim.x, warps, warp, lane);      // (one chunk of tokens: M <= 8*TG)
    } else {
        for (int idx = threadIdx.x; idx < 16 * COLS; idx += blockDim.x) {
            const int r = idx & 15, m = idx >> 4;
            epilogue_store<__nv_bfloat16>(out, mode, M, N, m, n0 + r, red[(size_t)r * PITCH + m], act);
        }
    }
}

// 17 to 64 tokens with a folded norm: one block owns 16 rows of W and every token (at most 8 TG).  Its warps take the
// 32-wide k steps round robin, then their partial tiles are summed in shared
// memory in warp order (a fixed order: results do not depend on timing).
// Weights do not depend on the kernel before this one, so the first batch of
// weight loads is issued before pdl_wait(): it overlaps the predecessor's tail.
template <int TG, int U>
__global__ void __launch_bounds__(256)
skinny_linear_bf16_kernel(const __nv_bfloat16* __restrict__ W, const __nv_bfloat16* __restrict__ X,
                          void* __restrict__ out, int M, int N, int K, int mode, act_t act, const NormArgs norm) {
    extern __shared__ float red[];                 // [warps][16][8*TG + 1], [8*TG] factors, [8*TG][n_partials_in] partial sums
    constexpr int COLS = 8 * TG, PITCH = COLS + 1;
    pdl_launch_dependents();
    const int warps = blockDim.x >> 5;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int g = lane >> 2, tig = lane & 3;
    const int n0 = blockIdx.x * 16;
    const int steps = (K + 31) >> 5;

    const int row_a = min(n0 + g, N - 1), row_b = min(n0 + g + 8, N - 1);
    const bool has_a = n0 + g < N, has_b = n0 + g + 8 < N;
    const __nv_bfloat16* wa_ptr = W + (size_t)row_a * K + tig * 8;
    const __nv_bfloat16* wb_ptr = W + (size_t)row_b * K + tig * 8;
    const uint4 zero = make_uint4(0u, 0u, 0u, 0u);

    uint4 wa[U], wb[U];
    auto load_weights = [&](int s0) {
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int k = (s0 + u * warps) << 5;
            const bool live = (s0 + u * warps) < steps && (k + tig * 8) < K;
            wa[u] = (live && has_a) ? __ldcs((const uint4*)(wa_ptr + k)) : zero;
            wb[u] = (live && has_b) ? __ldcs((const uint4*)(wb_ptr + k)) : zero;
        }
    };
    load_weights(warp);
    pdl_wait();                                    // activations (and the residual stream) are ready now

    const __nv_bfloat16* x_ptr[TG];
    bool has_x[TG];
#pragma unroll
    for (int t = 0; t < TG; ++t) {
        const int m = t * 8 + g;
        has_x[t] = m < M;
        const int safe = min(m, M - 1);
        x_ptr[t] = X + (size_t)(norm.rows ? norm.rows[safe] : safe) * K + tig * 8;
    }
    float* factor = red + (size_t)warps * 16 * PITCH;
    float* staged = factor + COLS;
    skinny_send_for_norm<COLS>(staged, norm, M);
    float acc[TG][4];
#pragma unroll
    for (int t = 0; t < TG; ++t) { acc[t][0] = acc[t][1] = acc[t][2] = acc[t][3] = 0.0f; }

    for (int s0 = warp; s0 < steps; s0 += warps * U) {
        if (s0 != warp) load_weights(s0);
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int k = (s0 + u * warps) << 5;
            const bool live = (s0 + u * warps) < steps && (k + tig * 8) < K;
#pragma unroll
            for (int t = 0; t < TG; ++t) {
                const uint4 xv = (live && has_x[t]) ? *(const uint4*)(x_ptr[t] + k) : zero;
                mma_bf16_16816(acc[t], wa[u].x, wb[u].x, wa[u].y, wb[u].y, xv.x, xv.y);
                mma_bf16_16816(acc[t], wa[u].z, wb[u].z, wa[u].w, wb[u].w, xv.z, xv.w);
            }
        }
    }
    skinny_norm_factors<COLS>(factor, staged, norm, K, warps, warp, lane);
    skinny_store<TG>(red, factor, acc, out, M, N, n0, mode, act, norm, warps, warp, lane);
}

// At most 16 tokens: the weights stream by once, and on their way they wait in shared memory.  Such a projection is bound by HBM
// and, in a decode step's chain of dependent kernels, by how much of its weights is on the SMs before the kernel in front has
// finished and how little must happen after that.  So:
//  * A lane copies (cp.async) the very 16 bytes that it will multiply into slots of its own, DEPTH steps of its warp ahead: no
//    registers for what is on its way, no barrier, and a wait for its own copies only.  The first DEPTH steps are asked for ahead
//    of the wait for the kernel in front, and asking goes on into the block's next tile, through its sums and stores.  128 KB on
//    its way an SM are needed: 64 KB a block and two blocks, or 96 to 144 KB in one.
//  * 16 warps share a tile of 16 rows, which leaves a warp 4 or 8 steps of the common inner sizes: their activations are read
//    once, all at the same time, and stay in registers for all of a block's tiles (XSTEPS).  Longer inner sizes bring theirs
//    through the slots beside the weights.
//  * A tile ends with one barrier; 128 threads per 8 tokens add the warps' sums up in warp order, and its gated pairs, squares and
//    stores need no other.  What they add to was asked for a tile ahead.
// Decode steps before (blocks of 4 to 16 warps that held the weights on their way in registers and came and went with the
// tiles, or walked them) and now, in us: Llama 2,048 x 22, 1 / 8 tokens 713 / 815 and 543 / 626; 4 layers of 4,096 with 14,336 at 1 / 16
// tokens 567 / 832 and 469 / 533; of 4,096 with 11,008 at 8 537 and 392; Zepavik 3,072 x 4 at 1 / 8 / 16 278 / 381 / 525 and 249 / 315 / 367.
// The same walk with the weights on their way in registers (two blocks of 8 warps, or 16 warps): 563 / 693 for the first pair.
constexpr int RING_WARPS = 16;

template <int TG, int XSTEPS, int DEPTH>
constexpr int ring_smem() { return RING_WARPS * DEPTH * (1024 + (XSTEPS ? 0 : 512 * TG)) + 2 * RING_WARPS * 16 * (8 * TG + 1) * 4; }

template <int TG, int XSTEPS, int DEPTH>
__global__ void __launch_bounds__(RING_WARPS * 32, 2 * (ring_smem<TG, XSTEPS, DEPTH>() + 1024) <= 228 * 1024 ? 2 : 1)
skinny_ring_bf16_kernel(const __nv_bfloat16* __restrict__ W, const __nv_bfloat16* __restrict__ X,
                        void* __restrict__ out, int M, int N, int K, int mode, act_t act, const NormArgs norm) {
    constexpr int PITCH = 8 * TG + 1, SLOT = 1024 + (XSTEPS ? 0 : 512 * TG);
    extern __shared__ __align__(128) unsigned char ring_raw[];
    float (*red)[RING_WARPS][16 * PITCH] = (float (*)[RING_WARPS][16 * PITCH])(ring_raw + RING_WARPS * DEPTH * SLOT);
    __shared__ float factor[8 * TG];
    pdl_launch_dependents();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int g = lane >> 2, tig = lane & 3;
    const int tiles = (N + 15) >> 4, per_tile = (((K + 31) >> 5) + RING_WARPS - 1) / RING_WARPS;
    const int k0 = warp * 32 + tig * 8;            // this lane's first k of a tile; a step further is RING_WARPS * 32 more
    const uint32_t mine_at = smem_u32(ring_raw) + warp * DEPTH * SLOT + lane * 16;

    int asked_tile = blockIdx.x, asked = 0, asked_slot = 0;      // the next step to ask for
    auto ask_weights = [&]() {
        if (asked_tile >= tiles) return;
        const int row = asked_tile * 16 + g, k = k0 + asked * (RING_WARPS * 32);
        const __nv_bfloat16* from = W + (size_t)row * K + k;
        const bool has_a = k < K && row < N, has_b = k < K && row + 8 < N;
        ring_copy(mine_at + asked_slot * SLOT, has_a ? from : W, has_a);
        ring_copy(mine_at + asked_slot * SLOT + 512, has_b ? from + (size_t)8 * K : W, has_b);
    };
    auto advance = [&]() {
        ring_commit();
        if (++asked_slot == DEPTH) asked_slot = 0;
        if (++asked == per_tile) { asked = 0; asked_tile += gridDim.x; }
    };
#pragma unroll
    for (int i = 0; i < DEPTH; ++i) { ask_weights(); advance(); }
    // the thread's output of a tile: column 16 tile + r of token m (the first 128 TG threads)
    const int r = threadIdx.x & 15, m = threadIdx.x >> 4;
    const bool stores = m < min(M, 8 * TG);
    const bool keeps = mode == MODE_ADD_F32 && norm.partials;
    int tile = blockIdx.x;
    float gamma = keeps && stores && tile * 16 + r < N ? norm.gamma_next[tile * 16 + r] : 0.0f;
    pdl_wait();                                    // activations (and the residual stream) are ready now

    const __nv_bfloat16* x_ptr[TG];
#pragma unroll
    for (int t = 0; t < TG; ++t) {
        const int safe = min(t * 8 + g, M - 1);
        x_ptr[t] = X + (size_t)(norm.rows ? norm.rows[safe] : safe) * K;
    }
    uint4 xv[XSTEPS ? XSTEPS : 1][TG];
    auto ask_x = [&](int step, int slot) {
        const int k = k0 + step * (RING_WARPS * 32);
#pragma unroll
        for (int t = 0; t < TG; ++t) {
            const bool live = t * 8 + g < M && k < K;
            ring_copy(mine_at + slot * SLOT + 1024 + 512 * t, live ? x_ptr[t] + k : X, live);
        }
    };
    if (XSTEPS) {
#pragma unroll
        for (int s = 0; s < XSTEPS; ++s)
#pragma unroll
            for (int t = 0; t < TG; ++t) {
                const int k = k0 + s * (RING_WARPS * 32);
                xv[s][t] = t * 8 + g < M && k < K ? *(const uint4*)(x_ptr[t] + k) : make_uint4(0u, 0u, 0u, 0u);
            }
    } else {
#pragma unroll
        for (int i = 0; i < DEPTH; ++i) ask_x(i % per_tile, i);
        ring_commit();
    }
    float old = 0.0f;
    if (mode == MODE_ADD_F32 && stores && tile * 16 + r < N) old = ((const float*)out)[(size_t)m * N + tile * 16 + r];
    if (norm.partials_in) {
        if (warp < M) {                            // a token a warp, lanes in a fixed order
            const float* row = norm.partials_in + (size_t)(norm.rows ? norm.rows[warp] : warp) * norm.stride_in;
            float total = 0.0f;
#pragma unroll 4
            for (int p = lane; p < norm.n_partials_in; p += 32) total += row[p];
            total = warp_sum(total);
            if (lane == 0) factor[warp] = 1.0f / sqrtf(total / (float)K + norm.eps_in);
        }
    } else if (norm.row_scale && threadIdx.x < M) {
        factor[threadIdx.x] = norm.row_scale[norm.rows ? norm.rows[threadIdx.x] : threadIdx.x];
    }
    if (!XSTEPS) ring_wait<0>();

    float acc[TG][4] = {};
    int slot = 0, parity = 0;
    auto step = [&](const uint4 (&kept)[TG]) {
        ring_wait<DEPTH - 1>();
        const uint32_t at = mine_at + slot * SLOT;
        const uint4 a = ring_read(at), b = ring_read(at + 512);
#pragma unroll
        for (int t = 0; t < TG; ++t) {
            const uint4 x = XSTEPS ? kept[t] : ring_read(at + 1024 + 512 * t);
            mma_bf16_16816(acc[t], a.x, b.x, a.y, b.y, x.x, x.y);
            mma_bf16_16816(acc[t], a.z, b.z, a.w, b.w, x.z, x.w);
        }
        // (the slot has been read: what the products needed is in registers)
        ask_weights();
        if (!XSTEPS && asked_tile < tiles) ask_x(asked, asked_slot);
        advance();
        if (++slot == DEPTH) slot = 0;
    };
    while (tile < tiles) {
        if (XSTEPS) {
#pragma unroll
            for (int s = 0; s < XSTEPS; ++s)
                if (s < per_tile) step(xv[s]);
        } else {
#pragma unroll 1
            for (int s = 0; s < per_tile; ++s) step(xv[0]);
        }
        float* mine = red[parity][warp];
#pragma unroll
        for (int t = 0; t < TG; ++t) {
            mine[g * PITCH + t * 8 + 2 * tig] = acc[t][0];
            mine[g * PITCH + t * 8 + 2 * tig + 1] = acc[t][1];
            mine[(g + 8) * PITCH + t * 8 + 2 * tig] = acc[t][2];
            mine[(g + 8) * PITCH + t * 8 + 2 * tig + 1] = acc[t][3];
            acc[t][0] = acc[t][1] = acc[t][2] = acc[t][3] = 0.0f;
        }
        __syncthreads();                           // (two buffers: the next tile's sums are written while this one's are read)
        const int n = tile * 16 + r;
        tile += gridDim.x;
        if (threadIdx.x < 128 * TG) {
            float sum = 0.0f;
#pragma unroll
            for (int w = 0; w < RING_WARPS; ++w) sum += red[parity][w][r * PITCH + m];       // in warp order, whatever the timing
            if (norm.partials_in || norm.row_scale) sum *= factor[m];
            const bool live = stores && n < N;
            if (mode == MODE_GATED) {
                const float up = __shfl_down_sync(0xffffffffu, sum, 8);
                if (live && r < 8)
                    ((__nv_bfloat16*)out)[(size_t)m * (N >> 1) + ((n >> 4) << 3) + r] = __float2bfloat16_rn(gated_product(sum, up, act));
            } else if (mode == MODE_ADD_F32) {
                const size_t at = (size_t)m * N + n;
                const float updated = live ? old + sum : 0.0f;
                if (live) ((float*)out)[at] = updated;
                if (keeps) {
                    // the updated row times the next norm's weight; its sum of squares over this tile's columns
                    if (live) norm.scaled_out[at] = __float2bfloat16_rn(updated * gamma);
                    float square = updated * updated;
#pragma unroll
                    for (int offset = 8; offset > 0; offset >>= 1) square += __shfl_xor_sync(0xffffffffu, square, offset);
                    if (r == 0 && stores) norm.partials[(size_t)m * norm.partial_stride + (n >> 4)] = square;
                }
                if (tile < tiles && stores && tile * 16 + r < N) {
                    old = ((const float*)out)[(size_t)m * N + tile * 16 + r];
                    if (keeps) gamma = norm.gamma_next[tile * 16 + r];
                }
            } else if (live) {
                epilogue_store<__nv_bfloat16>(out, mode, M, N, m, n, sum, act);
            }
        }
        parity ^= 1;
    }
    if (keeps && norm.counter) skinny_finish_partials(norm, M, N, tiles, RING_WARPS, warp, lane);
}

template <int TG, int XSTEPS, int DEPTH>
static int launch_ring_as(const void* a, const void* w, void* out, int M, int N, int K, int mode, act_t act, const NormArgs& norm,
                          int per_sm, cudaStream_t stream) {
    constexpr int smem = ring_smem<TG, XSTEPS, DEPTH>();
    if (int code = reserve_shared_once<skinny_ring_bf16_kernel<TG, XSTEPS, DEPTH>>("skv_linear(bfloat16)", smem)) return code;
    const int tiles = (N + 15) / 16, slots = per_sm * sm_count();
    return launch_pdl("skv_linear(bfloat16)", skinny_ring_bf16_kernel<TG, XSTEPS, DEPTH>, dim3(tiles < slots ? tiles : slots),
                      dim3(RING_WARPS * 32), smem, stream, (const __nv_bfloat16*)w, (const __nv_bfloat16*)a, out, M, N, K, mode, act, norm);
}

// Slots and blocks an SM by the inner size and the tiles, us a decode step (Llama 2,048 x 22 unless said otherwise).
// At most 8 tokens: two blocks of four slots fit an SM and overlap each other's ends, and where a projection has one an SM the next
// one's blocks are resident beside them (a single block of six or eight slots: 2,048 rows at 1 / 8 tokens 570 / 650 against 542 /
// 636, 2,560 rows 589 / 650, gate and up 556 / 648).  Inner sizes of 2,049 to 4,096 over more tiles than those two blocks hold:
// one block of eight, half the activations' reads (22,016 x 4,096 at 8 tokens, 4 layers and head 396 -> 380; 256 tiles are
// faster in twos, 474 against 479 at 1 token).  Where no norm is folded, kernels that stream through L1 stand between projections, and two
// blocks' slots leave them little of it: up to a tile an SM one block of six (Fidolix at 4 tokens 416 -> 386, Kedelorn at 8 364 -> 349,
// Vekanex at 1 213 -> 206).  Longer: six slots with their activations, 144 KB (2,048 x 5,632: 542, five 544, four
// 548; two blocks of three 583).
// 9 to 16 tokens take twice the registers for activations, so one block an SM (16 tokens, two blocks of four slots 910 against 750).
template <int TG>
static int launch_ring(const void* a, const void* w, void* out, int M, int N, int K, int mode, act_t act, const NormArgs& norm,
                       cudaStream_t stream) {
    const int steps = (K + 31) / 32;
    if (TG == 1) {
        if (steps <= 4 * RING_WARPS) {
            const bool folded = norm.partials || norm.partials_in || norm.row_scale;
            if (!folded && (N + 15) / 16 <= sm_count()) return launch_ring_as<1, 4, 6>(a, w, out, M, N, K, mode, act, norm, 1, stream);
            return launch_ring_as<1, 4, 4>(a, w, out, M, N, K, mode, act, norm, 2, stream);
        }
        if (steps <= 8 * RING_WARPS) {
            if ((N + 15) / 16 <= 2 * sm_count()) return launch_ring_as<1, 8, 4>(a, w, out, M, N, K, mode, act, norm, 2, stream);
            return launch_ring_as<1, 8, 8>(a, w, out, M, N, K, mode, act, norm, 1, stream);
        }
        return launch_ring_as<1, 0, 6>(a, w, out, M, N, K, mode, act, norm, 1, stream);
    }
    if (steps <= 4 * RING_WARPS) return launch_ring_as<2, 4, 6>(a, w, out, M, N, K, mode, act, norm, 1, stream);
    if (steps <= 8 * RING_WARPS) return launch_ring_as<2, 8, 8>(a, w, out, M, N, K, mode, act, norm, 1, stream);
    return launch_ring_as<2, 0, 4>(a, w, out, M, N, K, mode, act, norm, 1, stream);
}

template <int TG, int U>
static int launch_skinny(const void* a, const void* w, void* out, int M, int N, int K, int mode, act_t act,
                         const NormArgs& norm, cudaStream_t stream) {
    int warps = 8;
    while (warps > 1 && warps > (K + 31) / 32) warps >>= 1;          // never more warps than k steps
    const size_t smem = ((size_t)warps * 16 * (8 * TG + 1) + 8 * TG + (size_t)8 * TG * (norm.partials_in ? (norm.n_partials_in + 3) & ~3 : 0)) * sizeof(float);
    if (smem > 48 * 1024) return fail("skv_linear(bfloat16)", "too many partial sums for the consumer to stage: let the producer finish them");
    return launch_pdl("skv_linear(bfloat16)", skinny_linear_bf16_kernel<TG, U>, dim3((N + 15) / 16), dim3(warps * 32), smem, stream,
                      (const __nv_bfloat16*)w, (const __nv_bfloat16*)a, out, M, N, K, mode, act, norm);
}

// gemm_tcgen05.cu: the tensor-memory GEMM that serves steps with many tokens
int linear_tcgen05(const void* a, const void* w, void* out, int M, int N, int K, int mode, act_t act, int* flag,
                   cudaStream_t stream);

static int launch_linear(const void* a, const void* w, void* out, int M, int N, int K, int mode, act_t act,
                         int* flag, const NormArgs& norm, cudaStream_t stream) {
    if (K % 8 != 0)
        return fail("skv_linear(bfloat16)", "the inner size must be a multiple of 8 (16-byte rows)");
    if (((uintptr_t)a | (uintptr_t)w) & 15)
        return fail("skv_linear(bfloat16)", "operands must be 16-byte aligned");
    if ((norm.row_scale || norm.partials_in || norm.partials) && M > 64)
        return fail("skv_linear(bfloat16)", "the norm-fused form serves steps of at most 64 tokens");
    // above 16 tokens the tensor-memory kernels take over, unless a norm is folded into this projection
    // (from 9 tokens on they are faster over large weights, 16 tokens, 6,144 x 4,096 / 128,256 x 4,096 11.7 / 161 us against 17.5 /
    // 222, but tensor memory keeps a sum over the whole inner size and cuts it off at every step, where eight warps here sum an eighth
    // each: relative to float64 21e-7 against 4.7e-7, and 21e-7 against 2.4e-7 with an inner size of 2,048)
    if (M > 16 && !norm.row_scale && !norm.partials_in && !norm.partials)
        return linear_tcgen05(a, w, out, M, N, K, mode, act, flag, stream);
    if (M <= 8) return launch_ring<1>(a, w, out, M, N, K, mode, act, norm, stream);
    if (M <= 16) return launch_ring<2>(a, w, out, M, N, K, mode, act, norm, stream);
    if (M <= 32) return launch_skinny<4, 4>(a, w, out, M, N, K, mode, act, norm, stream);
    return launch_skinny<8, 4>(a, w, out, M, N, K, mode, act, norm, stream);
}
#endif

}  // namespace skv

using namespace skv;

static int check_linear(int M, int N, int K, int mode, act_t act) {
    if (N <= 0 || K <= 0) return fail("skv_linear", "N and K must be positive");
    if (mode < 0 || mode > 3) return fail("skv_linear", "unknown epilogue mode");
    if (mode == MODE_GATED && N % 16 != 0)
        return fail("skv_linear", "a gated weight must have a multiple of 16 rows (gate/up tiles of 8)");
    if ((act & 0xff) >= ACT_COUNT || (act & 0xffffffffLL & ~(0xffLL | ACT_ON_STORE)) || ((act & ACT_ON_STORE) && mode != MODE_STORE) ||
        ((act & 0xff) == ACT_SWIGLU_CLAMP && mode != MODE_GATED))
        return fail("skv_linear", "unknown activation");
    (void)M;
    return 0;
}

// `flag` (may be null): bit 2 (value 4) is raised if a pipeline wait inside a kernel timed out.
// With `scaled_out` (residual-add mode, at most 64 tokens, bfloat16 build) the kernel also leaves what the
// projection after the next norm needs (see NormArgs): the scaled rows, and the rows' sums of squares as
// `partials` [M, partial_stride] with partial_stride >= N/16 rounded up.  With `counter` (one zeroed word, left
// zeroed) it finishes them into `row_scale_out` too.
SKV_EXPORT int skv_linear(const void* a, const void* w, void* out, int M, int N, int K, int mode, act_t act,
                          int* flag, void* scaled_out, const float* gamma_next, float* partials, int partial_stride,
                          float* row_scale_out, float eps_next, unsigned int* counter, cudaStream_t stream) {
    if (M <= 0) return 0;
    if (mode == MODE_STORE_ACT) { mode = MODE_STORE; act |= ACT_ON_STORE; }
    if (int code = check_linear(M, N, K, mode, act)) return code;
    NormArgs norm = {};
    if (scaled_out) {
        if (mode != MODE_ADD_F32) return fail("skv_linear", "a norm is folded into the residual-add mode only");
        if (!gamma_next || !partials || partial_stride < (N + 15) / 16 || (counter && !row_scale_out))
            return fail("skv_linear", "the next norm's weight, room for N/16 partial sums per token and, with a counter, a place for the factors are needed");
        norm.partials = partials;
        norm.partial_stride = partial_stride;
        norm.gamma_next = gamma_next;
        norm.scaled_out = (decltype(norm.scaled_out))scaled_out;
        norm.counter = counter;
        norm.eps_next = eps_next;
        norm.row_scale_out = row_scale_out;
    }
    return launch_linear(a, w, out, M, N, K, mode, act, flag, norm, stream);
}

// The projection after a folded norm: `a` holds rows of (stream * norm weight) in bfloat16, token m reads
// row rows[m] (or m), and the result is multiplied by the row's factor: row_scale[row], or (row_scale null)
// 1 / sqrt(sum of partials[row, :n_partials] / K + eps).  bfloat16 build, at most 64 tokens.
SKV_EXPORT int skv_linear_normed(const void* a, const float* row_scale, const float* partials, int n_partials,
                                 int partial_stride, float eps, const int* rows, const void* w, void* out, int M,
                                 int N, int K, int mode, act_t act, cudaStream_t stream) {
    if (M <= 0) return 0;
    if (mode == MODE_STORE_ACT) { mode = MODE_STORE; act |= ACT_ON_STORE; }
    if (int code = check_linear(M, N, K, mode, act)) return code;
    if (!row_scale && (!partials || n_partials <= 0 || partial_stride < n_partials))
        return fail("skv_linear_normed", "the rows' factors, or their partial sums of squares, are needed");
    NormArgs norm = {};
    if (row_scale) {
        norm.row_scale = row_scale;
    } else {
        norm.partials_in = partials;
        norm.n_partials_in = n_partials;
        norm.stride_in = partial_stride;
        norm.eps_in = eps;
    }
    norm.rows = rows;
    return launch_linear(a, w, out, M, N, K, mode, act, nullptr, norm, stream);
}
