// Prefill attention on the 5th-generation tensor cores (bfloat16, head size 64 or 128): causal
// grouped-query flash attention over the paged cache with both matrix products in tcgen05.mma.
//
// It does the arithmetic of attention_prefill.cu (src/layers/attention.cpp:261-338 in the
// reference, which has no prefill kernel at all) with another division of labour.  A block takes
// 128 queries of one head; keys and values come in tiles of 64 positions:
//   warp 0   keys and scores: TMA loads of the Q tile (once) and of K tiles into two stages (a tile
//            is gathered from the cache blocks the sequence's block table names, whose entries the warp holds 32
//            at a time in registers), and S = Q.K^T (128 x 64 x head_dim) into tensor memory, as soon as the softmax
//            has taken the scores of the tile before;
//   warp 1   values and output: TMA loads of V tiles into two stages, and O += P.V
//            (128 x head_dim x 64) into the output accumulator, also in tensor memory; V is used as it lies
//            in the cache (positions x head_dim), as an MN-major operand.
//            Both warps walk their loops whole, and one elected lane issues.  A single issuing thread for
//            both products measured as the limit of the kernel: its four waits and sixteen small tcgen05
//            instructions a tile took 1,800 cycles, more than the softmax of the tile;
//   warps 4-7  one thread per query row: read the scores with tcgen05.ld, mask, 2^x on the
//            special-function unit (scores carry log2 e; scale, offset and sums two numbers an instruction), row sums,
//            probabilities as bfloat16 into tensor memory (the A operand of P.V).  The maximum the
//            exponentials are taken against is raised only when a tile exceeds it by 2^8; only then
//            is the accumulated output rescaled (tcgen05.ld / st), so most tiles never touch it.
//            At the end the output is read once, divided by the row sum and stored.
// The softmax is the long pole (at 2,048 queries behind 6,144 tokens the special-function unit takes an instruction in 55 % of the cycles at head size 64, 50 % at 128), so what
// counts is that two blocks share an SM and hide each other's waits.  Products that take both operands from shared memory read the
// 128 rows of A again for every 64 columns: with probabilities in shared memory too, and for head size 128 one block an SM, a
// tile took 1,150 cycles of shared memory alone.  Probabilities in tensor memory, one buffer of them and of scores and two stages of keys and
// values leave room for two blocks of either head size.  Before and now, us: 32 heads of 64 over 4 key heads, 2,048 tokens 43.4 and 40.1, behind 6,144
// others 227 and 207, 8 x 870 tokens 87 and 79; of 128 over 8, 64 x 384 tokens 358 and 229, 2,048 74.5 and 44.6, behind 6,144 426 and 223
// (1,070 TFLOP/s).  (A block that walks several query tiles measured slower, 8 x 870 tokens 107 against 87.)
// Every mbarrier wait is bounded; on time-out bit 2 (value 4) of the flag word is raised and the block drains.
#include "head_size.cuh"

#if SKV_DTYPE == SKV_BF16 && (SKV_HEAD_DIM == 64 || SKV_HEAD_DIM == 128)

#include <atomic>
#include <cuda.h>
#include <mutex>
#include <unordered_map>
#include <utility>
#include <vector>

namespace skv {

constexpr int AHD = SKV_HEAD_DIM;
constexpr int ACH = AHD / 64;                       // 64-wide (128-byte) chunks of a head
constexpr int ABM = 128, ABN = 64;                  // queries and keys per tile
constexpr int ATHREADS = 256;
constexpr uint32_t AWAIT = 1u << 20;
constexpr uint32_t TILE_BYTES = 128 * 128;          // one 128-row x 128-byte swizzled tile
constexpr uint32_t KV_TILE_BYTES = ABN * 128;       // one 64-row tile of keys or values

__device__ __forceinline__ uint32_t a_smem(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void a_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void a_expect(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void a_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ bool a_wait(uint32_t bar, uint32_t parity, int* flag) {
    for (uint32_t tries = 0; tries < AWAIT; ++tries) {
        uint32_t done;
        asm volatile(
            "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
            : "=r"(done) : "r"(bar), "r"(parity) : "memory");
        if (done) return true;
    }
    if (flag) atomicOr(flag, 4);
    return false;
}
// One lane of a converged warp (the compiler can then keep what the issuing lane computes in uniform registers)
__device__ __forceinline__ bool a_elect() {
    uint32_t chosen;
    asm volatile("{\n .reg .pred p;\n elect.sync _|p, 0xffffffff;\n selp.u32 %0, 1, 0, p;\n}\n" : "=r"(chosen));
    return chosen != 0;
}
__device__ __forceinline__ void a_tma(uint32_t dst, const CUtensorMap* map, int x, int y, uint32_t bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
        ::"r"(dst), "l"(map), "r"(x), "r"(y), "r"(bar) : "memory");
}
// 128-byte-swizzled tile with 128-byte rows; 1024 bytes between groups of 8 rows (see gemm_tcgen05.cu)
__device__ __forceinline__ uint64_t a_desc(uint32_t addr) {
    return (uint64_t)((addr & 0x3FFFFu) >> 4) | ((uint64_t)1 << 16) | ((uint64_t)(1024 >> 4) << 32) |
           ((uint64_t)1 << 46) | ((uint64_t)2 << 61);
}
// kind::f16, float accumulator, bfloat16 operands; b_mn = 1: B is MN-major (rows are the K index)
__device__ __forceinline__ constexpr uint32_t a_idesc(int m, int n, int b_mn) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)b_mn << 16) | ((uint32_t)(n >> 3) << 17) |
           ((uint32_t)(m >> 4) << 24);
}
__device__ __forceinline__ void a_mma(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n"
        ::"r"(d), "l"(a), "l"(b), "r"(idesc), "r"(accumulate) : "memory");
}
// The same with A in tensor memory: a lane a row, two bfloat16 a column
__device__ __forceinline__ void a_mma_tmem(uint32_t d, uint32_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n}\n"
        ::"r"(d), "r"(a), "l"(b), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ __forceinline__ void a_commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void a_ld32(uint32_t taddr, uint32_t (&v)[32]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
        "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
          "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]),
          "=r"(v[16]), "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]),
          "=r"(v[24]), "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
        : "r"(taddr) : "memory");
}
__device__ __forceinline__ float a_exp2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// Two floats as one operand: one instruction multiplies and adds, or adds, both
__device__ __forceinline__ uint64_t a_pair(float lo, float hi) {
    uint64_t v;
    asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "f"(lo), "f"(hi));
    return v;
}
__device__ __forceinline__ void a_split(uint64_t v, float& lo, float& hi) { asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v)); }
__device__ __forceinline__ uint64_t a_fma2(uint64_t a, uint64_t b, uint64_t c) {
    uint64_t d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ uint64_t a_add2(uint64_t a, uint64_t b) {
    uint64_t d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}

__device__ __forceinline__ float a_max3(float a, float b, float c) {
    float y;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(y) : "f"(a), "f"(b), "f"(c));
    return y;
}

__device__ __forceinline__ void a_ld16(uint32_t taddr, uint32_t (&v)[16]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
                 : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
                   "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
                 : "r"(taddr) : "memory");
}
__device__ __forceinline__ void a_cluster_barrier() {
    asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// The address, in the cluster's shared window, of what lies at `local` in block `rank` of the cluster
__device__ __forceinline__ uint32_t a_remote(uint32_t local, uint32_t rank) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(local), "r"(rank));
    return r;
}

__device__ __forceinline__ void a_st8(uint32_t taddr, const uint32_t (&v)[8]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};"
                 ::"r"(taddr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]) : "memory");
}

__device__ __forceinline__ void a_st32(uint32_t taddr, const uint32_t (&v)[32]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
        "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, "
        "%17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};"
        ::"r"(taddr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]),
          "r"(v[8]), "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15]),
          "r"(v[16]), "r"(v[17]), "r"(v[18]), "r"(v[19]), "r"(v[20]), "r"(v[21]), "r"(v[22]), "r"(v[23]),
          "r"(v[24]), "r"(v[25]), "r"(v[26]), "r"(v[27]), "r"(v[28]), "r"(v[29]), "r"(v[30]), "r"(v[31])
        : "memory");
}

// Keys and values come through two stages each, the scores and the probabilities through one buffer.  A stage of keys is free when
// the softmax has taken the scores of its tile, a stage of values (and the buffer of probabilities) when the product after it is complete.
// barriers: Q; K full and V full for each stage; S full/empty, P full/empty
enum { B_Q = 0, B_KF = 1, B_VF = 3, B_SF = 5, B_SE, B_PF, B_PE, B_COUNT };
// Tensor memory, in columns: 64 of scores, AHD of output, 32 of probabilities (two bfloat16 a column); handed out in powers of two.
constexpr uint32_t A_TMEM = 256;
// Two blocks an SM (three of head size 64 fit with 80 registers a thread: 2,048 tokens 48.1 us against 40.1, behind 6,144 others 216 against 207).
// Registers a thread: at launch (what two blocks leave each of their 8 warps), of the issuing warpgroup, of the softmax's.
constexpr int A_BLOCKS = 2, A_REGS = 128, A_REGS_ISSUE = 88, A_REGS_SOFTMAX = 2 * A_REGS - A_REGS_ISSUE;
// The blocks of a cluster may share a query tile's keys; what they tell each other lies where queries, keys and values were.
constexpr int A_MAX_SPLITS = 4, A_INBOX_AT = A_MAX_SPLITS * ABM * 8;
static_assert(A_INBOX_AT + ABM * (AHD + 4 * A_MAX_SPLITS) * 4 <= ACH * TILE_BYTES + 4 * ACH * KV_TILE_BYTES, "the merge takes the place of the queries, keys and values");

// The running maximum a row's exponentials are taken against is only raised when a tile's maximum
// exceeds it by more than this many powers of two; until then the accumulated output (in tensor
// memory) needs no rescaling and probabilities stay below 2^RESCALE_MARGIN.
constexpr float RESCALE_MARGIN = 8.0f;

// EXTRAS false: the instantiation without the bias table and the gate (nothing of them is compiled in).
template <bool EXTRAS>
__global__ void __launch_bounds__(ATHREADS, A_BLOCKS)
prefill_attention_tc_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                            const __grid_constant__ CUtensorMap map_v, const int* __restrict__ block_table,
                            int table_width, const int* __restrict__ cu_q, const int* __restrict__ ctx_after,
                            __nv_bfloat16* __restrict__ out, int num_heads, int num_kv_heads, int block_size,
                            int rows_per_load, float scale, int window, int tiles_per_seq, int* __restrict__ flag,
                            const AttentionExtras extras) {
    extern __shared__ __align__(1024) uint8_t a_raw[];             // (swizzled tiles start at 1024 bytes)
    uint8_t* q_tile = a_raw;                                       // ACH tiles of 128 rows
    uint8_t* k_ring = q_tile + ACH * TILE_BYTES;                   // 2 stages x ACH tiles of 64 rows
    uint8_t* v_ring = k_ring + 2 * ACH * KV_TILE_BYTES;            // the same
    uint64_t* bars = (uint64_t*)(v_ring + 2 * ACH * KV_TILE_BYTES);
    uint32_t* tmem_slot = (uint32_t*)(bars + B_COUNT);
    const uint32_t bar0 = a_smem(bars);
    auto bar = [&](int which, int index = 0) { return bar0 + 8u * (uint32_t)(which + index); };

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    // Heads run fastest (the heads of a KV head work on the same keys at the same time), and the query tiles
    // are handed out last first: under a causal mask the last tile of a prompt has the most keys, and the
    // blocks that start when the first ones have left should be the short ones.
    const int order = (int)(gridDim.y - 1 - blockIdx.y);
    const int seq = order / tiles_per_seq, tile = order - seq * tiles_per_seq;
    const int head = blockIdx.x;
    const int kv_head = head / (num_heads / num_kv_heads);
    pdl_launch_dependents();
    if (a_smem(a_raw) & 1023) {
        if (threadIdx.x == 0 && flag) atomicOr(flag, 4);
        return;
    }
    const int q_begin = cu_q[seq], q_len = cu_q[seq + 1] - q_begin;
    if (tile * ABM >= q_len) return;                               // the whole block leaves together
    const int ctx = ctx_after[seq], ctx_before = ctx - q_len;
    const int last_query = min(q_len, tile * ABM + ABM) - 1;
    const int kv_end = ctx_before + last_query + 1;
    const int kv_lo = window > 0 ? max(0, ctx_before + tile * ABM - window + 1) : 0;
    // The blocks of a cluster share the keys of the query tile.
    const int splits = gridDim.z, split = blockIdx.z;
    const int all_first = kv_lo / ABN, all_tiles = (kv_end + ABN - 1) / ABN - all_first;
    const int first_tile = all_first + all_tiles * split / splits, n_tiles = all_first + all_tiles * (split + 1) / splits - first_tile;

    if (threadIdx.x == 0) {
        a_init(bar(B_Q), 1);
        for (int i = 0; i < 2; ++i) { a_init(bar(B_KF, i), 1); a_init(bar(B_VF, i), 1); }
        a_init(bar(B_SF), 1); a_init(bar(B_SE), 4); a_init(bar(B_PF), 4); a_init(bar(B_PE), 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 2 && a_elect()) {
        for (const CUtensorMap* map : {&map_q, &map_k, &map_v}) asm volatile("prefetch.tensormap [%0];" ::"l"(map) : "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                     ::"r"(a_smem(tmem_slot)), "r"(A_TMEM) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = *tmem_slot;
    const uint32_t tmem_s = tmem, tmem_o = tmem + 64, tmem_p = tmem_o + AHD;
    pdl_wait();                                                    // q and the cache rows come from the kernels before

    // Cache rows of a tile of 64 keys, for the copies of either warp below: the block table's entries come 32 at a time
    // into one register per lane (a look-up per tile by the issuing lane alone would put the latency of a read from
    // global memory into every round of its loop).
    const int* table = block_table + (size_t)seq * table_width;
    int cached_from = -1, cached_entry = 0;
    auto cache_row = [&](int key) {                                    // called by the whole warp
        const int entry = key / block_size;
        if (cached_from < 0 || entry < cached_from || entry >= cached_from + 32) {
            cached_from = entry;
            cached_entry = table[min(entry + lane, table_width - 1)];
        }
        const int block = __shfl_sync(0xffffffffu, cached_entry, entry - cached_from);
        return (block * num_kv_heads + kv_head) * block_size + (key % block_size);
    };
    auto load_tile = [&](int which, int t) {                           // 0: keys, 1: values; tile t of this block
        const int st = t & 1;
        const uint32_t full = bar(which ? B_VF : B_KF, st);
        uint8_t* dst = (which ? v_ring : k_ring) + (size_t)st * ACH * KV_TILE_BYTES;
        const int key0 = (first_tile + t) * ABN;
        const bool issuer = a_elect();
        if (issuer) a_expect(full, ACH * KV_TILE_BYTES);
        for (int r = 0; r < ABN; r += rows_per_load) {
            const int row = cache_row(key0 + r);
            if (issuer) {
                for (int c = 0; c < ACH; ++c)
                    a_tma(a_smem(dst + c * KV_TILE_BYTES + r * 128), which ? &map_v : &map_k, 64 * c, row, full);
            }
        }
        __syncwarp();
    };
    if (warp < 4) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(A_REGS_ISSUE));
        if (warp == 0) {
            // ---- keys and scores: the whole warp walks the loop, one elected lane issues -----------------------
            // For tile i: wait until softmax i - 1 has taken its scores (which also says that its product is complete and its keys' stage
            // free), and for the keys of tile i; issue S = Q . K_i^T; then ask for the keys of tile i + 1.
            if (a_elect()) {
                a_expect(bar(B_Q), ACH * TILE_BYTES);
                for (int c = 0; c < ACH; ++c)
                    a_tma(a_smem(q_tile + c * TILE_BYTES), &map_q, head * AHD + 64 * c, q_begin + tile * ABM, bar(B_Q));
            }
            __syncwarp();
            for (int t = 0; t < 2 && t < n_tiles; ++t) load_tile(0, t);
            constexpr uint32_t idesc_s = a_idesc(ABM, ABN, 0);
            bool ok = a_wait(bar(B_Q), 0, flag);
            for (int i = 0; i < n_tiles && ok; ++i) {
                const int ks = i & 1;
                if (i >= 1) ok = a_wait(bar(B_SE), (i - 1) & 1, flag);
                if (ok) ok = a_wait(bar(B_KF, ks), (i >> 1) & 1, flag);
                if (!ok) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                if (a_elect()) {
#pragma unroll
                    for (int c = 0; c < ACH; ++c) {
                        const uint64_t qd = a_desc(a_smem(q_tile + c * TILE_BYTES));
                        const uint64_t kd = a_desc(a_smem(k_ring + (size_t)(ks * ACH + c) * KV_TILE_BYTES));
#pragma unroll
                        for (int k = 0; k < 4; ++k) a_mma(tmem_s, qd + 2 * k, kd + 2 * k, idesc_s, (c | k) ? 1u : 0u);
                    }
                    a_commit(bar(B_SF));
                }
                __syncwarp();
                if (i >= 1 && i + 1 < n_tiles) load_tile(0, i + 1);
            }
            if (!ok) {
                // a wait gave up: let the copies in flight land (microseconds) before the block may leave
                for (int t = 0; t < 64; ++t) __nanosleep(1000);
            }
        } else if (warp == 1) {
            // ---- values and output products: O += P_j . V_j once the probabilities are in tensor and the values in shared memory; then
            // the values of tile j + 1 are asked for, into the stage of tile j - 1: its product is complete, or the softmax could
            // not have written the probabilities of tile j where those of j - 1 lay.
            constexpr uint32_t idesc_o = a_idesc(ABM, 64, 1);
            for (int t = 0; t < 2 && t < n_tiles; ++t) load_tile(1, t);
            bool ok = true;
            for (int j = 0; j < n_tiles && ok; ++j) {
                const int vs = j & 1;
                ok = a_wait(bar(B_VF, vs), (j >> 1) & 1, flag) && a_wait(bar(B_PF), j & 1, flag);
                if (!ok) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                if (a_elect()) {
#pragma unroll
                    for (int kk = 0; kk < ABN / 16; ++kk) {               // 16 keys per instruction
#pragma unroll
                        for (int c = 0; c < ACH; ++c) {
                            // V tile rows are keys: 16 keys further is 16 x 128 bytes = 128 descriptor units
                            const uint64_t vd = a_desc(a_smem(v_ring + (size_t)(vs * ACH + c) * KV_TILE_BYTES)) + 128 * kk;
                            a_mma_tmem(tmem_o + (uint32_t)(64 * c), tmem_p + (uint32_t)(8 * kk), vd, idesc_o, (j | kk) ? 1u : 0u);
                        }
                    }
                    a_commit(bar(B_PE));                                  // the output holds tiles 0..j; V_j and P_j are free
                }
                __syncwarp();
                if (j >= 1 && j + 1 < n_tiles) load_tile(1, j + 1);
            }
            if (!ok) {
                for (int t = 0; t < 64; ++t) __nanosleep(1000);
            }
        }
    } else {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(A_REGS_SOFTMAX));
        // ---- softmax and output: one thread per query row -----------------------------------------
        const int quarter = warp & 3;
        const int row = quarter * 32 + lane;                          // row of the tile = TMEM lane
        const int q_row = tile * ABM + row;                           // index among the sequence's new tokens
        const int pos = ctx_before + q_row;
        const uint32_t lane_bits = (uint32_t)(quarter * 32) << 16;
        const float scale_log2 = scale * 1.4426950408889634f;
        // with a bias by distance the scores are brought to units of log2 when the bias is taken off them,
        // and what follows multiplies by one
        const float* bias_row = EXTRAS && extras.bias ? extras.bias + (size_t)head * extras.bias_len : nullptr;
        const bool capped = EXTRAS && extras.softcap > 0.0f;
        const float unit = EXTRAS && (bias_row || capped) ? 1.0f : scale_log2;
        const float cap_log2 = capped ? extras.softcap * 1.4426950408889634f : 0.0f;
        const float to_cap = capped ? scale / extras.softcap : 0.0f;
        float used_max = -INFINITY, row_sum = 0.0f;                   // in units of log2, after the scale
        bool ok = true;
        for (int j = 0; j < n_tiles && ok; ++j) {
            const int key0 = (first_tile + j) * ABN;
            ok = a_wait(bar(B_SF), j & 1, flag);
            if (!ok) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            // a row needs masks only in tiles that reach past its own position, past the sequence's end or
            // below its window; everywhere else the raw scores are used as they are
            const bool plain = key0 + ABN - 1 <= pos && key0 + ABN - 1 < ctx && (window == 0 || key0 > pos - window);
            auto visible = [&](int key) { return key <= pos && key < ctx && (window == 0 || key > pos - window); };
            uint32_t v0[32], v1[32];                                  // the row's 64 scores
            a_ld32(tmem_s + lane_bits, v0);
            a_ld32(tmem_s + lane_bits + 32u, v1);
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) a_arrive(bar(B_SE));                     // the scores are in registers
            float sc[ABN];
            if (plain) {
#pragma unroll
                for (int e = 0; e < 32; ++e) { sc[e] = __uint_as_float(v0[e]); sc[32 + e] = __uint_as_float(v1[e]); }
            } else {
#pragma unroll
                for (int e = 0; e < 32; ++e) {
                    sc[e] = visible(key0 + e) ? __uint_as_float(v0[e]) : -INFINITY;
                    sc[32 + e] = visible(key0 + 32 + e) ? __uint_as_float(v1[e]) : -INFINITY;
                }
            }
            if (EXTRAS && bias_row) {
                const int nearest = pos - key0 - (ABN - 1);            // the distance of the tile's last key
                if (nearest >= 0 && pos - key0 < extras.bias_len) {
                    // every distance of the tile lies inside the table: one load and one multiply-add a score
                    const float* at = bias_row + (pos - key0);
#pragma unroll
                    for (int e = 0; e < ABN; ++e) sc[e] = fmaf(sc[e], scale_log2, -__ldg(at - e));
                } else {
#pragma unroll
                    for (int e = 0; e < ABN; ++e) {                    // (a masked score stays -infinity)
                        const int distance = min(max(pos - key0 - e, 0), extras.bias_len - 1);
                        sc[e] = fmaf(sc[e], scale_log2, -__ldg(bias_row + distance));
                    }
                }
            }
            if (capped) {
                // c * tanh(score / c), left in units of log2; with a bias the scores are in those units already.  A masked
                // score must stay -infinity (its tanh would be -1).
                const float into = bias_row ? 1.0f / cap_log2 : to_cap;
#pragma unroll
                for (int e = 0; e < ABN; ++e)
                    sc[e] = sc[e] == -INFINITY ? -INFINITY : cap_log2 * tanh_by_exp2(sc[e] * into);
            }
            float m4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
            for (int e = 0; e < ABN; e += 8) {                         // (three-input maxima: two scores an instruction)
#pragma unroll
                for (int c = 0; c < 4; ++c) m4[c] = a_max3(m4[c], sc[e + 2 * c], sc[e + 2 * c + 1]);
            }
            const float tile_max = fmaxf(fmaxf(m4[0], m4[1]), fmaxf(m4[2], m4[3])) * unit;   // scale > 0
            // raise the maximum in use (and rescale what has been accumulated) only when it matters
            const bool raise = tile_max > used_max + RESCALE_MARGIN;
            // once the product of the previous tile has finished the output accumulator may be touched and the probabilities
            // rewritten, both in tensor memory: the fence orders either behind the wait
            if (j > 0) {
                ok = a_wait(bar(B_PE), (j - 1) & 1, flag);
                if (!ok) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            }
            if (j > 0 && __any_sync(0xffffffffu, raise)) {
                const float corr = raise ? a_exp2(used_max - tile_max) : 1.0f;     // 0 if nothing was seen before
#pragma unroll 1
                for (int c = 0; c < AHD; c += 32) {
                    uint32_t v[32];
                    a_ld32(tmem_o + lane_bits + (uint32_t)c, v);
                    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                    for (int e = 0; e < 32; ++e) v[e] = __float_as_uint(__uint_as_float(v[e]) * corr);
                    a_st32(tmem_o + lane_bits + (uint32_t)c, v);
                }
                asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                row_sum *= corr;
            }
            if (raise) used_max = tile_max;
            const float offset = used_max == -INFINITY ? 0.0f : used_max;      // nothing visible yet: every p is 0
            const uint64_t unit2 = a_pair(unit, unit), offset2 = a_pair(-offset, -offset);
            uint64_t sums[2] = {0ull, 0ull};                            // four running sums, two an addition
#pragma unroll
            for (int piece = 0; piece < ABN / 16; ++piece) {            // 16 keys = 8 columns
                uint32_t packed[8];
#pragma unroll
                for (int e = 0; e < 8; ++e) {
                    // (a masked score is -infinity, the offset is finite and the scale positive: 2^-infinity = 0)
                    float lo, hi;
                    a_split(a_fma2(a_pair(sc[16 * piece + 2 * e], sc[16 * piece + 2 * e + 1]), unit2, offset2), lo, hi);
                    lo = a_exp2(lo);
                    hi = a_exp2(hi);
                    sums[e & 1] = a_add2(sums[e & 1], a_pair(lo, hi));
                    const __nv_bfloat162 pair = __floats2bfloat162_rn(lo, hi);
                    packed[e] = *(const uint32_t*)&pair;
                }
                a_st8(tmem_p + lane_bits + (uint32_t)(8 * piece), packed);
            }
            float s4[4];
            a_split(sums[0], s4[0], s4[1]);
            a_split(sums[1], s4[2], s4[3]);
            row_sum += (s4[0] + s4[1]) + (s4[2] + s4[3]);
            asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) a_arrive(bar(B_PF));                     // probabilities in place (and any rescale done)
        }
        // the last product has finished: read the output once, normalise, store
        if (ok && n_tiles > 0) ok = a_wait(bar(B_PE), (n_tiles - 1) & 1, flag);
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const int token = q_begin + min(q_row, q_len - 1);
        // (a sink has no key and no value and is not scaled; the sums are in units of log2 below used_max)
        const float sink_log2 = EXTRAS && extras.sink ? extras.sink[head] * 1.4426950408889634f : 0.0f;
        const float* gate_row = EXTRAS && extras.gate && extras.gate_per_element
            ? extras.gate + (size_t)token * extras.gate_stride + (size_t)head * AHD : nullptr;
        __nv_bfloat16* dst = out + ((size_t)token * num_heads + head) * AHD;
        const float gate = EXTRAS ? gate_factor(extras, token, head) : 1.0f;
        // eight numbers of the row from column d on, times `by`
        auto store = [&](float (&v)[8], int d, float by) {
            if (EXTRAS && gate_row) {                                  // a gate for every number of the output
#pragma unroll
                for (int e = 0; e < 8; e += 4) {
                    const float4 logit = *(const float4*)(gate_row + d + e);
                    v[e] = __fdividef(v[e], 1.0f + __expf(-logit.x));
                    v[e + 1] = __fdividef(v[e + 1], 1.0f + __expf(-logit.y));
                    v[e + 2] = __fdividef(v[e + 2], 1.0f + __expf(-logit.z));
                    v[e + 3] = __fdividef(v[e + 3], 1.0f + __expf(-logit.w));
                }
            }
            uint32_t packed[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const __nv_bfloat162 pair = __floats2bfloat162_rn(v[2 * e] * by, v[2 * e + 1] * by);
                packed[e] = *(const uint32_t*)&pair;
            }
            *(uint4*)(dst + d) = make_uint4(packed[0], packed[1], packed[2], packed[3]);
        };
        if (splits == 1) {
            if (ok && n_tiles > 0) {
                const float sunk = EXTRAS && extras.sink ? a_exp2(sink_log2 - used_max) : 0.0f;
                const float inverse = gate / (row_sum + sunk);
#pragma unroll 1
                for (int c = 0; c < AHD; c += 32) {
                    uint32_t v[32];
                    a_ld32(tmem_o + lane_bits + (uint32_t)c, v);
                    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                    if (q_row < q_len) {
#pragma unroll
                        for (int d = 0; d < 32; d += 8) {
                            float x[8];
#pragma unroll
                            for (int e = 0; e < 8; ++e) x[e] = __uint_as_float(v[d + e]);
                            store(x, c + d, inverse);
                        }
                    }
                }
            }
        } else {
            // Each block tells the others its rows' maxima and sums, then brings its output to the common maximum and pushes it, by
            // columns, to the blocks that own them (AHD / splits columns each), which add up in rank order and store.  All of it
            // lies where the queries, keys and values were: the first barrier is passed when every block's products are complete.
            float2* rows = (float2*)a_raw;                                // [splits][128] (maximum, sum)
            const uint32_t rows_at = a_smem(rows);
            a_cluster_barrier();                                          // nobody's products read shared memory any more
            for (int to = 0; to < splits; ++to) {
                const uint32_t at = a_remote(rows_at + (uint32_t)(split * ABM + row) * 8u, (uint32_t)to);
                asm volatile("st.shared::cluster.v2.f32 [%0], {%1, %2};" ::"r"(at), "f"(ok ? used_max : -INFINITY), "f"(ok ? row_sum : 0.0f) : "memory");
            }
            a_cluster_barrier();
            float top = -INFINITY, total = 0.0f;
            for (int from = 0; from < splits; ++from) top = fmaxf(top, rows[from * ABM + row].x);
            // (a block none of whose keys the row sees has a sum of zero; one whose visible scores are all NaN has no maximum either, and its
            // sum is NaN, which must reach the result.  So must a value that is not finite, however little it weighs)
            for (int from = 0; from < splits; ++from) {
                const float2 r = rows[from * ABM + row];
                total += r.x != -INFINITY ? a_exp2(r.x - top) * r.y : r.y;
            }
            const float weight = a_exp2(used_max - top);
            const bool sees = ok && used_max != -INFINITY;                // (with no keys the output was never written)
            const int columns = AHD / splits, pitch = columns + 4;        // (the pitch spreads a warp's rows over the banks)
            float* inbox = (float*)(a_raw + A_INBOX_AT);                  // [splits][128][pitch]
            const uint32_t inbox_at = a_smem(inbox);
            for (int c = 0; c < AHD; c += 16) {
                uint32_t v[16];
                if (n_tiles > 0) {
                    a_ld16(tmem_o + lane_bits + (uint32_t)c, v);
                    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                }
                const uint32_t at = a_remote(inbox_at + (uint32_t)((split * ABM + row) * pitch + c % columns) * 4u, (uint32_t)(c / columns));
#pragma unroll
                for (int e = 0; e < 16; e += 4) {
                    float x[4];
#pragma unroll
                    for (int f = 0; f < 4; ++f) x[f] = sees ? __uint_as_float(v[e + f]) * weight : 0.0f;
                    asm volatile("st.shared::cluster.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(at + 4u * e), "f"(x[0]), "f"(x[1]), "f"(x[2]), "f"(x[3]) : "memory");
                }
            }
            a_cluster_barrier();
            if (q_row < q_len) {
                const float sunk = EXTRAS && extras.sink ? a_exp2(sink_log2 - top) : 0.0f;
                const float inverse = gate / (total + sunk);
                for (int d = 0; d < columns; d += 8) {
                    float x[8] = {};
                    for (int from = 0; from < splits; ++from) {
                        const float* at = inbox + (from * ABM + row) * pitch + d;
                        const float4 lo = *(const float4*)at, hi = *(const float4*)(at + 4);
                        x[0] += lo.x; x[1] += lo.y; x[2] += lo.z; x[3] += lo.w;
                        x[4] += hi.x; x[5] += hi.y; x[6] += hi.z; x[7] += hi.w;
                    }
                    store(x, split * columns + d, inverse);
                }
            }
        }
    }
    if (splits > 1 && warp < 4) {
        a_cluster_barrier();
        a_cluster_barrier();
        a_cluster_barrier();
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 1) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(A_TMEM) : "memory");
    }
}

// ---- host side -----------------------------------------------------------------------------------
typedef CUresult (*AEncode)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                            const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                            CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static AEncode a_encoder() {
    static AEncode fn = [] {
        void* entry = nullptr;
        cudaDriverEntryPointQueryResult result;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &entry, cudaEnableDefault, &result) != cudaSuccess ||
            result != cudaDriverEntryPointSuccess)
            entry = nullptr;
        return (AEncode)entry;
    }();
    return fn;
}

// Whether the compiler gave the kernels the registers that their warpgroups share out (the softmax's share is taken from what the block was
// launched with): with another number its request would wait forever, and prompts go to attention_prefill.cu.  Without a GPU nobody can tell.
static bool a_registers_fit() {
    static std::atomic<int> known{-1};
    if (known.load(std::memory_order_relaxed) < 0) {
        cudaFuncAttributes plain, extras;
        if (cudaFuncGetAttributes(&plain, prefill_attention_tc_kernel<false>) != cudaSuccess ||
            cudaFuncGetAttributes(&extras, prefill_attention_tc_kernel<true>) != cudaSuccess) {
            cudaGetLastError();
            return true;
        }
        known.store(plain.numRegs == A_REGS && extras.numRegs == A_REGS, std::memory_order_relaxed);
    }
    return known.load(std::memory_order_relaxed) != 0;
}

// Blocks that share a query tile's keys.  Fewer query tiles than SMs over long contexts (as long as the block tables have room for): their keys are shared
// out, which starts every block for less work and ends in a merge (512 queries behind 4,096 others, 32 heads of 64, 128 blocks: 68.2 -> 44.0 us; 512
// blocks 207 -> 212; from 512 keys on 200 queries behind 800, 24 heads of 128, 16.3 -> 21.7).
static int a_splits(long long query_tiles, int heads, int table_width, int block_size, int window, int sms) {
    const long long most_keys = (long long)table_width * block_size, keys = window > 0 && window + ABM < most_keys ? window + ABM : most_keys;
    int splits = 1;
    while (splits < A_MAX_SPLITS && query_tiles * heads * 2 * splits <= A_BLOCKS * sms && keys >= 1024 * splits) splits *= 2;
    return splits;
}

// bfloat16 matrix [rows, cols] row-major, box of box_rows x 64 columns, 128-byte swizzle
static int a_map(const void* base, long long rows, int cols, int box_rows, CUtensorMap* out) {
    struct Key { const void* base; long long rows; int cols, box; };
    static std::mutex lock;
    static std::vector<std::pair<Key, CUtensorMap>> cache;
    std::lock_guard<std::mutex> guard(lock);
    for (auto& entry : cache)
        if (entry.first.base == base && entry.first.rows == rows && entry.first.cols == cols && entry.first.box == box_rows) {
            *out = entry.second;
            return 0;
        }
    AEncode encode = a_encoder();
    if (!encode) return fail("skv_attention_prefill_tc", "cuTensorMapEncodeTiled is not available from this driver");
    const cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
    const cuuint64_t strides[1] = {(cuuint64_t)cols * 2};
    const cuuint32_t box[2] = {64, (cuuint32_t)box_rows};
    const cuuint32_t elem[2] = {1, 1};
    CUtensorMap map;
    const CUresult status = encode(&map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides, box,
                                   elem, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                                   CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (status != CUDA_SUCCESS) return fail("skv_attention_prefill_tc", "cuTensorMapEncodeTiled failed");
    if (cache.size() > 1024) cache.clear();
    cache.push_back({Key{base, rows, cols, box_rows}, map});
    *out = map;
    return 0;
}

}  // namespace skv

using namespace skv;

// As skv_attention_prefill; cache_blocks is the number of blocks of the layer's cache tensors
// [cache_blocks][kv_heads][block_size][head_dim]; n_tokens the rows of q and out.
// `bias` [num_heads][bias_len] and `gate` (logits, rows gate_stride apart) may be null: see AttentionExtras.
SKV_EXPORT int skv_attention_prefill_tc_extras(const void* q, const void* k_cache, const void* v_cache, int cache_blocks,
                                               const int* block_table, int table_width, const int* cu_q,
                                               const int* ctx_after, void* out, int n_seqs, int n_tokens, int max_q_len,
                                               int num_heads, int num_kv_heads, int head_dim, int block_size, float scale,
                                               int window, const float* bias, int bias_len, const float* gate,
                                               int gate_stride, float softcap, int gate_per_element, const float* sink,
                                               int* flag, cudaStream_t stream) {
    if (n_seqs <= 0 || max_q_len <= 0) return 0;
    if ((bias && bias_len <= 0) || (gate && gate_stride < num_heads * (gate_per_element ? head_dim : 1)) ||
        (gate_per_element && (!gate || gate_stride % 4 != 0 || ((uintptr_t)gate & 15))) || softcap < 0.0f)
        return fail("skv_attention_prefill_tc", "a bias table needs its length, a gate rows of at least heads numbers (with a gate per number: heads * head_dim, 16-byte aligned rows), a cap must not be negative");
    const AttentionExtras extras = {bias, bias_len, gate, gate_stride, softcap, gate_per_element, sink};
    if (head_dim != AHD) return fail("skv_attention_prefill_tc", "this library was built for another head size");
    if (num_heads <= 0 || num_kv_heads <= 0 || num_heads % num_kv_heads != 0)
        return fail("skv_attention_prefill_tc", "heads must be a positive multiple of kv heads");
    if (block_size < 16 || (block_size & (block_size - 1)) != 0)
        return fail("skv_attention_prefill_tc", "block_size must be a power of two, at least 16");
    if (((uintptr_t)q | (uintptr_t)k_cache | (uintptr_t)v_cache | (uintptr_t)out) & 15)
        return fail("skv_attention_prefill_tc", "operands must be 16-byte aligned");
    const int rows_per_load = block_size < ABN ? block_size : ABN;
    CUtensorMap map_q, map_k, map_v;
    if (int code = a_map(q, n_tokens, num_heads * AHD, 128, &map_q)) return code;
    const long long cache_rows = (long long)cache_blocks * num_kv_heads * block_size;
    if (int code = a_map(k_cache, cache_rows, AHD, rows_per_load, &map_k)) return code;
    if (int code = a_map(v_cache, cache_rows, AHD, rows_per_load, &map_v)) return code;
    const int tiles_per_seq = (max_q_len + ABM - 1) / ABM;
    const long long blocks = (long long)n_seqs * tiles_per_seq;
    if (blocks > 65535) return fail("skv_attention_prefill_tc", "too many query tiles in one step (65,535 at most)");
    const size_t smem = (size_t)ACH * TILE_BYTES + (size_t)4 * ACH * KV_TILE_BYTES + B_COUNT * 8 + 16;
    if (!a_registers_fit()) return fail("skv_attention_prefill_tc", "built with another number of registers than the warpgroups share out");
    if (int code = reserve_shared_once<prefill_attention_tc_kernel<false>>("skv_attention_prefill_tc", smem)) return code;
    if (int code = reserve_shared_once<prefill_attention_tc_kernel<true>>("skv_attention_prefill_tc", smem)) return code;
    const int splits = a_splits(blocks, num_heads, table_width, block_size, window, sm_count());
    cudaLaunchConfig_t config = {};
    config.gridDim = dim3(num_heads, (unsigned)blocks, splits);
    config.blockDim = dim3(ATHREADS);
    config.dynamicSmemBytes = smem;
    config.stream = stream;
    cudaLaunchAttribute attributes[2];
    attributes[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attributes[0].val.programmaticStreamSerializationAllowed = pdl_enabled();
    attributes[1].id = cudaLaunchAttributeClusterDimension;
    attributes[1].val.clusterDim.x = attributes[1].val.clusterDim.y = 1;
    attributes[1].val.clusterDim.z = splits;
    config.attrs = attributes;
    config.numAttrs = splits > 1 ? 2 : 1;
    auto kernel = bias || gate || sink || softcap > 0.0f ? prefill_attention_tc_kernel<true> : prefill_attention_tc_kernel<false>;
    const cudaError_t status = cudaLaunchKernelEx(&config, kernel, map_q, map_k, map_v, block_table, table_width, cu_q, ctx_after,
                                                  (__nv_bfloat16*)out, num_heads, num_kv_heads, block_size, rows_per_load, scale, window,
                                                  tiles_per_seq, flag, extras);
    if (status != cudaSuccess) return fail("skv_attention_prefill_tc", cudaGetErrorString(status));
    return 0;
}

SKV_EXPORT int skv_attention_prefill_tc(const void* q, const void* k_cache, const void* v_cache, int cache_blocks,
                                        const int* block_table, int table_width, const int* cu_q,
                                        const int* ctx_after, void* out, int n_seqs, int n_tokens, int max_q_len,
                                        int num_heads, int num_kv_heads, int head_dim, int block_size, float scale,
                                        int window, int* flag, cudaStream_t stream) {
    return skv_attention_prefill_tc_extras(q, k_cache, v_cache, cache_blocks, block_table, table_width, cu_q, ctx_after,
                                           out, n_seqs, n_tokens, max_q_len, num_heads, num_kv_heads, head_dim, block_size,
                                           scale, window, nullptr, 0, nullptr, 0, 0.0f, 0, nullptr, flag, stream);
}

SKV_EXPORT int skv_has_attention_prefill_tc() { return a_registers_fit(); }

// Blocks that share the keys of a query tile of such a call (`query_tiles`: sequences x tiles of 128 of the longest) on a GPU of `sms` SMs.
SKV_EXPORT int skv_attention_prefill_tc_splits(int query_tiles, int heads, int table_width, int block_size, int window, int sms) {
    return a_splits(query_tiles, heads, table_width, block_size, window, sms);
}

#else

SKV_EXPORT int skv_attention_prefill_tc(const void*, const void*, const void*, int, const int*, int, const int*,
                                        const int*, void*, int, int, int, int, int, int, int, float, int, int*,
                                        cudaStream_t) {
    return skv::fail("skv_attention_prefill_tc", "this build (float32, or a head size other than 64 or 128) has no such kernel");
}

SKV_EXPORT int skv_attention_prefill_tc_extras(const void*, const void*, const void*, int, const int*, int, const int*,
                                               const int*, void*, int, int, int, int, int, int, int, float, int,
                                               const float*, int, const float*, int, float, int, const float*, int*,
                                               cudaStream_t) {
    return skv::fail("skv_attention_prefill_tc", "this build (float32, or a head size other than 64 or 128) has no such kernel");
}

SKV_EXPORT int skv_has_attention_prefill_tc() { return 0; }

#endif
