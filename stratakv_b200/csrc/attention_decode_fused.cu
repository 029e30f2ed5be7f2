// Decode attention with its neighbours folded in (bfloat16): rotary encoding of the new
// token's queries and key, the write of that key and value into the paged cache, the
// split-KV attention itself, and the merge of the splits, as one kernel.
//
// It replaces four launches of the unfused path (rope_kv_write_kernel, decode_attention_kernel,
// decode_combine_kernel; in the reference: generate_rope_frequencies, rope_split_half x2, two
// cache-append copies and paged_attention_decode_kernel, src/models/transformer_block.cpp:
// 457-518).  The arithmetic is the same as in elementwise.cu and attention_decode.cu: pairs
// (i, i + head_dim/2) rotate in float with a host-built cos/sin table, queries and keys are
// rounded to bfloat16 once, scores / softmax / output accumulate in float.
//
// The kernel is built around its latency chain, since a decode step gives it little else to
// win: at batch 8 and 2,048 keys a block reads 64 KB.  Over long contexts a warp's own chain counts as much: it copies its own 16 keys
// and values of a chunk and waits for them alone (no block-wide barrier in the loop), looks the cache block up once a group (its rows lie one behind the
// other), keeps two chains of score products and rescales its output only where a maximum was raised.  Before and now, us over caches beyond L2:
// 8 sequences x 32 heads of 128 over 400 / 1,600 keys 16.5 / 47.7 and 12.6 / 34.0 (6.2 TB/s), 64 x 8 shared by 4 35.8 / 97.9 and 29.3 / 72.5.
//  * Keys and values of earlier positions cannot change during the step, so a block starts
//    streaming its piece of the context into shared memory (cp.async, two stages of 128 keys)
//    as soon as it is resident, before it waits for the q|k|v projection in front of it.
//  * After the wait one round of 16-byte loads fetches the queries (and the new key and value in
//    the block that owns the newest position); they are rotated into a shared tile, the new row
//    goes to the cache and straight into the staged keys.  Fragments come from ldmatrix.
//  * The splits of one (sequence, KV head) are the blocks of a thread-block cluster.  Each block
//    pushes its partial (max, sum, output) rows into the shared memory of the block that owns the
//    row, one cluster barrier makes them visible, and the owner merges and writes the row.  No
//    scratch in global memory, no second kernel, no barrier after the merge.
#include "head_size.cuh"

#include <mutex>
#include <vector>

// Two stages of 128 keys and values must fit one block's shared memory, which holds for head sizes up
// to 192; above that this kernel is not built and the separate kernels (elementwise.cu,
// attention_decode.cu) serve, as skv_has_attention_decode_fused() tells the caller.
#if SKV_DTYPE == SKV_BF16 && SKV_HEAD_DIM <= 192

namespace skv {

constexpr int FHD = SKV_HEAD_DIM;
constexpr int FKSTEPS = FHD / 16, FOTILES = FHD / 8;
constexpr int FWIDE = 8, FNARROW = 4;               // warps of a block's two forms (see the launch)
constexpr int FMAX_STAGES = 4;                      // stages per launch: 2 .. FMAX_STAGES (see the launch below)
// Staged rows: ldmatrix reads 16 bytes of each of 8 neighbouring rows at once, which must fall on different banks.
// Rows of whole 128-byte multiples are stored with their 16-byte pieces exchanged (piece ^ (row & 7)), at no cost
// in space; other head sizes get 16 bytes of padding per row.
constexpr bool FSWIZZLED = (FHD * 2) % 128 == 0;
constexpr int FROW = FSWIZZLED ? FHD * 2 : FHD * 2 + 16;
constexpr int FQROW = FHD * 2 + 16;                 // bytes between rows of the query tile and the new rows (padded)
__device__ __forceinline__ uint32_t f_staged(int row, int piece) {          // byte offset of a row's 16-byte piece in a stage
    return (uint32_t)(row * FROW + ((FSWIZZLED ? piece ^ (row & 7) : piece) << 4));
}
constexpr int FPIECES = FHD / 8;                    // 16-byte pieces per row
constexpr int FWARP_BYTES = 2 * 16 * FROW;            // what 16 keys and 16 values, one group per warp, take of a stage
constexpr int FPITCH = FHD + 2;                     // floats per partial row: outputs, max, sum
constexpr int FINBOX_ROWS = 24;                     // >= ceil(16 / blocks) * blocks for 1..8 and 16 blocks

// shared memory, in bytes from the start
constexpr int F_Q_AT = 0;                                           // [16][FQROW] rotated queries
constexpr int F_NEW_AT = F_Q_AT + 16 * FQROW;                       // new key row, new value row
constexpr int F_ANGLES_AT = F_NEW_AT + 2 * FQROW;                   // [FHD/2] (cos, sin)
constexpr int F_INBOX_AT = F_ANGLES_AT + (FHD / 2) * 8;             // [FINBOX_ROWS][FPITCH] floats, written by the cluster
constexpr int FTABLE = 512;                                         // entries of the block table kept in shared memory
constexpr int F_TABLE_AT = F_INBOX_AT + FINBOX_ROWS * FPITCH * 4;   // [FTABLE] ints
constexpr int F_STAGES_AT = (F_TABLE_AT + FTABLE * 4 + 127) / 128 * 128;   // also the warps' merge area after the loop
constexpr int F_SMEM_LIMIT = 227 * 1024;
static_assert(16 * FPITCH * 4 <= 2 * FWARP_BYTES, "the merge area reuses the stages");
static_assert(F_STAGES_AT + 2 * FWIDE * FWARP_BYTES <= F_SMEM_LIMIT, "shared memory");
// Whether two blocks of four warps share an SM's 228 KB (each takes 1 KB besides its own): head sizes up to 160.
constexpr bool FNARROW_PAIRS = 2 * (F_STAGES_AT + 2 * FNARROW * FWARP_BYTES + 1024) <= 228 * 1024;

__device__ __forceinline__ void f_ldmatrix(uint32_t (&r)[4], uint32_t address) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];\n"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(address));
}

__device__ __forceinline__ void f_ldmatrix_trans(uint32_t (&r)[4], uint32_t address) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];\n"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(address));
}

// 16 bytes global -> shared, asynchronously; `bytes` 0 writes zeros instead
__device__ __forceinline__ void f_copy16(uint32_t dst, const void* src, int bytes) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void f_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int PENDING>
__device__ __forceinline__ void f_wait_copies() { asm volatile("cp.async.wait_group %0;\n" ::"n"(PENDING) : "memory"); }

__device__ __forceinline__ void f_cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;\n" ::: "memory"); }
__device__ __forceinline__ void f_cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;\n" ::: "memory"); }
__device__ __forceinline__ uint32_t f_cluster_rank() {
    uint32_t r; asm volatile("mov.u32 %0, %%cluster_ctarank;\n" : "=r"(r)); return r;
}
__device__ __forceinline__ uint32_t f_cluster_size() {
    uint32_t r; asm volatile("mov.u32 %0, %%cluster_nctarank;\n" : "=r"(r)); return r;
}
// the address, in the cluster's shared window, of `local` (a shared address of this block) in block `rank`
__device__ __forceinline__ uint32_t f_remote(uint32_t local, uint32_t rank) {
    uint32_t r; asm volatile("mapa.shared::cluster.u32 %0, %1, %2;\n" : "=r"(r) : "r"(local), "r"(rank)); return r;
}
__device__ __forceinline__ void f_remote_store(uint32_t address, float v) {
    asm volatile("st.shared::cluster.f32 [%0], %1;\n" ::"r"(address), "f"(v) : "memory");
}

__device__ __forceinline__ float f_exp2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

__device__ __forceinline__ uint32_t f_pack(float lo, float hi) {
    const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *(const uint32_t*)&v;
}

// What a design may want done to the new token's queries, key and value before they are used and cached: biases
// (float, [heads * head_dim], [kv_heads * head_dim] twice; null: none) and, with value_norm, each value head divided
// by sqrt(mean(v^2) + value_eps).  row_stride: floats from one token's row of qkv to the next (a row may hold more
// than the queries, keys and values; one of a layer that does not write the cache may hold its queries only).
// qk_norm: every query head and the key head divided by sqrt(mean(.^2) + qk_eps) (head sizes that are powers of two);
// q_temp_every > 0: the queries times 1 + q_temp_coef * ln(floor((position + 1) / q_temp_every) + 1).
struct NewTokenFinish {
    const float* q_bias; const float* k_bias; const float* v_bias;
    int value_norm; float value_eps; int row_stride;
    int qk_norm; float qk_eps; float q_temp_coef; int q_temp_every;
};

__device__ __forceinline__ float4 f_add4(float4 a, const float* bias) {
    const float4 b = *(const float4*)bias;
    return make_float4(a.x + b.x, a.y + b.y, a.z + b.z, a.w + b.w);
}

// Warps of a block.  Above head size 64 a block of eight fills an SM, and where there are more blocks than SMs each wave's start
// and end lie bare: blocks of four warps on stages of 64 keys share an SM in twos, where they fit (head size 128: 8 sequences x 24
// key heads over 430 keys 21 -> 16 us, 64 x 8 over 390 keys 48 -> 35, 64 x 32 over 1,000 keys 277 -> 225; at 192, where one block
// has the SM to itself, four warps lose: 8 x 24 over 430 keys 28 -> 36 us, 32 x 24 over 1,000 156 -> 226).  Long pieces are bound by bytes, so that a last wave of twos that is half empty
// costs more than it hides (16 x 24 over 1,000 keys: 384 blocks are three waves of one and four halves of two, 58 us against 63):
// there the eight warps stay.
static int fused_warps(long long blocks, long long keys, int splits, int sms) {
    const long long waves = (blocks + sms - 1) / sms, pairs = 2 * ((blocks + 2 * sms - 1) / (2 * sms));
    return FNARROW_PAIRS && FHD > 64 && blocks > sms && (10 * pairs <= 11 * waves || keys <= 512 * splits) ? FNARROW : FWIDE;
}

// EXTRAS false: the instantiation without any of the optional steps (nothing of them is compiled in, so the plain
// rotary decoder runs the code it ran before they existed).
// FWARPS: 8, or 4 where blocks of a wide head outnumber the SMs.
template <bool EXTRAS, int FWARPS>
__global__ void __launch_bounds__(FWARPS * 32, FHD <= 64 || FWARPS == FNARROW ? 2 : 1)
decode_attention_fused_kernel(const float* __restrict__ qkv, const float2* __restrict__ cos_sin,
                              __nv_bfloat16* k_cache, __nv_bfloat16* v_cache,
                              const int* __restrict__ block_table, int table_width,
                              const int* __restrict__ ctx_after, __nv_bfloat16* __restrict__ out, int num_heads,
                              int num_kv_heads, int block_size, float scale, int window, int splits, int m_tiles,
                              int write_kv, int block_shift, int stages, const NewTokenFinish finish,
                              const AttentionExtras extras) {
    extern __shared__ __align__(128) unsigned char fused_smem[];
    constexpr int HALF = FHD / 2, FTHREADS = FWARPS * 32;
    constexpr int FCHUNK = FWARPS * 16, FSTAGE_BYTES = FWARPS * FWARP_BYTES;       // keys per stage
    pdl_launch_dependents();
    f_cluster_arrive();                               // "this block is running": waited for before the first remote store
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int g = lane >> 2, tig = lane & 3;
    const int seq = blockIdx.x;
    const int kv_head = blockIdx.y / m_tiles, m_tile = blockIdx.y - kv_head * m_tiles;
    const int split = blockIdx.z;
    const int group_size = num_heads / num_kv_heads;
    const int head0 = kv_head * group_size + m_tile * 16;
    const int rows = min(16, group_size - m_tile * 16);
    const int q_dim = num_heads * FHD, kv_dim = num_kv_heads * FHD;

    // The block table's row goes to shared memory while the context length is on its way, so that the
    // copies below start after one round trip to memory, not two.
    const int* table = block_table + (size_t)seq * table_width;
    int* table_near = (int*)(fused_smem + F_TABLE_AT);
    for (int i = threadIdx.x; i < min(table_width, FTABLE); i += FTHREADS) table_near[i] = table[i];
    const int ctx = ctx_after[seq];
    const int pos = ctx - 1;                          // the new token's position
    const int lo = window > 0 ? max(0, ctx - window) : 0;
    const int first_group = lo >> 4, end_group = (ctx + 15) >> 4;
    const int per_split = (end_group - first_group + splits - 1) / splits;
    const int my_first = first_group + split * per_split;
    const int my_end = min(end_group, my_first + per_split);
    const int n_chunks = my_end > my_first ? (my_end - my_first + FWARPS - 1) / FWARPS : 0;
    const float scale_log2 = scale * 1.4426950408889634f;
    const float cap_log2 = EXTRAS ? extras.softcap * 1.4426950408889634f : 0.0f;
    const float inverse_cap_log2 = EXTRAS && extras.softcap > 0.0f ? 1.0f / cap_log2 : 0.0f;
    const float* token = qkv + (size_t)seq * (EXTRAS ? finish.row_stride : q_dim + 2 * kv_dim);
    const int newest_group = pos >> 4;
    const bool owns_newest = newest_group >= my_first && newest_group < my_end;

    const uint32_t smem = smem_u32(fused_smem);
    float2* angles = (float2*)(fused_smem + F_ANGLES_AT);
    float* inbox = (float*)(fused_smem + F_INBOX_AT);
    // rotation angles of the new position come from a table that the step does not write
    static_assert(FHD / 2 <= FTHREADS, "one angle per thread");
    float2 my_angle = make_float2(1.0f, 0.0f);
    if (cos_sin && threadIdx.x < HALF) my_angle = cos_sin[(size_t)pos * HALF + threadIdx.x];
    __syncthreads();                                  // the table is in shared memory
    auto block_of = [&](int key) {
        const int index = block_shift >= 0 ? key >> block_shift : key / block_size;
        return index < FTABLE ? table_near[index] : table[index];
    };
    auto row_in_block = [&](int key) { return block_shift >= 0 ? key & (block_size - 1) : key % block_size; };

    // Stage this warp's 16 keys and values of chunk c (groups my_first + FWARPS c ...): a warp waits for its own copies alone.  Rows past
    // the context are zero-filled: a masked key has weight 0, and 0 times whatever lay in shared memory need not be 0.
    // A group's rows lie in one cache block, one behind the other: one look-up, and every piece is at a constant distance.
    auto issue_chunk = [&](int c) {
        const int group = my_first + c * FWARPS + warp;
        if (group < my_end) {
            const int key0 = group << 4, live = ctx - key0;
            const size_t base = ((size_t)(block_of(key0) * num_kv_heads + kv_head) * block_size + row_in_block(key0)) * FHD;
            const __nv_bfloat16 *k_from = k_cache + base + lane * 8, *v_from = v_cache + base + lane * 8;
            const uint32_t stage = smem + F_STAGES_AT + (c % stages) * FSTAGE_BYTES + warp * 16 * FROW;
#pragma unroll
            for (int it = 0; it < FHD / 16; ++it) {
                const int i = lane + 32 * it, row = i / FPIECES, piece = i - row * FPIECES;
                const uint32_t dst = stage + f_staged(row, piece);
                f_copy16(dst, k_from + 256 * it, row < live ? 16 : 0);
                f_copy16(dst + FCHUNK * FROW, v_from + 256 * it, row < live ? 16 : 0);
            }
        }
        f_commit();
    };
    // Keys and values of earlier positions were written by earlier steps (and the one row that this step
    // writes is replaced below), so the copies need not wait for the kernel in front.
    for (int c = 0; c < stages; ++c) issue_chunk(c);
    if (EXTRAS) {
        // Biases are weights, which nothing in front writes and which the layers between have pushed out of L2: they are
        // asked into it ahead of the wait, where a load after it (or in each chunk) would wait for HBM by itself.  With that and
        // a chunk's biases read while its keys land, 24 heads of 128 with a bias by distance over 430 / 4,000 keys of 8
        // sequences take 18.1 / 135 us in place of 19.4 / 145.
        auto ask = [&](const float* from, int count) {
            for (int i = 32 * threadIdx.x; i < count + 31; i += 32 * FTHREADS)
                asm volatile("prefetch.global.L2 [%0];" :: "l"(from + min(i, count - 1)));
        };
        if (extras.bias && n_chunks > 0) {
            const int near = min(max(0, pos - ((my_end << 4) - 1)), extras.bias_len - 1);
            const int far = min(pos - max(lo, my_first << 4), extras.bias_len - 1);
            for (int r = 0; r < rows; ++r) ask(extras.bias + (size_t)(head0 + r) * extras.bias_len + near, far - near + 1);
        }
        if (finish.q_bias) ask(finish.q_bias + (size_t)head0 * FHD, rows * FHD);
        if (owns_newest && write_kv && finish.k_bias) ask(finish.k_bias + (size_t)kv_head * FHD, FHD);
        if (owns_newest && write_kv && finish.v_bias) ask(finish.v_bias + (size_t)kv_head * FHD, FHD);
    }
    if (threadIdx.x < HALF) angles[threadIdx.x] = my_angle;
    // query rows that no head fills stay zero
    for (int i = threadIdx.x; i < 16 * FQROW / 16; i += FTHREADS)
        *(uint4*)(fused_smem + F_Q_AT + i * 16) = make_uint4(0u, 0u, 0u, 0u);
    __syncthreads();
    pdl_wait();

    // Queries (and the new key, where this block owns the newest position and the layer writes its cache):
    // item `rows` is the key.  One thread rotates four pairs (d, d + HALF).
    {
        const bool with_key = owns_newest && write_kv;
        const int items = (rows + (with_key ? 1 : 0)) * (HALF / 4);
        size_t new_at = 0;
        if (owns_newest)
            new_at = ((size_t)(block_of(pos) * num_kv_heads + kv_head) * block_size + row_in_block(pos)) * FHD;
        float temperature = 1.0f;
        if (EXTRAS && finish.q_temp_every > 0)
            temperature = 1.0f + finish.q_temp_coef * logf((float)((pos + 1) / finish.q_temp_every) + 1.0f);
        for (int i = threadIdx.x; i < items; i += FTHREADS) {
            const int item = i / (HALF / 4), quad = i - item * (HALF / 4);
            const float* x = item < rows ? token + (size_t)(head0 + item) * FHD : token + q_dim + (size_t)kv_head * FHD;
            float4 a = *(const float4*)(x + 4 * quad), b = *(const float4*)(x + HALF + 4 * quad);
            if (EXTRAS) {
                const float* x_bias = item < rows ? (finish.q_bias ? finish.q_bias + (size_t)(head0 + item) * FHD : nullptr)
                                                  : (finish.k_bias ? finish.k_bias + (size_t)kv_head * FHD : nullptr);
                if (x_bias) { a = f_add4(a, x_bias + 4 * quad); b = f_add4(b, x_bias + HALF + 4 * quad); }
                float factor = item < rows ? temperature : 1.0f;
                if (finish.qk_norm) {
                    // the HALF / 4 threads of a head are neighbours of one warp, all of them here or none (the
                    // launcher admits this for head sizes that are powers of two)
                    const unsigned here = __activemask();
                    float squares = a.x * a.x + a.y * a.y + a.z * a.z + a.w * a.w + b.x * b.x + b.y * b.y + b.z * b.z + b.w * b.w;
#pragma unroll
                    for (int offset = HALF / 8; offset > 0; offset >>= 1) squares += __shfl_xor_sync(here, squares, offset);
                    factor *= 1.0f / sqrtf(squares / (float)FHD + finish.qk_eps);
                }
                a = make_float4(a.x * factor, a.y * factor, a.z * factor, a.w * factor);
                b = make_float4(b.x * factor, b.y * factor, b.z * factor, b.w * factor);
            }
            const float xa[4] = {a.x, a.y, a.z, a.w}, xb[4] = {b.x, b.y, b.z, b.w};
            float first[4], second[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const float2 cs = angles[4 * quad + e];
                first[e] = xa[e] * cs.x - xb[e] * cs.y;          // as rotated() of elementwise.cu
                second[e] = xa[e] * cs.y + xb[e] * cs.x;
            }
            const uint2 low = make_uint2(f_pack(first[0], first[1]), f_pack(first[2], first[3]));
            const uint2 high = make_uint2(f_pack(second[0], second[1]), f_pack(second[2], second[3]));
            unsigned char* row = item < rows ? fused_smem + F_Q_AT + item * FQROW : fused_smem + F_NEW_AT;
            *(uint2*)(row + 8 * quad) = low;
            *(uint2*)(row + 2 * HALF + 8 * quad) = high;
            if (item == rows) {
                *(uint2*)(k_cache + new_at + 4 * quad) = low;
                *(uint2*)(k_cache + new_at + HALF + 4 * quad) = high;
            }
        }
        if (EXTRAS && owns_newest && write_kv && finish.value_norm) {
            // the new value row divided by its root mean square: the first warp holds the row (the launcher
            // admits head sizes up to 128 here), four numbers a lane
            if (warp == 0) {
                float4 v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                if (lane < FHD / 4) {
                    v = *(const float4*)(token + q_dim + kv_dim + (size_t)kv_head * FHD + 4 * lane);
                    if (finish.v_bias) v = f_add4(v, finish.v_bias + (size_t)kv_head * FHD + 4 * lane);
                }
                const float squares = warp_sum(v.x * v.x + v.y * v.y + v.z * v.z + v.w * v.w);
                const float inverse = 1.0f / sqrtf(squares / (float)FHD + finish.value_eps);
                if (lane < FHD / 4) {
                    const uint2 packed = make_uint2(f_pack(v.x * inverse, v.y * inverse), f_pack(v.z * inverse, v.w * inverse));
                    *(uint2*)(v_cache + new_at + 4 * lane) = packed;
                    *(uint2*)(fused_smem + F_NEW_AT + FQROW + 8 * lane) = packed;
                }
            }
        } else if (owns_newest) {
            // the new value row (not rotated); or, for a layer that reads a cache which another layer of this
            // step has written, that row and its key as they now stand in the cache
            for (int i = threadIdx.x; i < (write_kv ? 1 : 2) * (FHD / 4); i += FTHREADS) {
                const int which = write_kv ? 1 : i / (FHD / 4), quad = i % (FHD / 4);
                uint2 packed;
                if (write_kv) {
                    float4 v = *(const float4*)(token + q_dim + kv_dim + (size_t)kv_head * FHD + 4 * quad);
                    if (EXTRAS && finish.v_bias) v = f_add4(v, finish.v_bias + (size_t)kv_head * FHD + 4 * quad);
                    packed = make_uint2(f_pack(v.x, v.y), f_pack(v.z, v.w));
                    *(uint2*)(v_cache + new_at + 4 * quad) = packed;
                } else {
                    packed = *(const uint2*)((which ? v_cache : k_cache) + new_at + 4 * quad);
                }
                *(uint2*)(fused_smem + F_NEW_AT + which * FQROW + 8 * quad) = packed;
            }
        }
    }
    __syncthreads();

    // query fragments: rows g and g+8 are heads head0+g, head0+g+8
    uint32_t qa[FKSTEPS][4];
#pragma unroll
    for (int s = 0; s < FKSTEPS; ++s)
        f_ldmatrix(qa[s], smem + F_Q_AT + ((lane & 7) + ((lane >> 3) & 1) * 8) * FQROW + (16 * s + (lane >> 4) * 8) * 2);

    float o[FOTILES][4];
#pragma unroll
    for (int j = 0; j < FOTILES; ++j) { o[j][0] = o[j][1] = o[j][2] = o[j][3] = 0.0f; }
    float row_max[2] = {-INFINITY, -INFINITY}, row_sum[2] = {0.0f, 0.0f};

    const float *bias_top = nullptr, *bias_bottom = nullptr;     // what the distance takes off the scores of rows g and g + 8
    if (EXTRAS && extras.bias) {
        bias_top = extras.bias + (size_t)(head0 + min(g, rows - 1)) * extras.bias_len;
        bias_bottom = extras.bias + (size_t)(head0 + min(g + 8, rows - 1)) * extras.bias_len;
    }
    for (int c = 0; c < n_chunks; ++c) {
        float bias[2][4];                             // on its way while the chunk lands
        if (EXTRAS && extras.bias) {
            const int away = pos - ((my_first + c * FWARPS + warp) << 4) - 2 * tig;
#pragma unroll
            for (int t = 0; t < 2; ++t)
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const int at = min(max(away - 8 * t - e, 0), extras.bias_len - 1);
                    bias[t][e] = g < rows ? __ldg(bias_top + at) : 0.0f;
                    bias[t][e + 2] = rows > 8 ? __ldg(bias_bottom + at) : 0.0f;
                }
        }
        // chunk c has landed (this thread's part) once all but the stages - 1 groups committed after it are complete
        if (stages == 2) f_wait_copies<1>();
        else if (stages == 3) f_wait_copies<2>();
        else f_wait_copies<3>();
        __syncwarp();                                 // ... and the warp's
        const int group0 = my_first + c * FWARPS;
        const uint32_t stage = smem + F_STAGES_AT + (c % stages) * FSTAGE_BYTES;
        if (newest_group == group0 + warp && newest_group < my_end) {
            // the newest position's row, which the copy fetched as the cache had it before this step
            const int row = pos - (group0 << 4);
            unsigned char* base = fused_smem + F_STAGES_AT + (c % stages) * FSTAGE_BYTES;
            for (int i = lane; i < 2 * FPIECES; i += 32) {
                const int which = i / FPIECES, piece = i - which * FPIECES;
                *(uint4*)(base + which * FCHUNK * FROW + f_staged(row, piece)) =
                    *(const uint4*)(fused_smem + F_NEW_AT + which * FQROW + piece * 16);
            }
            __syncwarp();
        }
        const int group = group0 + warp;
        if (group < my_end) {
            const int j0 = group << 4;
            const uint32_t k_rows = stage + warp * 16 * FROW, v_rows = k_rows + FCHUNK * FROW;
            float s[2][4] = {}, odd[2][4] = {};           // (two chains of products each: every second step)
#pragma unroll
            for (int step = 0; step < FKSTEPS; ++step) {
                uint32_t kb[4];                       // keys 0-7: dims 0-7, 8-15 of the step; keys 8-15 likewise
                f_ldmatrix(kb, k_rows + f_staged((lane & 7) + (lane >> 4) * 8, 2 * step + ((lane >> 3) & 1)));
                mma_bf16_16816(step & 1 ? odd[0] : s[0], qa[step][0], qa[step][1], qa[step][2], qa[step][3], kb[0], kb[1]);
                mma_bf16_16816(step & 1 ? odd[1] : s[1], qa[step][0], qa[step][1], qa[step][2], qa[step][3], kb[2], kb[3]);
            }
#pragma unroll
            for (int e = 0; e < 4; ++e) { s[0][e] += odd[0][e]; s[1][e] += odd[1][e]; }
            float tile_max[2] = {-INFINITY, -INFINITY};
#pragma unroll
            for (int t = 0; t < 2; ++t) {
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const int key = j0 + 8 * t + 2 * tig + (e & 1);
                    float v = (key < ctx && key >= lo) ? s[t][e] * scale_log2 : -INFINITY;
                    if (EXTRAS && extras.bias && v != -INFINITY) v -= bias[t][e];
                    // (capped: in units of log2; a masked score stays -infinity)
                    if (EXTRAS && extras.softcap > 0.0f && v != -INFINITY) v = cap_log2 * tanh_by_exp2(v * inverse_cap_log2);
                    s[t][e] = v;
                    tile_max[e >> 1] = fmaxf(tile_max[e >> 1], v);
                }
            }
            float corr[2];
#pragma unroll
            for (int r = 0; r < 2; ++r) {
                float m = tile_max[r];
                m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 1));
                m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 2));
                const float new_max = fmaxf(row_max[r], m);
                corr[r] = new_max == -INFINITY ? 1.0f : f_exp2(row_max[r] - new_max);
                row_max[r] = new_max;
            }
            // (nothing seen yet: a score of -infinity weighs nothing against any offset, and one that is NaN stays NaN)
            const float offset[2] = {row_max[0] == -INFINITY ? 0.0f : row_max[0], row_max[1] == -INFINITY ? 0.0f : row_max[1]};
            float p[2][4];
#pragma unroll
            for (int t = 0; t < 2; ++t) {
#pragma unroll
                for (int e = 0; e < 4; ++e) p[t][e] = f_exp2(s[t][e] - offset[e >> 1]);
            }
#pragma unroll
            for (int r = 0; r < 2; ++r)
                row_sum[r] = row_sum[r] * corr[r] + p[0][2 * r] + p[0][2 * r + 1] + p[1][2 * r] + p[1][2 * r + 1];
            if (__any_sync(0xffffffffu, corr[0] != 1.0f || corr[1] != 1.0f)) {       // (a maximum was raised)
#pragma unroll
                for (int j = 0; j < FOTILES; ++j) {
                    o[j][0] *= corr[0]; o[j][1] *= corr[0]; o[j][2] *= corr[1]; o[j][3] *= corr[1];
                }
            }
            const uint32_t a0 = f_pack(p[0][0], p[0][1]), a1 = f_pack(p[0][2], p[0][3]);
            const uint32_t a2 = f_pack(p[1][0], p[1][1]), a3 = f_pack(p[1][2], p[1][3]);
#pragma unroll
            for (int j = 0; j < FOTILES; j += 2) {
                uint32_t vb[4];                       // dims 8j..: keys 0-7, 8-15; dims 8j+8..: keys 0-7, 8-15
                f_ldmatrix_trans(vb, v_rows + f_staged((lane & 7) + ((lane >> 3) & 1) * 8, j + (lane >> 4)));
                mma_bf16_16816(o[j], a0, a1, a2, a3, vb[0], vb[1]);
                mma_bf16_16816(o[j + 1], a0, a1, a2, a3, vb[2], vb[3]);
            }
        }
        __syncwarp();                                 // the stage is free
        issue_chunk(c + stages);
    }
    f_wait_copies<0>();
    __syncthreads();

    // the warps' partial rows (outputs, max, sum), in what were the stages
    float* partial = (float*)(fused_smem + F_STAGES_AT);
#pragma unroll
    for (int r = 0; r < 2; ++r) {
        row_sum[r] += __shfl_xor_sync(0xffffffffu, row_sum[r], 1);
        row_sum[r] += __shfl_xor_sync(0xffffffffu, row_sum[r], 2);
    }
    float* mine = partial + (size_t)warp * 16 * FPITCH;
#pragma unroll
    for (int j = 0; j < FOTILES; ++j) {
        mine[g * FPITCH + 8 * j + 2 * tig] = o[j][0];
        mine[g * FPITCH + 8 * j + 2 * tig + 1] = o[j][1];
        mine[(g + 8) * FPITCH + 8 * j + 2 * tig] = o[j][2];
        mine[(g + 8) * FPITCH + 8 * j + 2 * tig + 1] = o[j][3];
    }
    if (tig == 0) {
        mine[g * FPITCH + FHD] = row_max[0];
        mine[g * FPITCH + FHD + 1] = row_sum[0];
        mine[(g + 8) * FPITCH + FHD] = row_max[1];
        mine[(g + 8) * FPITCH + FHD + 1] = row_sum[1];
    }
    __syncthreads();
    f_cluster_wait();                                 // every block of the cluster runs: its shared memory may be written

    // Merge the warps, and push each row to the block that owns it: row r belongs to block r % blocks and
    // lands in that block's inbox at [(r / blocks) * blocks + this block's rank].  What has no maximum has a weight of zero and sums of
    // zero, or sums of NaN, where all of its scores are NaN: those go on into the result.
    const int rank = (int)f_cluster_rank(), blocks = (int)f_cluster_size();
    const uint32_t inbox_local = smem + F_INBOX_AT;
    for (int idx = threadIdx.x; idx < rows * FPITCH; idx += FTHREADS) {
        const int r = idx / FPITCH, d = idx - r * FPITCH;
        float m = -INFINITY;
#pragma unroll
        for (int w = 0; w < FWARPS; ++w) m = fmaxf(m, partial[((size_t)w * 16 + r) * FPITCH + FHD]);
        float value = m;
        if (d != FHD) {
            value = 0.0f;
            const float top = m == -INFINITY ? 0.0f : m;
#pragma unroll
            for (int w = 0; w < FWARPS; ++w) {
                const float* tile = partial + ((size_t)w * 16 + r) * FPITCH;
                value += f_exp2(tile[FHD] - top) * tile[d];        // column FHD+1 (the sums) is weighted the same way
            }
        }
        const int slot = (r / blocks) * blocks + rank;
        f_remote_store(f_remote(inbox_local + (slot * FPITCH + d) * 4, (uint32_t)(r % blocks)), value);
    }
    f_cluster_arrive();
    f_cluster_wait();                                 // the pushes are visible; nobody reads another block from here on

    for (int idx = threadIdx.x; idx < ((rows - rank + blocks - 1) / blocks) * FHD; idx += FTHREADS) {
        const int mine_index = idx / FHD, d = idx - mine_index * FHD;
        const int r = mine_index * blocks + rank;
        const float* slots = inbox + (size_t)mine_index * blocks * FPITCH;
        float m = -INFINITY;
        for (int b = 0; b < blocks; ++b) m = fmaxf(m, slots[b * FPITCH + FHD]);
        const float top = m == -INFINITY ? 0.0f : m;
        float total = 0.0f, sum = 0.0f;
        for (int b = 0; b < blocks; ++b) {
            const float weight = f_exp2(slots[b * FPITCH + FHD] - top);
            total += weight * slots[b * FPITCH + d];
            sum += weight * slots[b * FPITCH + FHD + 1];
        }
        out[((size_t)seq * num_heads + head0 + r) * FHD + d] = __float2bfloat16_rn(
            EXTRAS ? total / sum * gate_factor(extras, seq, head0 + r) * gate_element(extras, seq, head0 + r, FHD, d) : total / sum);
    }
}

// How many clusters like this launch's the GPU runs at once.  A kernel, its shared memory and a device have one answer for good, so it is asked for
// once (0.3 us of the host's time a launch otherwise) and an error of the caller's is not cleared with each launch.
static int f_clusters_at_once(const void* kernel, const cudaLaunchConfig_t& config) {
    struct Known { const void* kernel; size_t smem; int device, count; };
    static std::mutex lock;
    static std::vector<Known> known;                  // (two kernels, two to four stages)
    int device = 0;
    if (cudaGetDevice(&device) != cudaSuccess) return 0;
    std::lock_guard<std::mutex> guard(lock);
    for (const Known& k : known)
        if (k.kernel == kernel && k.smem == config.dynamicSmemBytes && k.device == device) return k.count;
    int count = 0;
    if (cudaOccupancyMaxActiveClusters(&count, kernel, &config) != cudaSuccess) {
        cudaGetLastError();                           // (a refusal is an answer)
        count = 0;
    }
    known.push_back({kernel, config.dynamicSmemBytes, device, count});
    return count;
}

}  // namespace skv

using namespace skv;

// qkv: float [n_seqs, (heads + 2 kv_heads) * head_dim] (the q|k|v projection of each sequence's new
// token); cos_sin: float [positions, head_dim/2, 2] or null; ctx_after[s]: keys cached for sequence s
// once this token's key is in (so the token's position is ctx_after[s] - 1).  splits is 1..8; of 8 the launcher
// makes 16 where that is faster (below).
// The _extras form: rows of qkv are row_stride floats apart (0: exactly queries, keys and values); biases, the
// value norm (value_norm != 0, head sizes up to 128), a bias table by distance and a gate as NewTokenFinish and
// AttentionExtras say, each off when null or 0.
SKV_EXPORT int skv_attention_decode_fused_extras(const float* qkv, int row_stride, const float* cos_sin, void* k_cache,
                                                 void* v_cache, const int* block_table, int table_width,
                                                 const int* ctx_after, void* out, int n_seqs, int num_heads,
                                                 int num_kv_heads, int head_dim, int block_size, float scale, int window,
                                                 int splits, int write_kv, const float* q_bias, const float* k_bias,
                                                 const float* v_bias, int value_norm, float value_eps, const float* bias,
                                                 int bias_len, const float* gate, int gate_stride, int qk_norm,
                                                 float qk_eps, float q_temp_coef, int q_temp_every, float softcap,
                                                 int gate_per_element, cudaStream_t stream) {
    if (n_seqs <= 0) return 0;
    const int row_floats = (num_heads + 2 * num_kv_heads) * head_dim;
    if (row_stride == 0) row_stride = row_floats;
    // (a layer that does not write the cache reads its queries only)
    if (row_stride < (write_kv ? row_floats : num_heads * head_dim) || row_stride % 4 != 0)
        return fail("skv_attention_decode_fused", "a row of qkv must hold its queries, keys and values and be a multiple of 16 bytes");
    if (value_norm && head_dim > 128) return fail("skv_attention_decode_fused", "the value norm is built for head sizes up to 128");
    if (qk_norm && (head_dim & (head_dim - 1)) != 0)
        return fail("skv_attention_decode_fused", "the unit norm of queries and keys is built for head sizes that are powers of two");
    if (q_temp_every < 0 || softcap < 0.0f) return fail("skv_attention_decode_fused", "a temperature's period and a cap must not be negative");
    if ((bias && bias_len <= 0) || (gate && gate_stride < num_heads * (gate_per_element ? head_dim : 1)) || (gate_per_element && !gate))
        return fail("skv_attention_decode_fused", "a bias table needs its length and a gate rows of at least heads numbers (heads * head_dim with a gate per number)");
    if (((uintptr_t)q_bias | (uintptr_t)k_bias | (uintptr_t)v_bias) & 15)
        return fail("skv_attention_decode_fused", "biases must be 16-byte aligned");
    const NewTokenFinish finish = {q_bias, k_bias, v_bias, value_norm, value_eps, row_stride,
                                   qk_norm, qk_eps, q_temp_coef, q_temp_every};
    const AttentionExtras extras = {bias, bias_len, gate, gate_stride, softcap, gate_per_element};
    if (head_dim != FHD) return fail("skv_attention_decode_fused", "this library was built for another head size");
    if (num_heads <= 0 || num_kv_heads <= 0 || num_heads % num_kv_heads != 0)
        return fail("skv_attention_decode_fused", "heads must be a positive multiple of kv heads");
    if (block_size <= 0 || block_size % 16 != 0)
        return fail("skv_attention_decode_fused", "block_size must be a positive multiple of 16");
    if (splits < 1 || splits > 8) return fail("skv_attention_decode_fused", "splits must be 1..8 (one cluster)");
    if (((uintptr_t)k_cache | (uintptr_t)v_cache | (uintptr_t)qkv) & 15)
        return fail("skv_attention_decode_fused", "operands must be 16-byte aligned");
    const int group_size = num_heads / num_kv_heads;
    const int m_tiles = (group_size + 15) / 16;
    const long long most_keys = (long long)table_width * block_size;
    int block_shift = -1;                             // log2 of block_size where it is a power of two
    for (int bit = 4; bit < 31; ++bit)
        if (block_size == (1 << bit)) block_shift = bit;
    static int sm_count = 0;
    if (sm_count == 0) {
        int device = 0, count = 0;
        if (cudaGetDevice(&device) != cudaSuccess ||
            cudaDeviceGetAttribute(&count, cudaDevAttrMultiProcessorCount, device) != cudaSuccess || count <= 0)
            return fail("skv_attention_decode_fused", "cannot read the number of SMs");
        for (auto kernel : {decode_attention_fused_kernel<false, FWIDE>, decode_attention_fused_kernel<true, FWIDE>,
                            decode_attention_fused_kernel<false, FNARROW>, decode_attention_fused_kernel<true, FNARROW>}) {
            cudaError_t status = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, F_SMEM_LIMIT);
            if (status == cudaSuccess) status = cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
            if (status != cudaSuccess) return fail("skv_attention_decode_fused", cudaGetErrorString(status));
        }
        sm_count = count;
    }
    // Two stages of 128 keys let two blocks of head size 64 share an SM.  A block that has an SM to itself, and whose
    // piece of the longest context is at most four stages, fetches the whole piece ahead instead (measured: batch 8 at
    // 2,048 keys gains 3 % that way, while deeper staging of longer pieces loses 10 %).
    const long long blocks = (long long)n_seqs * num_kv_heads * m_tiles * splits;
    const int warps = fused_warps(blocks, most_keys, splits, sm_count), stage_bytes = warps * FWARP_BYTES;
    const bool narrow = warps == FNARROW;
    const long long piece_chunks = (most_keys / splits + warps * 16 - 1) / (warps * 16);
    const int room = (F_SMEM_LIMIT - F_STAGES_AT) / stage_bytes;
    // (a third stage for longer pieces, which two blocks of head size 64 could still share an SM with, gains nothing)
    int stages = 2;
    if (blocks <= sm_count && piece_chunks <= FMAX_STAGES && piece_chunks <= room) stages = (int)(piece_chunks < 2 ? 2 : piece_chunks);
    const size_t smem = (size_t)F_STAGES_AT + (size_t)stages * stage_bytes;
    cudaLaunchConfig_t config = {};
    config.gridDim = dim3(n_seqs, num_kv_heads * m_tiles, splits);
    config.blockDim = dim3(warps * 32);
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
    const bool any_extras = q_bias || k_bias || v_bias || value_norm || bias || gate || row_stride != row_floats ||
                            qk_norm || q_temp_every > 0 || softcap > 0.0f;
    auto kernel = narrow ? (any_extras ? decode_attention_fused_kernel<true, FNARROW> : decode_attention_fused_kernel<false, FNARROW>)
                         : (any_extras ? decode_attention_fused_kernel<true, FWIDE> : decode_attention_fused_kernel<false, FWIDE>);
    // Eight pieces of a long context over few heads leave most of the GPU idle: sixteen, where as many clusters of sixteen run at once as
    // there are (1 sequence of 8,100 tokens, 32 heads over 4: 14 -> 8 us, the step of 22 layers 699 -> 575).
    const long long clusters = (long long)n_seqs * num_kv_heads * m_tiles;
    if (splits == 8 && 16 * clusters <= sm_count && most_keys >= 4096 && (window <= 0 || window >= 4096)) {
        cudaLaunchConfig_t wider = config;
        cudaLaunchAttribute cluster = attributes[0];
        cluster.val.clusterDim.z = 16;
        wider.gridDim.z = 16;
        wider.attrs = &cluster;
        wider.numAttrs = 1;
        const long long chunks = (most_keys / 16 + warps * 16 - 1) / (warps * 16);
        wider.dynamicSmemBytes = (size_t)F_STAGES_AT + (size_t)(chunks <= FMAX_STAGES && chunks <= room ? (chunks < 2 ? 2 : chunks) : 2) * stage_bytes;
        if (f_clusters_at_once((const void*)kernel, wider) >= clusters) {
            splits = 16;
            stages = (int)((wider.dynamicSmemBytes - F_STAGES_AT) / stage_bytes);
            config.gridDim.z = attributes[0].val.clusterDim.z = 16;
            config.dynamicSmemBytes = wider.dynamicSmemBytes;
        }
    }
    const cudaError_t status = cudaLaunchKernelEx(
        &config, kernel, qkv, (const float2*)cos_sin, (__nv_bfloat16*)k_cache,
        (__nv_bfloat16*)v_cache, block_table, table_width, ctx_after, (__nv_bfloat16*)out, num_heads, num_kv_heads,
        block_size, scale, window, splits, m_tiles, write_kv, block_shift, stages, finish, extras);
    if (status != cudaSuccess) return fail("skv_attention_decode_fused", cudaGetErrorString(status));
    return 0;
}

SKV_EXPORT int skv_attention_decode_fused(const float* qkv, const float* cos_sin, void* k_cache, void* v_cache,
                                          const int* block_table, int table_width, const int* ctx_after,
                                          void* out, int n_seqs, int num_heads, int num_kv_heads, int head_dim,
                                          int block_size, float scale, int window, int splits, int write_kv,
                                          cudaStream_t stream) {
    return skv_attention_decode_fused_extras(qkv, 0, cos_sin, k_cache, v_cache, block_table, table_width, ctx_after, out,
                                             n_seqs, num_heads, num_kv_heads, head_dim, block_size, scale, window, splits,
                                             write_kv, nullptr, nullptr, nullptr, 0, 0.0f, nullptr, 0, nullptr, 0, 0, 0.0f, 0.0f, 0,
                                             0.0f, 0, stream);
}

SKV_EXPORT int skv_has_attention_decode_fused() { return 1; }

// Warps that a block of such a step takes on a GPU of `sms` SMs.
SKV_EXPORT int skv_attention_decode_fused_warps(int blocks, int keys, int splits, int sms) { return fused_warps(blocks, keys, splits, sms); }

#else

SKV_EXPORT int skv_attention_decode_fused(const float*, const float*, void*, void*, const int*, int, const int*, void*,
                                          int, int, int, int, int, float, int, int, int, cudaStream_t) {
    return skv::fail("skv_attention_decode_fused",
                     "this kernel exists in the bfloat16 build for head sizes up to 192 only");
}

SKV_EXPORT int skv_attention_decode_fused_extras(const float*, int, const float*, void*, void*, const int*, int, const int*,
                                                 void*, int, int, int, int, int, float, int, int, int, const float*,
                                                 const float*, const float*, int, float, const float*, int, const float*,
                                                 int, int, float, float, int, float, int, cudaStream_t) {
    return skv::fail("skv_attention_decode_fused",
                     "this kernel exists in the bfloat16 build for head sizes up to 192 only");
}

SKV_EXPORT int skv_has_attention_decode_fused() { return 0; }

SKV_EXPORT int skv_attention_decode_fused_warps(int, int, int, int) { return 0; }

#endif
