// The real-gated linear recurrent unit of a Griffin-style recurrent block, over packed steps of several sequences.
//
// The block's two input projections arrive as one float matrix yx [tokens, row_stride]: channels 0 .. C-1 are the
// gate branch before its bias and activation, channels x_offset .. x_offset + C-1 the recurrent branch before its
// bias.  Per channel c and position p of a sequence:
//
//   xb_p  = x_p + x_bias                                   u_p = conv_b + sum_k conv_w[c, k] * xb_(p - (taps-1-k))
//   r, i  = sigmoid(block-diagonal matrices on u + biases)  (the matrix products are headwise_linear's)
//   a     = exp(-8 * r * softplus(lam))                     S_p = a * S_(p-1) + sqrt(1 - a^2) * i * u_p
//   out_p = S_p * gelu_tanh(y_p + y_bias)                   (compute dtype: the input of the output projection)
//
// Everything here is float.  Per sequence the cache keeps float state, one row per slot:
//   [2][C]     S after the last position, in the half chosen by that position's parity: a step reads the half of
//              the position before its first and writes the half of its last, so a one-token step that runs twice
//              (a graph's capture after its warm-up) computes the same thing both times;
//   [taps][C]  xb of the last `taps` positions, at row (position mod taps): a one-token step writes the row that
//              none of its own taps reads.
// Positions before a sequence's start count as zero input and zero state.
#include "common.cuh"

namespace skv {

constexpr float RGLRU_DECAY_SCALE = 8.0f;

struct RecurrentBatch {
    const int* positions;      // [tokens]
    const int* token_seq;      // [tokens]
    const int* cu_q;           // [seqs + 1]
    const int* slot_ids;       // [seqs]
    float* state;              // [slots][state_stride]
    int state_stride;          // floats per slot: (2 + taps) * C
};

// u[t, c]: a block row per token (what is known per token is looked up once a block), threads over the channels.
__global__ void __launch_bounds__(256)
rglru_conv_kernel(const float* __restrict__ yx, int row_stride, int x_offset, const float* __restrict__ x_bias,
                  const float* __restrict__ conv_w, const float* __restrict__ conv_b, float* __restrict__ u,
                  int first_token, int channels, int taps, const RecurrentBatch batch) {
    pdl_launch_dependents();
    pdl_wait();
    const int t = first_token + blockIdx.y, c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= channels) return;
    const int p = batch.positions[t], s = batch.token_seq[t];
    const int first = batch.cu_q[s];
    const float* ring = batch.state + (size_t)batch.slot_ids[s] * batch.state_stride + 2 * (size_t)channels;
    const float bias = x_bias[c];
    float sum = conv_b[c];
    for (int k = 0; k < taps; ++k) {
        const int back = taps - 1 - k;
        if (p - back < 0) continue;
        const float v = t - back >= first ? yx[(size_t)(t - back) * row_stride + x_offset + c] + bias
                                          : ring[(size_t)((p - back) % taps) * channels + c];
        sum = fmaf(conv_w[(size_t)c * taps + k], v, sum);
    }
    u[(size_t)t * channels + c] = sum;
}

// The same for four taps, four neighbouring channels and eight tokens a thread (channels a multiple of 4, rows 16-byte aligned): a
// row is read once for its four uses and the weights once for eight tokens.  Bound by bytes for many tokens, where the kernel above
// waited on four loads of one number each: 4,000 tokens of 2,048 channels 62 us there, 15 here.
constexpr int RGLRU_CONV_TOKENS = 8;
__global__ void __launch_bounds__(128)
rglru_conv_wide_kernel(const float* __restrict__ yx, int row_stride, int x_offset, const float* __restrict__ x_bias,
                       const float* __restrict__ conv_w, const float* __restrict__ conv_b, float* __restrict__ u,
                       int first_token, int n_tokens, int channels, const RecurrentBatch batch) {
    constexpr int TOK = RGLRU_CONV_TOKENS;
    const int c = 4 * (blockIdx.x * blockDim.x + threadIdx.x), t0 = first_token + blockIdx.y * TOK;
    if (c >= channels) return;
    const float4 bias = *(const float4*)(x_bias + c), begin = *(const float4*)(conv_b + c);
    float4 w[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) w[i] = *(const float4*)(conv_w + 4 * (size_t)(c + i));
    pdl_launch_dependents();
    pdl_wait();
    float4 x[TOK + 3];
#pragma unroll
    for (int i = 0; i < TOK + 3; ++i) {
        const int t = min(max(t0 + i - 3, 0), n_tokens - 1);
        const float4 v = *(const float4*)(yx + (size_t)t * row_stride + x_offset + c);
        x[i] = make_float4(v.x + bias.x, v.y + bias.y, v.z + bias.z, v.w + bias.w);
    }
#pragma unroll
    for (int i = 0; i < TOK; ++i) {
        const int t = t0 + i;
        if (t >= n_tokens) break;
        const int p = batch.positions[t], s = batch.token_seq[t], first = batch.cu_q[s];
        float4 sum = begin;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const int back = 3 - k;
            if (p - back < 0) continue;
            float4 v = x[i + k];
            if (t - back < first)
                v = *(const float4*)(batch.state + (size_t)batch.slot_ids[s] * batch.state_stride + (size_t)(2 + ((p - back) & 3)) * channels + c);
            sum.x = fmaf(k == 0 ? w[0].x : k == 1 ? w[0].y : k == 2 ? w[0].z : w[0].w, v.x, sum.x);
            sum.y = fmaf(k == 0 ? w[1].x : k == 1 ? w[1].y : k == 2 ? w[1].z : w[1].w, v.y, sum.y);
            sum.z = fmaf(k == 0 ? w[2].x : k == 1 ? w[2].y : k == 2 ? w[2].z : w[2].w, v.z, sum.z);
            sum.w = fmaf(k == 0 ? w[3].x : k == 1 ? w[3].y : k == 2 ? w[3].z : w[3].w, v.w, sum.w);
        }
        *(float4*)(u + (size_t)t * channels + c) = sum;
    }
}

__device__ __forceinline__ float sigmoid_f(float z) { return 1.0f / (1.0f + expf(-z)); }
__device__ __forceinline__ float softplus_f(float z) { return z > 20.0f ? z : log1pf(expf(z)); }

// rate[c] = 8 * softplus(lam[c]): the part of the decay's exponent that does not depend on the token, made once when
// the weights are loaded.
__global__ void rglru_rate_kernel(const float* __restrict__ lam, float* __restrict__ rate, int channels) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c < channels) rate[c] = RGLRU_DECAY_SCALE * softplus_f(lam[c]);
}

// Per (token, channel): from the gates' matrix products (gates [tokens, 2C]: per part of `part` channels first the
// part's r rows, then its i rows) to the decay a and the driven input sqrt(1 - a^2) * i * u, which replace them in
// place; and the gate branch's activation in place of its pre-activation in yx.
__global__ void __launch_bounds__(256)
rglru_gates_kernel(float* __restrict__ gates, const float* __restrict__ u, float* __restrict__ yx, int row_stride,
                   const float* __restrict__ y_bias, const float* __restrict__ r_bias,
                   const float* __restrict__ i_bias, const float* __restrict__ rate, int n_tokens, int channels,
                   int part) {
    pdl_launch_dependents();
    pdl_wait();
    const long long item = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (item >= (long long)n_tokens * channels) return;
    const int t = (int)(item / channels), c = (int)(item - (long long)t * channels);
    const int b = c / part, within = c - b * part;
    float* pair = gates + (size_t)t * 2 * channels + (size_t)b * 2 * part + within;
    const float r = sigmoid_f(pair[0] + r_bias[c]);
    const float i = sigmoid_f(pair[part] + i_bias[c]);
    const float a = expf(-r * rate[c]);
    pair[0] = a;
    pair[part] = sqrtf(fmaxf(1.0f - a * a, 0.0f)) * i * u[(size_t)t * channels + c];
    float* y = yx + (size_t)t * row_stride + c;
    *y = gelu_tanh(*y + y_bias[c]);
}

// The same four neighbouring channels a thread (channels and parts multiples of 4, rows 16-byte aligned), the weights ahead of
// the wait: 4,000 tokens of 2,048 channels 43 us, 75 above.
__global__ void __launch_bounds__(256)
rglru_gates_wide_kernel(float* __restrict__ gates, const float* __restrict__ u, float* __restrict__ yx, int row_stride,
                        const float* __restrict__ y_bias, const float* __restrict__ r_bias,
                        const float* __restrict__ i_bias, const float* __restrict__ rate, int n_tokens, int channels,
                        int part) {
    const int quads = channels / 4;
    const long long item = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const int t = (int)(item / quads), c = 4 * (int)(item - (long long)t * quads);
    const float4 yb = *(const float4*)(y_bias + c), rb = *(const float4*)(r_bias + c), ib = *(const float4*)(i_bias + c),
                 rt = *(const float4*)(rate + c);
    pdl_launch_dependents();
    pdl_wait();
    if (t >= n_tokens) return;
    const int b = c / part, within = c - b * part;
    float* pair = gates + (size_t)t * 2 * channels + (size_t)b * 2 * part + within;
    float* y = yx + (size_t)t * row_stride + c;
    const float4 r4 = *(const float4*)pair, i4 = *(const float4*)(pair + part), y4 = *(const float4*)y,
                 u4 = *(const float4*)(u + (size_t)t * channels + c);
    auto decay = [](float z, float bias, float scale) { return expf(-sigmoid_f(z + bias) * scale); };
    auto driven = [](float a, float z, float bias, float x) { return sqrtf(fmaxf(1.0f - a * a, 0.0f)) * sigmoid_f(z + bias) * x; };
    const float4 a = make_float4(decay(r4.x, rb.x, rt.x), decay(r4.y, rb.y, rt.y), decay(r4.z, rb.z, rt.z), decay(r4.w, rb.w, rt.w));
    *(float4*)pair = a;
    *(float4*)(pair + part) = make_float4(driven(a.x, i4.x, ib.x, u4.x), driven(a.y, i4.y, ib.y, u4.y), driven(a.z, i4.z, ib.z, u4.z),
                                          driven(a.w, i4.w, ib.w, u4.w));
    *(float4*)y = make_float4(gelu_tanh(y4.x + yb.x), gelu_tanh(y4.y + yb.y), gelu_tanh(y4.z + yb.z), gelu_tanh(y4.w + yb.w));
}

// The recurrence.  A sequence's tokens of this step are cut into chunks of `chunk` tokens and a thread walks one
// chunk of one channel.  With more than one chunk a first pass (rglru_chunk_kernel) leaves for every chunk the product
// A of its decays and the state B that it reaches from zero; the chunk's true first state then follows from the state
// before the step and the (A, B) of the chunks in front: S <- A S + B, chunk by chunk.  So a prompt of thousands of
// tokens is tens of short walks side by side and not one long one.  `summary` is [seqs][max_chunks][2][C] floats.
__global__ void __launch_bounds__(128)
rglru_chunk_kernel(const float* __restrict__ gates, float* __restrict__ summary, int n_seqs, int channels, int part,
                   int chunk, int max_chunks, const int* __restrict__ cu_q) {
    pdl_launch_dependents();
    pdl_wait();
    const int c = blockIdx.x * blockDim.x + threadIdx.x, s = blockIdx.y, k = blockIdx.z;
    if (c >= channels || s >= n_seqs) return;
    const int first = cu_q[s] + k * chunk, last = min(cu_q[s + 1] - 1, first + chunk - 1);
    if (first > last) return;
    const int b = c / part, within = c - b * part;
    const float* pair = gates + (size_t)b * 2 * part + within;
    float A = 1.0f, B = 0.0f;
#pragma unroll 4
    for (int t = first; t <= last; ++t) {
        const float a = pair[(size_t)t * 2 * channels], driven = pair[(size_t)t * 2 * channels + part];
        A *= a;
        B = fmaf(a, B, driven);
    }
    float* mine = summary + ((size_t)s * max_chunks + k) * 2 * channels;
    mine[c] = A;
    mine[channels + c] = B;
}

template <typename T>
__global__ void __launch_bounds__(128)
rglru_scan_kernel(const float* __restrict__ gates, const float* __restrict__ yx, int row_stride, int x_offset,
                  const float* __restrict__ x_bias, T* __restrict__ out, int out_stride, int n_seqs, int channels,
                  int part, int taps, int chunk, int max_chunks, const float* __restrict__ summary,
                  const RecurrentBatch batch) {
    pdl_launch_dependents();
    pdl_wait();
    const int c = blockIdx.x * blockDim.x + threadIdx.x, s = blockIdx.y, k = blockIdx.z;
    if (c >= channels || s >= n_seqs) return;
    const int seq_first = batch.cu_q[s], seq_last = batch.cu_q[s + 1] - 1;
    const int first = seq_first + k * chunk, last = min(seq_last, first + chunk - 1);
    if (first > last) return;
    const int p_first = batch.positions[seq_first], p_last = p_first + (seq_last - seq_first);
    float* state = batch.state + (size_t)batch.slot_ids[s] * batch.state_stride;
    const int b = c / part, within = c - b * part;
    const float* pair = gates + (size_t)b * 2 * part + within;
    float S = p_first > 0 ? state[(size_t)((p_first - 1) & 1) * channels + c] : 0.0f;
    for (int j = 0; j < k; ++j) {                      // through the chunks in front of this one
        const float* theirs = summary + ((size_t)s * max_chunks + j) * 2 * channels;
        S = fmaf(theirs[c], S, theirs[channels + c]);
    }
#pragma unroll 4
    for (int t = first; t <= last; ++t) {
        const float a = pair[(size_t)t * 2 * channels], driven = pair[(size_t)t * 2 * channels + part];
        const float y = yx[(size_t)t * row_stride + c];
        S = fmaf(a, S, driven);
        out[(size_t)t * out_stride + c] = from_float<T>(S * y);
    }
    if (last != seq_last) return;                      // the sequence's last chunk leaves the state
    state[(size_t)(p_last & 1) * channels + c] = S;
    float* ring = state + 2 * (size_t)channels;
    const float bias = x_bias[c];
    for (int back = 0; back < taps && seq_last - back >= seq_first; ++back)
        ring[(size_t)((p_last - back) % taps) * channels + c] = yx[(size_t)(seq_last - back) * row_stride + x_offset + c] + bias;
}

}  // namespace skv

using namespace skv;

static int check_batch(const char* name, const int* positions, const int* token_seq, const int* cu_q,
                       const int* slot_ids, float* state, int state_stride, int channels, int taps) {
    if (!positions || !token_seq || !cu_q || !slot_ids || !state) return fail(name, "the step's metadata and the state are needed");
    if (channels <= 0 || taps <= 0) return fail(name, "channels and taps must be positive");
    if (state_stride < (2 + taps) * channels) return fail(name, "a slot's state is too small: (2 + taps) * channels floats are needed");
    return 0;
}

SKV_EXPORT int skv_rglru_conv(const float* yx, int row_stride, int x_offset, const float* x_bias, const float* conv_w,
                              const float* conv_b, float* u, int n_tokens, int channels, int taps,
                              const int* positions, const int* token_seq, const int* cu_q, const int* slot_ids,
                              float* state, int state_stride, cudaStream_t stream) {
    if (n_tokens <= 0) return 0;
    if (int code = check_batch("skv_rglru_conv", positions, token_seq, cu_q, slot_ids, state, state_stride, channels, taps)) return code;
    if (x_offset < 0 || row_stride < x_offset + channels) return fail("skv_rglru_conv", "a row is shorter than its two branches");
    const RecurrentBatch batch = {positions, token_seq, cu_q, slot_ids, state, state_stride};
    const uintptr_t places = (uintptr_t)yx | (uintptr_t)x_bias | (uintptr_t)conv_w | (uintptr_t)conv_b | (uintptr_t)u | (uintptr_t)state;
    // (fewer tokens leave threads idle that way: 8 of 2,048 channels 2.8 us a number a thread, 3.0 four a thread)
    if (taps == 4 && n_tokens >= RGLRU_CONV_TOKENS * sm_count() && ((channels | row_stride | x_offset | state_stride) & 3) == 0 && (places & 15) == 0) {
        for (int done = 0; done < n_tokens; done += 65535 * RGLRU_CONV_TOKENS) {
            const int rows = (n_tokens - done + RGLRU_CONV_TOKENS - 1) / RGLRU_CONV_TOKENS;
            if (int code = launch_pdl("skv_rglru_conv", rglru_conv_wide_kernel, dim3((channels / 4 + 127) / 128, rows < 65535 ? rows : 65535),
                                      dim3(128), 0, stream, yx, row_stride, x_offset, x_bias, conv_w, conv_b, u, done, n_tokens,
                                      channels, batch))
                return code;
        }
        return 0;
    }
    // (grid.y holds 65,535 rows at most: longer steps go in pieces)
    for (int done = 0; done < n_tokens; done += 65535) {
        const int rows = n_tokens - done < 65535 ? n_tokens - done : 65535;
        if (int code = launch_pdl("skv_rglru_conv", rglru_conv_kernel, dim3((channels + 255) / 256, rows), dim3(256), 0, stream,
                                  yx, row_stride, x_offset, x_bias, conv_w, conv_b, u, done, channels, taps, batch))
            return code;
    }
    return 0;
}

// rate [channels] float = 8 * softplus(lam [channels] float).
SKV_EXPORT int skv_rglru_rate(const float* lam, float* rate, int channels, cudaStream_t stream) {
    if (channels <= 0) return 0;
    rglru_rate_kernel<<<(channels + 255) / 256, 256, 0, stream>>>(lam, rate, channels);
    return check_launch("skv_rglru_rate");
}

// `rate`: what skv_rglru_rate made of the layer's lam.
SKV_EXPORT int skv_rglru_gates(float* gates, const float* u, float* yx, int row_stride, const float* y_bias,
                               const float* r_bias, const float* i_bias, const float* rate, int n_tokens, int channels,
                               int part, cudaStream_t stream) {
    if (n_tokens <= 0) return 0;
    if (channels <= 0 || part <= 0 || channels % part != 0) return fail("skv_rglru_gates", "the channels must split into equal parts");
    if (row_stride < channels) return fail("skv_rglru_gates", "a row is shorter than its channels");
    const long long blocks = ((long long)n_tokens * channels + 255) / 256;
    if (blocks > 0x7fffffffLL) return fail("skv_rglru_gates", "too many tokens in one step");
    const uintptr_t places = (uintptr_t)gates | (uintptr_t)u | (uintptr_t)yx | (uintptr_t)y_bias | (uintptr_t)r_bias | (uintptr_t)i_bias | (uintptr_t)rate;
    if (((channels | part | row_stride) & 3) == 0 && (places & 15) == 0)
        return launch_pdl("skv_rglru_gates", rglru_gates_wide_kernel, dim3((unsigned)((blocks + 3) / 4)), dim3(256), 0, stream, gates, u, yx,
                          row_stride, y_bias, r_bias, i_bias, rate, n_tokens, channels, part);
    return launch_pdl("skv_rglru_gates", rglru_gates_kernel, dim3((unsigned)blocks), dim3(256), 0, stream, gates, u, yx,
                      row_stride, y_bias, r_bias, i_bias, rate, n_tokens, channels, part);
}

constexpr int RGLRU_CHUNK = 64;

// Floats of `summary` that a step whose longest sequence brings max_q_len tokens needs (0: none, it runs as one chunk).
SKV_EXPORT long long skv_rglru_scan_scratch(int n_seqs, int max_q_len, int channels) {
    if (max_q_len <= 2 * RGLRU_CHUNK) return 0;
    return (long long)n_seqs * ((max_q_len + RGLRU_CHUNK - 1) / RGLRU_CHUNK) * 2 * channels;
}

// out [tokens, out_stride] in the compute dtype: S * activated gate branch, the input of the output projection.
// max_q_len: the most tokens a sequence brings; summary: skv_rglru_scan_scratch floats (null where that is 0).
SKV_EXPORT int skv_rglru_scan(const float* gates, const float* yx, int row_stride, int x_offset, const float* x_bias,
                              void* out, int out_stride, int n_seqs, int channels, int part, int taps, int max_q_len,
                              float* summary,
                              const int* positions, const int* token_seq, const int* cu_q, const int* slot_ids,
                              float* state, int state_stride, cudaStream_t stream) {
    if (n_seqs <= 0) return 0;
    if (int code = check_batch("skv_rglru_scan", positions, token_seq, cu_q, slot_ids, state, state_stride, channels, taps)) return code;
    if (part <= 0 || channels % part != 0) return fail("skv_rglru_scan", "the channels must split into equal parts");
    if (n_seqs > 65535) return fail("skv_rglru_scan", "too many sequences in one step");
    if (out_stride < channels) return fail("skv_rglru_scan", "a row of the output is shorter than its channels");
    const RecurrentBatch batch = {positions, token_seq, cu_q, slot_ids, state, state_stride};
    if (max_q_len <= 0) return fail("skv_rglru_scan", "the longest sequence's token count is needed");
    const bool chunked = skv_rglru_scan_scratch(n_seqs, max_q_len, channels) > 0;
    if (chunked && !summary) return fail("skv_rglru_scan", "a step this long needs scratch for its chunks");
    const int chunk = chunked ? RGLRU_CHUNK : max_q_len;
    const int max_chunks = (max_q_len + chunk - 1) / chunk;
    if (max_chunks > 65535) return fail("skv_rglru_scan", "too many tokens of one sequence in one step");
    const dim3 grid((channels + 127) / 128, n_seqs, max_chunks);
    if (chunked)
        if (int code = launch_pdl("skv_rglru_scan", rglru_chunk_kernel, grid, dim3(128), 0, stream, gates, summary, n_seqs,
                                  channels, part, chunk, max_chunks, cu_q))
            return code;
    return launch_pdl("skv_rglru_scan", rglru_scan_kernel<skv_t>, grid, dim3(128), 0,
                      stream, gates, yx, row_stride, x_offset, x_bias, (skv_t*)out, out_stride, n_seqs, channels, part,
                      taps, chunk, max_chunks, (const float*)summary, batch);
}
