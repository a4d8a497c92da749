// Gated delta rule: a linear-attention mixer whose memory is one matrix per head.
//
// Per head, with a state S [dim x vdim] in float that a request carries from token to token:
//     S <- g S;   u = beta (v - S^T k);   S <- S + k u^T;   o = S^T q
// where q, k (unit vectors per head, q times `q_scale`) and v come from projections that pass a short
// causal convolution over time and silu; beta = sigmoid(b) and g = exp(-exp(A_log) softplus(a + dt_bias))
// are per head and token.  The read-out sees the token's own write.
//
// Kernels, all float inside:
//   delta_prep        per token and head: convolution over the last `taps` inputs (from the step's rows or, before
//                     the portion's start, from the request's saved tail), silu, unit norms, beta, decay;
//                     delta_prep_rows the same for long steps, 16 tokens a warp
//   delta_tail        per request: the last taps - 1 raw inputs of the portion become the saved tail
//   delta_scan        per (request, head, 32 or 16 value columns): the recurrence over the portion's tokens,
//                     one value column's state spread over eight lanes' registers, inputs staged
//                     through shared memory a chunk of tokens ahead by a warp of its own; delta_step the
//                     same for steps of as many tokens as requests
//   delta_gated_norm  per (token, head): o / rms(o) * w * silu(gate)
//
// A request's state row is [heads][vdim][dim] floats (a column of S is contiguous) followed by the
// convolution tail [taps - 1][channels]; channels are q | k | v in the projection's column order.  A
// portion that starts at position 0 ignores what the row holds.  Every sum's order depends only on the
// token's place in its sequence, so results do not change with how a sequence is cut or batched.
#include "common.cuh"

#define DELTA_PARTS 8            // lanes that share one value column
#define DELTA_COLS 32            // value columns of a block (16 when that fills the GPU better)

// One block per (token, unit): a unit is one query head, one key head (dim channels each) or one value
// head (vdim channels, and the head's beta and decay), so that even a single token spreads over many SMs.
template <typename T, typename TW>
__global__ void __launch_bounds__(128) delta_prep_kernel(
    const T* __restrict__ proj, long ld, const TW* __restrict__ conv_w, const TW* __restrict__ a_log,
    const TW* __restrict__ dt_bias, const float* __restrict__ state, long state_stride, long tail_off,
    const int* __restrict__ tok_req, const int* __restrict__ positions, const int* __restrict__ req_ctx,
    const int* __restrict__ req_slot, float* __restrict__ work, long work_ld,
    int heads, int kv_heads, int dim, int vdim, int taps, float unit_eps, float q_scale) {
    pdl_wait();
    pdl_trigger();
    extern __shared__ float conv_out[];                      // [max(dim, vdim)]
    __shared__ float scratch[32];
    const int t = blockIdx.x, unit = blockIdx.y, tid = threadIdx.x;
    const int qk_cols = kv_heads * dim, hv = heads * vdim;
    const int channels = 2 * qk_cols + hv;
    const bool is_v = unit >= 2 * kv_heads;
    const int first = is_v ? 2 * qk_cols + (unit - 2 * kv_heads) * vdim : unit * dim;
    const int count = is_v ? vdim : dim;
    const int r = tok_req[t], pos = positions[t], ctx = req_ctx[r];
    const float* tail = state + (long)req_slot[r] * state_stride + tail_off;
    const T* row = proj + (long)t * ld;
    float ss = 0.0f;
    for (int i = tid; i < count; i += blockDim.x) {
        const int c = first + i;
        float acc = 0.0f;
        for (int back = taps - 1; back >= 0; --back) {        // oldest input first
            const int p = pos - back;
            if (p < 0) continue;
            const float x = p >= ctx ? to_f32<T>(row[c - (long)back * ld])
                                     : tail[(long)(p - ctx + taps - 1) * channels + c];
            acc += to_f32<TW>(conv_w[(long)c * taps + (taps - 1 - back)]) * x;
        }
        const float y = acc / (1.0f + expf(-acc));
        conv_out[i] = y;
        ss += y * y;
    }
    float* out_row = work + (long)t * work_ld;               // work row: q | k | v | beta | decay | o
    if (!is_v) {
        ss = block_sum(ss, scratch);
        const float f = (unit < kv_heads ? q_scale : 1.0f) / sqrtf(ss + unit_eps);
        for (int i = tid; i < count; i += blockDim.x) out_row[first + i] = conv_out[i] * f;   // each thread its own
        return;
    }
    for (int i = tid; i < count; i += blockDim.x) out_row[first + i] = conv_out[i];
    if (tid == 0) {
        const int h = unit - 2 * kv_heads;
        // two numbers a head and token, and the decay is multiplied up over thousands of tokens: formed in
        // double and rounded once, so that no bias of a float exponential adds up along a sequence
        const double b = (double)to_f32<T>(row[channels + hv + h]);
        const double a = (double)to_f32<T>(row[channels + hv + heads + h]) + (double)to_f32<TW>(dt_bias[h]);
        const double softplus = a > 30.0 ? a : log1p(exp(a));
        out_row[channels + h] = (float)(1.0 / (1.0 + exp(-b)));
        out_row[channels + heads + h] = (float)exp(-exp((double)to_f32<TW>(a_log[h])) * softplus);
    }
}

// The same for prompts with heads of 128 channels on both sides and up to four taps: a warp takes PREP_TOKENS neighbouring
// tokens of one unit, four channels a lane, so the taps are read once, a unit's sum of squares stays in the warp and 16
// tokens' decays (double precision, a thread each) are formed side by side.  A block a (token, unit) takes 96 us for 2048
// tokens of 32 units, most of it blocks coming and going; this takes 42.  Sums in the order of the block's: the four
// groups of 32 channels by themselves, then (0 + 2) + (1 + 3).
#define PREP_TOKENS 16
template <typename T, typename TW>
__global__ void __launch_bounds__(128) delta_prep_rows_kernel(
    const T* __restrict__ proj, long ld, const TW* __restrict__ conv_w, const TW* __restrict__ a_log,
    const TW* __restrict__ dt_bias, const float* __restrict__ state, long state_stride, long tail_off,
    const int* __restrict__ tok_req, const int* __restrict__ positions, const int* __restrict__ req_ctx,
    const int* __restrict__ req_slot, float* __restrict__ work, long work_ld, int n_tokens,
    int heads, int kv_heads, int taps, float unit_eps, float q_scale) {
    pdl_wait();
    pdl_trigger();
    constexpr int D = 128;
    const int lane = threadIdx.x & 31, unit = blockIdx.y * 4 + (threadIdx.x >> 5);
    if (unit >= 2 * kv_heads + heads) return;
    const int t0 = blockIdx.x * PREP_TOKENS, t1 = min(n_tokens, t0 + PREP_TOKENS);
    const int qk_cols = kv_heads * D, hv = heads * D, channels = 2 * qk_cols + hv, first = unit * D + lane;
    const bool is_v = unit >= 2 * kv_heads;
    float w[4][4];                                           // [channel group][tap, oldest first; from 4 - taps on]
#pragma unroll
    for (int e = 0; e < 4; ++e)
#pragma unroll
        for (int k = 0; k < 4; ++k) w[e][k] = k >= 4 - taps ? to_f32<TW>(conv_w[(long)(first + 32 * e) * taps + k - (4 - taps)]) : 0.0f;
#pragma unroll 2
    for (int t = t0; t < t1; ++t) {
        const int r = tok_req[t], pos = positions[t], ctx = req_ctx[r];
        const float* tail = state + (long)req_slot[r] * state_stride + tail_off;
        const T* row = proj + (long)t * ld;
        float y[4], ss[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int c = first + 32 * e;
            float acc = 0.0f;
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const int back = 3 - k, p = pos - back;
                if (back >= taps || p < 0) continue;
                const float x = p >= ctx ? to_f32<T>(row[c - (long)back * ld]) : tail[(long)(p - ctx + taps - 1) * channels + c];
                acc = fmaf(w[e][k], x, acc);
            }
            y[e] = acc / (1.0f + expf(-acc));
            ss[e] = y[e] * y[e];
        }
        float f = 1.0f;
        if (!is_v) {
#pragma unroll
            for (int e = 0; e < 4; ++e) ss[e] = warp_sum(ss[e]);
            f = (unit < kv_heads ? q_scale : 1.0f) / sqrtf((ss[0] + ss[2]) + (ss[1] + ss[3]) + unit_eps);
        }
#pragma unroll
        for (int e = 0; e < 4; ++e) work[(long)t * work_ld + first + 32 * e] = is_v ? y[e] : y[e] * f;
    }
    if (is_v && t0 + lane < t1) {
        const int t = t0 + lane, h = unit - 2 * kv_heads;
        const T* row = proj + (long)t * ld;
        const double b = (double)to_f32<T>(row[channels + hv + h]);
        const double a = (double)to_f32<T>(row[channels + hv + heads + h]) + (double)to_f32<TW>(dt_bias[h]);
        const double softplus = a > 30.0 ? a : log1p(exp(a));
        work[(long)t * work_ld + channels + h] = (float)(1.0 / (1.0 + exp(-b)));
        work[(long)t * work_ld + channels + heads + h] = (float)exp(-exp((double)to_f32<TW>(a_log[h])) * softplus);
    }
}

template <typename T>
__global__ void delta_tail_kernel(const T* __restrict__ proj, long ld, float* __restrict__ state, long state_stride,
                                  long tail_off, const int* __restrict__ req_start, const int* __restrict__ req_ctx,
                                  const int* __restrict__ req_qlen, const int* __restrict__ req_slot, int channels,
                                  int taps) {
    pdl_wait();
    pdl_trigger();
    const int r = blockIdx.y;
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= channels) return;
    const int start = req_start[r], ctx = req_ctx[r], qlen = req_qlen[r];
    float* tail = state + (long)req_slot[r] * state_stride + tail_off;
    // entry j holds the input at position end - (taps - 1) + j; an older entry moves down from j + qlen,
    // which lies above j, so going upwards in place is safe
    for (int j = 0; j < taps - 1; ++j) {
        const int p = ctx + qlen - (taps - 1) + j;
        float x = 0.0f;
        if (p >= ctx) x = to_f32<T>(proj[(long)(start + p - ctx) * ld + c]);
        else if (p >= 0) x = tail[(long)(j + qlen) * channels + c];
        tail[(long)j * channels + c] = x;
    }
}

// One block: one request, one head, COLS value columns.  Thread (col, part) keeps the DPT elements
// d = part * DPT + i of column `col` of S.  The tokens' inputs (k, q of the head, the block's v columns,
// beta, decay, and q . k, which no state enters) come through shared memory in chunks of DELTA_CHUNK tokens, the next
// chunk fetched (cp.async) and its q . k summed by a warp of its own while this one is consumed: the threads that walk
// the recurrence do nothing else, a warp of them being alone on its scheduler.  In shared memory
// a part's k (and q) elements are contiguous and parts are DPT + 4 floats apart, so a thread fetches them
// four at a time without bank conflicts.
// What bounds a long prompt: 2048 tokens, 16 heads of 128 x 128 take 310 us, 151 ns a token.  Without the reads of shared
// memory it would be 242 us, without the sums across lanes 233, without both 200: no part of it alone (sums over the state
// two tokens ahead, a shorter chain with more instructions, took 342).  676 us with the fetches and q . k on the same threads (156 instructions a token and warp, a fifth of the
// time at the barrier behind the two warps that fetched) and one multiply-add an element.
// Registers are kept to what lets two blocks of 32 columns share an SM: several requests' prompts bring more blocks than SMs
// (8 x 100 tokens, 16 heads of 128 x 128: 121 us with one block an SM, 96 with two).
#define DELTA_CHUNK 16

__device__ __forceinline__ void delta_cp16(float* smem, const float* gmem) {
    const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(s), "l"(gmem));
}

__device__ __forceinline__ void delta_cp4(float* smem, const float* gmem) {
    const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(s), "l"(gmem));
}

__device__ __forceinline__ float2 delta_fma2(const float2 a, const float2 b, const float2 c) {
    float2 d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;"
        : "=l"(reinterpret_cast<unsigned long long&>(d))
        : "l"(reinterpret_cast<const unsigned long long&>(a)), "l"(reinterpret_cast<const unsigned long long&>(b)),
          "l"(reinterpret_cast<const unsigned long long&>(c)));
    return d;
}
__device__ __forceinline__ float2 delta_mul2(const float2 a, const float2 b) {
    float2 d;
    asm("mul.rn.f32x2 %0, %1, %2;"
        : "=l"(reinterpret_cast<unsigned long long&>(d))
        : "l"(reinterpret_cast<const unsigned long long&>(a)), "l"(reinterpret_cast<const unsigned long long&>(b)));
    return d;
}

template <int DPT, int COLS>
__global__ void __launch_bounds__(COLS * DELTA_PARTS + 32, COLS == 32 && DPT <= 16 ? 2 : 1) delta_scan_kernel(
    float* __restrict__ work, long work_ld, float* __restrict__ state, long state_stride,
    const int* __restrict__ req_start, const int* __restrict__ req_ctx, const int* __restrict__ req_qlen,
    const int* __restrict__ req_slot, int heads, int kv_heads, int dim, int vdim) {
    static_assert(DPT % 4 == 0, "a thread's elements are fetched four at a time");
    pdl_wait();
    pdl_trigger();
    constexpr int THREADS = COLS * DELTA_PARTS;              // ... that walk the recurrence; 32 more fetch
    constexpr int PART = DPT + 4;                            // floats between parts
    constexpr int KQ = DELTA_PARTS * PART;                   // k (and q) of one token
    constexpr int PER_TOKEN = 2 * KQ + COLS + 4;             // k | q | v COLS | beta | decay | q . k | pad
    extern __shared__ __align__(16) float delta_in[];        // [2][DELTA_CHUNK][PER_TOKEN]
    const int r = blockIdx.x / heads, h = blockIdx.x % heads;
    const int g = h / (heads / kv_heads);
    const bool fetches = threadIdx.x >= THREADS;
    const int part = threadIdx.x & (DELTA_PARTS - 1), col = fetches ? 0 : threadIdx.x / DELTA_PARTS;
    const int j = blockIdx.y * COLS + col;
    const bool live = j < vdim && !fetches;
    const int jj = j < vdim ? j : vdim - 1;                  // idle columns shadow the last one and store nothing
    const int start = req_start[r], qlen = req_qlen[r];
    float* s_col = state + (long)req_slot[r] * state_stride + ((long)h * vdim + jj) * dim;
    const int qk_cols = kv_heads * dim, hv = heads * vdim;
    const int v0 = blockIdx.y * COLS;
    if (dim < DELTA_PARTS * DPT) {                           // the k and q places beyond dim are read: they stay 0
        const int used = (qlen < DELTA_CHUNK ? qlen : 2 * DELTA_CHUNK) * PER_TOKEN;
        for (int idx = threadIdx.x; idx < used; idx += blockDim.x) delta_in[idx] = 0.0f;
        __syncthreads();
    }
    // k and q, and the block's v, are copied four floats at a time where their pieces are all 16-byte aligned, else one at a
    // time; either way a lane keeps its place in the row and walks the tokens (a place worked out per element left the
    // recurrence waiting for this warp: 2048 tokens of a head in rows of 514 floats took 2264 us and take 384)
    const bool wide = dim % 4 == 0 && vdim % 4 == 0 && work_ld % 4 == 0 && ((uintptr_t)work & 15) == 0;
    const bool wide_v = wide && v0 + COLS <= vdim;
    auto fetch = [&](int buf, int first) {                   // tokens first .. first + DELTA_CHUNK - 1 of the portion
        float* dst = delta_in + (long)buf * DELTA_CHUNK * PER_TOKEN;
        const int n_tok = min(DELTA_CHUNK, qlen - first);
        const float* row = work + (long)(start + first) * work_ld;
        const int lane = threadIdx.x & 31;
        if (wide) {
            for (int d = lane * 4; d < dim; d += 128) {                           // k and q, four elements a lane
                const float* src = row + g * dim + d;
                float* to = dst + (d / DPT) * PART + d % DPT;
                for (int n = 0; n < n_tok; ++n, src += work_ld, to += PER_TOKEN) {
                    delta_cp16(to, src + qk_cols);
                    delta_cp16(to + KQ, src);
                }
            }
        } else {
            for (int d = lane; d < dim; d += 32) {
                const float* src = row + g * dim + d;
                float* to = dst + (d / DPT) * PART + d % DPT;
#pragma unroll 2
                for (int n = 0; n < n_tok; ++n, src += work_ld, to += PER_TOKEN) {
                    delta_cp4(to, src + qk_cols);
                    delta_cp4(to + KQ, src);
                }
            }
        }
        const int v_lanes = wide_v ? COLS / 4 : COLS;        // lanes with a piece of v each, then beta, decay
        for (int p = lane; p < v_lanes + 2; p += 32) {
            const bool is_v = p < v_lanes;
            const int e = p - v_lanes, c = wide_v ? p * 4 : p;
            const float* src = row + 2 * qk_cols + (is_v ? h * vdim + min(v0 + c, vdim - 1) : hv + e * heads + h);
            float* to = dst + 2 * KQ + (is_v ? c : COLS + e);
#pragma unroll 2
            for (int n = 0; n < n_tok; ++n, src += work_ld, to += PER_TOKEN) {
                if (is_v && wide_v) delta_cp16(to, src);
                else delta_cp4(to, src);
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    // q . k of the chunk's tokens, a token's eight parts side by side
    auto products = [&](int buf, int first) {
        const int n_tok = min(DELTA_CHUNK, qlen - first);
        for (int n0 = 0; n0 < n_tok; n0 += 4) {
            const int n = n0 + ((threadIdx.x & 31) >> 3);
            float* tok = delta_in + ((long)buf * DELTA_CHUNK + min(n, n_tok - 1)) * PER_TOKEN;
            float c[2] = {0.0f, 0.0f};
#pragma unroll
            for (int i = 0; i < DPT; i += 4) {
                const float4 kv = *reinterpret_cast<const float4*>(tok + part * PART + i);
                const float4 qv = *reinterpret_cast<const float4*>(tok + KQ + part * PART + i);
                c[0] = fmaf(qv.x, kv.x, c[0]);
                c[1] = fmaf(qv.y, kv.y, c[1]);
                c[0] = fmaf(qv.z, kv.z, c[0]);
                c[1] = fmaf(qv.w, kv.w, c[1]);
            }
            float qk = c[0] + c[1];
#pragma unroll
            for (int o = 1; o < DELTA_PARTS; o <<= 1) qk += __shfl_xor_sync(0xffffffffu, qk, o);
            if (part == 0 && n < n_tok) tok[2 * KQ + COLS + 2] = qk;
        }
    };
    if (fetches) {
        fetch(0, 0);
        for (int first = 0, buf = 0; first < qlen; first += DELTA_CHUNK, buf ^= 1) {
            asm volatile("cp.async.wait_group 0;" ::: "memory");
            __syncwarp();
            products(buf, first);
            __syncthreads();                                 // chunk `first` is there, the one before has been consumed
            if (first + DELTA_CHUNK < qlen) fetch(buf ^ 1, first + DELTA_CHUNK);
        }
        return;
    }
    float2 S[DPT / 2];
    const bool fresh = req_ctx[r] == 0;
#pragma unroll
    for (int i = 0; i < DPT; ++i) {
        const int d = part * DPT + i;
        const float v = (!fresh && d < dim) ? s_col[d] : 0.0f;
        if (i & 1) S[i / 2].y = v;
        else S[i / 2].x = v;
    }
    float* o_tok = work + (long)start * work_ld + 2 * qk_cols + hv + 2 * heads + h * vdim + j;
    for (int first = 0, buf = 0; first < qlen; first += DELTA_CHUNK, buf ^= 1) {
        __syncthreads();
        const float* in = delta_in + (long)buf * DELTA_CHUNK * PER_TOKEN;
        const int n_tok = min(DELTA_CHUNK, qlen - first);
        // With a = S^T k, b = S^T q (S before the token) and c = q . k:  u = beta (v - g a) and the read-out of the updated
        // state is g b + c u.  Only u stands between this token's sums and the next token's: the next token's inputs are
        // fetched, and the state is multiplied by its decay, while the sums cross the column's lanes.
        float4 kn[DPT / 4], qn[DPT / 4], sn;
        float vn;
        auto ask = [&](const float* tok) {
#pragma unroll
            for (int i = 0; i < DPT / 4; ++i) {
                kn[i] = *reinterpret_cast<const float4*>(tok + part * PART + 4 * i);
                qn[i] = *reinterpret_cast<const float4*>(tok + KQ + part * PART + 4 * i);
            }
            vn = tok[2 * KQ + col];
            sn = *reinterpret_cast<const float4*>(tok + 2 * KQ + COLS);           // beta, decay, q . k
        };
        ask(in);
#pragma unroll 2
        for (int n = 0; n < n_tok; ++n) {
            float2 k[DPT / 2], a = make_float2(0.0f, 0.0f), b = make_float2(0.0f, 0.0f);
#pragma unroll
            for (int i = 0; i < DPT / 4; ++i) {
                k[2 * i] = make_float2(kn[i].x, kn[i].y);
                k[2 * i + 1] = make_float2(kn[i].z, kn[i].w);
                a = delta_fma2(S[2 * i], k[2 * i], a);
                b = delta_fma2(S[2 * i], make_float2(qn[i].x, qn[i].y), b);
                a = delta_fma2(S[2 * i + 1], k[2 * i + 1], a);
                b = delta_fma2(S[2 * i + 1], make_float2(qn[i].z, qn[i].w), b);
            }
            float dot = a.x + a.y, read = b.x + b.y;
            const float v = vn;
            const float4 sc = sn;
            if (n + 1 < n_tok) in += PER_TOKEN;
            ask(in);
#pragma unroll
            for (int o = 1; o < DELTA_PARTS; o <<= 1) {
                dot += __shfl_xor_sync(0xffffffffu, dot, o);
                read += __shfl_xor_sync(0xffffffffu, read, o);
            }
            const float2 decay2 = make_float2(sc.y, sc.y);
#pragma unroll
            for (int i = 0; i < DPT / 2; ++i) S[i] = delta_mul2(decay2, S[i]);
            const float u = __fmul_rn(sc.x, fmaf(-sc.y, dot, v));
            const float2 u2 = make_float2(u, u);
#pragma unroll
            for (int i = 0; i < DPT / 2; ++i) S[i] = delta_fma2(k[i], u2, S[i]);
            if (live && part == 0) *o_tok = fmaf(sc.y, read, sc.z * u);
            o_tok += work_ld;
        }
    }
    if (live) {
#pragma unroll
        for (int i = 0; i < DPT; ++i) {
            const int d = part * DPT + i;
            if (d < dim) s_col[d] = i & 1 ? S[i / 2].y : S[i / 2].x;
        }
    }
}

// The same for steps of as many tokens as requests, all of which bring one token as a rule: reading and writing the state is
// all the work then.  (Requests that bring none and others that bring several are walked token by token.)  A
// thread asks for its elements of S first (16 bytes at a time where every column starts on 16 bytes), k and q come
// through shared memory meanwhile.  (8 and 16 requests, 16 heads of 128 x 128: 6.5 and 9.8 us, through the scan's chunk
// stages 7.0 and 11.3.)
template <int DPT>
__global__ void __launch_bounds__(DELTA_COLS * DELTA_PARTS) delta_step_kernel(
    float* __restrict__ work, long work_ld, float* __restrict__ state, long state_stride,
    const int* __restrict__ req_start, const int* __restrict__ req_ctx, const int* __restrict__ req_qlen,
    const int* __restrict__ req_slot, int heads, int kv_heads, int dim, int vdim) {
    pdl_wait();
    pdl_trigger();
    constexpr int PART = DPT + 4, KQ = DELTA_PARTS * PART;   // as in the scan
    __shared__ __align__(16) float kq_s[2 * KQ];
    const int r = blockIdx.x / heads, h = blockIdx.x % heads;
    const int part = threadIdx.x & (DELTA_PARTS - 1), j = blockIdx.y * DELTA_COLS + threadIdx.x / DELTA_PARTS;
    const int jj = min(j, vdim - 1);                         // idle columns shadow the last one and store nothing
    const int qk_cols = kv_heads * dim, hv = heads * vdim, g = h / (heads / kv_heads);
    float* row = work + (long)req_start[r] * work_ld;
    float* s_col = state + (long)req_slot[r] * state_stride + ((long)h * vdim + jj) * dim;
    const bool fresh = req_ctx[r] == 0;
    const bool whole = dim == DELTA_PARTS * DPT && state_stride % 4 == 0 && ((uintptr_t)state & 15) == 0;
    float S[DPT];
    if (whole) {
#pragma unroll
        for (int i = 0; i < DPT; i += 4) {
            const float4 v = fresh ? make_float4(0.0f, 0.0f, 0.0f, 0.0f) : *reinterpret_cast<const float4*>(s_col + part * DPT + i);
            S[i] = v.x; S[i + 1] = v.y; S[i + 2] = v.z; S[i + 3] = v.w;
        }
    } else {
#pragma unroll
        for (int i = 0; i < DPT; ++i) {
            const int d = part * DPT + i;
            S[i] = (!fresh && d < dim) ? s_col[d] : 0.0f;
        }
    }
    const int qlen = req_qlen[r];
    for (int n = 0; n < qlen; ++n, row += work_ld) {
        if (n > 0) __syncthreads();                          // the token before has been read
        for (int i = threadIdx.x; i < 2 * DELTA_PARTS * DPT; i += DELTA_COLS * DELTA_PARTS) {       // k, then q
            const int side = i / (DELTA_PARTS * DPT), d = i - side * (DELTA_PARTS * DPT);
            kq_s[side * KQ + (d / DPT) * PART + d % DPT] = d < dim ? row[(side == 0 ? qk_cols : 0) + g * dim + d] : 0.0f;
        }
        const float v = row[2 * qk_cols + h * vdim + jj], beta = row[2 * qk_cols + hv + h], decay = row[2 * qk_cols + hv + heads + h];
        __syncthreads();
        float k[DPT], a[2] = {0.0f, 0.0f}, b[2] = {0.0f, 0.0f}, c[2] = {0.0f, 0.0f};
#pragma unroll
        for (int i = 0; i < DPT; i += 4) {
            const float4 kv = *reinterpret_cast<const float4*>(kq_s + part * PART + i);
            const float4 qv = *reinterpret_cast<const float4*>(kq_s + KQ + part * PART + i);
            k[i] = kv.x; k[i + 1] = kv.y; k[i + 2] = kv.z; k[i + 3] = kv.w;
            const float q[4] = {qv.x, qv.y, qv.z, qv.w};
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                a[e & 1] = fmaf(S[i + e], k[i + e], a[e & 1]);
                b[e & 1] = fmaf(S[i + e], q[e], b[e & 1]);
                c[e & 1] = fmaf(q[e], k[i + e], c[e & 1]);
            }
        }
        float dot = a[0] + a[1], read = b[0] + b[1], qk = c[0] + c[1];
#pragma unroll
        for (int o = 1; o < DELTA_PARTS; o <<= 1) {
            dot += __shfl_xor_sync(0xffffffffu, dot, o);
            read += __shfl_xor_sync(0xffffffffu, read, o);
            qk += __shfl_xor_sync(0xffffffffu, qk, o);
        }
        const float u = __fmul_rn(beta, fmaf(-decay, dot, v));
        if (part == 0 && j < vdim) row[2 * qk_cols + hv + 2 * heads + h * vdim + j] = fmaf(decay, read, qk * u);
#pragma unroll
        for (int i = 0; i < DPT; ++i) S[i] = fmaf(k[i], u, __fmul_rn(decay, S[i]));
    }
    if (j >= vdim) return;
    if (whole) {
#pragma unroll
        for (int i = 0; i < DPT; i += 4)
            *reinterpret_cast<float4*>(s_col + part * DPT + i) = make_float4(S[i], S[i + 1], S[i + 2], S[i + 3]);
    } else {
#pragma unroll
        for (int i = 0; i < DPT; ++i)
            if (part * DPT + i < dim) s_col[part * DPT + i] = S[i];
    }
}

// out[t, h, :] = o[t, h, :] / rms(o[t, h, :]) * w * silu(gate[t, h, :]); one warp per (token, head).
template <typename T, typename TW>
__global__ void __launch_bounds__(128) delta_gated_norm_kernel(const float* __restrict__ o, long o_ld, const T* __restrict__ gate,
                                                               long gate_ld, const TW* __restrict__ w, T* __restrict__ out,
                                                               long out_ld, int heads, int vdim, float eps) {
    pdl_wait();
    pdl_trigger();
    const int t = blockIdx.x, lane = threadIdx.x & 31;
    const int h = blockIdx.y * 4 + (threadIdx.x >> 5);
    if (h >= heads) return;
    const float* x = o + (long)t * o_ld + h * vdim;
    const T* gr = gate + (long)t * gate_ld + h * vdim;
    T* dst = out + (long)t * out_ld + h * vdim;
    float ss = 0.0f;
    for (int i = lane; i < vdim; i += 32) ss += x[i] * x[i];
    ss = warp_sum(ss);
    const float inv = 1.0f / sqrtf(ss / (float)vdim + eps);
    for (int i = lane; i < vdim; i += 32) {
        const float z = to_f32<T>(gr[i]);
        dst[i] = from_f32<T>(x[i] * inv * to_f32<TW>(w[i]) * (z / (1.0f + expf(-z))));
    }
}

// proj: [n_tokens, ld] with columns q | k | v | gate | b | a.
FL_API int fl_delta_prep(const void* proj, int dtype, long ld, const void* conv_w, const void* a_log, const void* dt_bias,
                         int w_dtype, float* state, long state_stride, long tail_off, const int* tok_req,
                         const int* positions, const int* req_start, const int* req_ctx, const int* req_qlen,
                         const int* req_slot, float* work, long work_ld, int n_tokens, int n_requests,
                         int heads, int kv_heads, int dim, int vdim, int taps, float unit_eps, float q_scale,
                         cudaStream_t stream) {
    if (n_tokens <= 0) return 0;
    const int channels = 2 * kv_heads * dim + heads * vdim;
    const int units = 2 * kv_heads + heads, widest = dim > vdim ? dim : vdim;
    if (taps < 1 || heads % kv_heads || n_requests > 65535 || units > 65535 || (size_t)widest * sizeof(float) > 48 * 1024)
        return (int)cudaErrorInvalidValue;
    int rc = 0;
    // A warp takes some 37 us for its 16 tokens however few warps there are; a block a (token, unit) takes 3 us and 1.4 ns for
    // each: with 32 units 16 us for 256 tokens, 27 for 512, 50 for 1024 and 96 for 2048 (the warps 37, 38, 38 and 42).
    if (dim == 128 && vdim == 128 && taps <= 4 && (long)n_tokens * units >= 24000)
        FL_DISPATCH(dtype, T, FL_DISPATCH(w_dtype, TW,
            rc = fl_launch(delta_prep_rows_kernel<T, TW>, dim3((n_tokens + PREP_TOKENS - 1) / PREP_TOKENS, (units + 3) / 4), dim3(128), 0,
                           stream, (const T*)proj, ld, (const TW*)conv_w, (const TW*)a_log, (const TW*)dt_bias, (const float*)state,
                           state_stride, tail_off, tok_req, positions, req_ctx, req_slot, work, work_ld, n_tokens, heads, kv_heads,
                           taps, unit_eps, q_scale)))
    else
        FL_DISPATCH(dtype, T, FL_DISPATCH(w_dtype, TW,
            rc = fl_launch(delta_prep_kernel<T, TW>, dim3(n_tokens, units), dim3(128), (size_t)widest * sizeof(float), stream,
                       (const T*)proj, ld, (const TW*)conv_w, (const TW*)a_log, (const TW*)dt_bias, (const float*)state,
                       state_stride, tail_off, tok_req, positions, req_ctx, req_slot, work, work_ld, heads, kv_heads,
                       dim, vdim, taps, unit_eps, q_scale)))
    if (rc || taps == 1) return rc;
    FL_DISPATCH(dtype, T,
        return fl_launch(delta_tail_kernel<T>, dim3((channels + 255) / 256, n_requests), dim3(256), 0, stream,
                         (const T*)proj, ld, state, state_stride, tail_off, req_start, req_ctx, req_qlen, req_slot,
                         channels, taps));
    return 0;
}

// single_tokens: the step has as many tokens as requests, one each as a rule (a kernel of its own).
// work: [n_tokens, work_ld] floats, a row = q | k (kv_heads x dim each) | v (heads x vdim) | beta | decay (heads
// each) | o (heads x vdim): fl_delta_prep fills all but o, fl_delta_scan reads them and fills o.
FL_API int fl_delta_scan(float* work, long work_ld, float* state, long state_stride,
                         const int* req_start, const int* req_ctx, const int* req_qlen, const int* req_slot,
                         int n_requests, int heads, int kv_heads, int dim, int vdim, int single_tokens, cudaStream_t stream) {
    if (n_requests <= 0) return 0;
    if (heads % kv_heads || dim < 1 || dim > 32 * DELTA_PARTS) return (int)cudaErrorInvalidValue;
    const int per_thread = (dim + DELTA_PARTS - 1) / DELTA_PARTS;
    // a block takes 32 value columns, or 16 when blocks of 32 would leave most of the GPU idle (a lone
    // request's prompt): the recurrence is a chain per token, so what counts is how many SMs walk it
    const bool narrow = (long)n_requests * heads * ((vdim + 31) / 32) < 96 && vdim > 16;
    const int cols = narrow ? 16 : DELTA_COLS;
    dim3 grid(n_requests * heads, (vdim + cols - 1) / cols);
    if (grid.y > 65535) return (int)cudaErrorInvalidValue;
#define FL_DELTA_SCAN_COLS(DPT, COLS)                                                                               \
    {                                                                                                               \
        const size_t smem = (size_t)2 * DELTA_CHUNK * (2 * DELTA_PARTS * (DPT + 4) + COLS + 4) * sizeof(float);     \
        static bool raised = false;                                                                                 \
        if (smem > 48 * 1024 && !raised) {                                                                          \
            const cudaError_t rc = cudaFuncSetAttribute(delta_scan_kernel<DPT, COLS>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem); \
            if (rc != cudaSuccess) return (int)rc;                                                                  \
            raised = true;                                                                                          \
        }                                                                                                           \
        return fl_launch(delta_scan_kernel<DPT, COLS>, grid, dim3(COLS * DELTA_PARTS + 32), smem, stream, work, work_ld, state, \
                         state_stride, req_start, req_ctx, req_qlen, req_slot, heads, kv_heads, dim, vdim);         \
    }
#define FL_DELTA_SCAN(DPT)                                                                                          \
    if (per_thread <= DPT) {                                                                                        \
        if (single_tokens)                                                                                          \
            return fl_launch(delta_step_kernel<DPT>, dim3(grid.x, (vdim + DELTA_COLS - 1) / DELTA_COLS), dim3(DELTA_COLS * DELTA_PARTS), 0, \
                             stream, work, work_ld, state, state_stride, req_start, req_ctx, req_qlen, req_slot, heads, kv_heads, dim, vdim); \
        if (narrow) FL_DELTA_SCAN_COLS(DPT, 16) else FL_DELTA_SCAN_COLS(DPT, 32)                                    \
    }
    FL_DELTA_SCAN(4);
    FL_DELTA_SCAN(8);
    FL_DELTA_SCAN(12);
    FL_DELTA_SCAN(16);
    FL_DELTA_SCAN(24);
    FL_DELTA_SCAN(32);
#undef FL_DELTA_SCAN_COLS
#undef FL_DELTA_SCAN
    return (int)cudaErrorInvalidValue;
}

FL_API int fl_delta_gated_norm(const float* o, long o_ld, const void* gate, int dtype, long gate_ld, const void* w, int w_dtype,
                               void* out, long out_ld, int n_tokens, int heads, int vdim, float eps, cudaStream_t stream) {
    if (n_tokens <= 0) return 0;
    dim3 grid(n_tokens, (heads + 3) / 4);
    if (grid.y > 65535) return (int)cudaErrorInvalidValue;
    FL_DISPATCH(dtype, T, FL_DISPATCH(w_dtype, TW,
        return fl_launch(delta_gated_norm_kernel<T, TW>, grid, dim3(128), 0, stream, o, o_ld, (const T*)gate, gate_ld,
                         (const TW*)w, (T*)out, out_ld, heads, vdim, eps)));
    return 0;
}
