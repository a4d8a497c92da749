// Routed experts: each token's feed-forward is a weighted sum of a few small gated feed-forwards
// chosen by a router.
//
//   moe_pick      per token, from the router's float logits z (a product the caller makes): score
//                 s = sigmoid(z) (or a softmax over the experts); the `top` experts with the largest
//                 s + bias are chosen (the bias steers the choice only), ties to the lower index; the
//                 weights are the chosen s, optionally renormalised to sum 1 (divided by their sum + an
//                 epsilon) and multiplied by `weight_scale`.  With groups, the experts form `n_groups`
//                 equal groups of neighbours, a group's score is the sum of the `group_top` largest
//                 s + bias in it (1: the largest), and only experts of the `keep` best groups (ties to
//                 the lower index) can be chosen
//   moe_gate_up   per (token, choice): act(W_gate[e] h) * (W_up[e] h), a warp a feature or several; experts
//                 without a gate: act(W_up[e] h), the unit's f(x, 1)
//   moe_down      per token: sum over its choices, in order of choice, of weight * W_down[e] a (with
//                 `accumulate` added to what `out` holds: a shared unit's result)
//
// The last two read an expert's matrices once per token that chose it: the right shape for decode
// steps, where tokens are few and the matrices stream from memory.  A token's weight multiplies its expert's output, or
// (weight_on_input) what the expert reads: the gate and up sums then, which are linear in it, before the activation.  All sums are float and depend only
// on the token itself.
#include "tcgen05.cuh"

// One warp per token; z: float logits [n_tokens, experts] (the router's product, made by the caller).
template <typename TW>
__global__ void __launch_bounds__(128) moe_pick_kernel(const float* __restrict__ z, long z_ld, const TW* __restrict__ bias,
                                                       int* __restrict__ chosen, float* __restrict__ weights, int n_tokens,
                                                       int experts, int top, int softmax_scores, int renormalise,
                                                       int n_groups, int keep, float renorm_eps, int group_top,
                                                       float weight_scale) {
    pdl_wait();
    pdl_trigger();
    extern __shared__ float route_s[];                  // per warp: [experts] scores, [experts] scores + bias, [n_groups]
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int t = blockIdx.x * 4 + warp;
    if (t >= n_tokens) return;
    float* score = route_s + (long)warp * (2 * experts + n_groups);
    float* pick = score + experts;
    const float* zr = z + (long)t * z_ld;
    if (softmax_scores) {
        float mx = -CUDART_INF_F;
        for (int e = lane; e < experts; e += 32) mx = fmaxf(mx, zr[e]);
        mx = warp_max(mx);
        float sum = 0.0f;
        for (int e = lane; e < experts; e += 32) sum += expf(zr[e] - mx);
        sum = warp_sum(sum);
        for (int e = lane; e < experts; e += 32) score[e] = expf(zr[e] - mx) / sum;
    } else {
        for (int e = lane; e < experts; e += 32) score[e] = 1.0f / (1.0f + expf(-zr[e]));
    }
    for (int e = lane; e < experts; e += 32) pick[e] = score[e] + (bias ? to_f32<TW>(bias[e]) : 0.0f);
    __syncwarp();
    if (n_groups > 1 && keep < n_groups) {
        const int per = experts / n_groups;
        float* group = pick + experts;
        for (int g = lane; g < n_groups; g += 32) {
            float b = 0.0f, last = CUDART_INF_F;        // the sum of the group's `group_top` largest, in falling order
            int last_at = -1;
            for (int n = 0; n < group_top && n < per; ++n) {
                float best = -CUDART_INF_F;
                int at = per;
                for (int i = 0; i < per; ++i) {
                    const float v = pick[g * per + i];
                    if ((v < last || (v == last && i > last_at)) && v > best) { best = v; at = i; }
                }
                if (at == per) break;
                b += best;
                last = best;
                last_at = at;
            }
            group[g] = b;
        }
        __syncwarp();
        for (int g = lane; g < n_groups; g += 32) {
            const float mine = group[g];
            int ahead = 0;                              // groups that come before this one
            for (int o = 0; o < n_groups; ++o) ahead += (group[o] > mine) || (group[o] == mine && o < g);
            if (ahead >= keep)
                for (int i = 0; i < per; ++i) pick[g * per + i] = -CUDART_INF_F;
        }
        __syncwarp();
    }
    float total = 0.0f;
    for (int k = 0; k < top; ++k) {
        float best = -CUDART_INF_F;
        int at = experts;
        for (int e = lane; e < experts; e += 32)
            if (pick[e] > best) { best = pick[e]; at = e; }
        for (int o = 16; o > 0; o >>= 1) {
            const float ob = __shfl_xor_sync(0xffffffffu, best, o);
            const int oa = __shfl_xor_sync(0xffffffffu, at, o);
            if (ob > best || (ob == best && oa < at)) { best = ob; at = oa; }
        }
        if (at >= experts) at = 0;                      // every remaining score is NaN or -inf
        if (lane == 0) {
            chosen[(long)t * top + k] = at;
            weights[(long)t * top + k] = score[at];
            pick[at] = -CUDART_INF_F;
        }
        total += score[at];
        __syncwarp();
    }
    if (lane == 0)
        for (int k = 0; k < top; ++k) {
            float w = weights[(long)t * top + k];
            if (renormalise) w /= total + renorm_eps;
            weights[(long)t * top + k] = w * weight_scale;
        }
}

// The order of a row's sum x . w, whichever kernel makes it: 32 chains, chain c adding up the elements c, c + 32, ... with
// fused multiply-adds, and the chains added in a tree (neighbours 16 apart first).  The kernels for any size give a warp a
// row and a lane a chain, which fetches 2 bytes a lane: 8 tokens x 4 of 32 experts of 2048 x 1408 took 85 + 62 us a layer,
// bound by the number of loads (57 + 44 by rows).  Where rows are whole blocks of 32 elements and 16-byte aligned, a lane takes
// the MoeRows::V neighbouring chains that 16 bytes hold, 32 / V lanes a row, and a warp several rows at once.
template <typename TW> struct MoeRows {
    static constexpr int V = 16 / (int)sizeof(TW);       // chains a lane
    static constexpr int LPR = 32 / V;                   // lanes a row
    static constexpr int ROWS = 32 / LPR;                // rows a warp
};

// acc[r][v] += x . w of this lane's chains for `ROWS` rows `second` elements apart; x and w begin at the lane's first chain
template <int ROWS, int U, typename TW>
__device__ __forceinline__ void moe_rows_dot(const float* __restrict__ x, const TW* __restrict__ w, long second, int n,
                                             float (&acc)[ROWS][MoeRows<TW>::V]) {
    constexpr int V = MoeRows<TW>::V;
    for (int i = 0; i < n; i += U * 32) {
        uint4 raw[ROWS][U];
#pragma unroll
        for (int j = 0; j < U; ++j)
#pragma unroll
            for (int r = 0; r < ROWS; ++r)
                if (i + j * 32 < n) raw[r][j] = *reinterpret_cast<const uint4*>(w + r * second + i + j * 32);
#pragma unroll
        for (int j = 0; j < U; ++j) {
            if (i + j * 32 >= n) break;
#pragma unroll
            for (int v = 0; v < V; v += 4) {
                const float4 xv = *reinterpret_cast<const float4*>(x + i + j * 32 + v);
#pragma unroll
                for (int r = 0; r < ROWS; ++r) {
                    const TW* e = reinterpret_cast<const TW*>(&raw[r][j]) + v;
                    acc[r][v] = fmaf(xv.x, to_f32<TW>(e[0]), acc[r][v]);
                    acc[r][v + 1] = fmaf(xv.y, to_f32<TW>(e[1]), acc[r][v + 1]);
                    acc[r][v + 2] = fmaf(xv.z, to_f32<TW>(e[2]), acc[r][v + 2]);
                    acc[r][v + 3] = fmaf(xv.w, to_f32<TW>(e[3]), acc[r][v + 3]);
                }
            }
        }
    }
}
// the sum of a row's 32 chains, in every lane of the row
template <int V> __device__ __forceinline__ float moe_rows_sum(float (&acc)[V]) {
#pragma unroll
    for (int o = 16; o >= V; o >>= 1)
#pragma unroll
        for (int v = 0; v < V; ++v) acc[v] += __shfl_xor_sync(0xffffffffu, acc[v], o / V);
#pragma unroll
    for (int o = V / 2; o > 0; o >>= 1)
#pragma unroll
        for (int v = 0; v < o; ++v) acc[v] += acc[v + o];
    return acc[0];
}

// w_gu: [experts][2 ff][width] (gate rows, then up rows), or [experts][ff][width] without a gate;
// a: [tokens x top][ff] float
// U: blocks of 32 elements on their way at once, of each row.  With more warps than the SMs hold at a time, fewer of them
// and more warps resident are faster (8 tokens x 4, both products out of a cold cache: 101 us with 4 and 8, 114 with 8 and
// 11); with fewer warps than that, more (one token: 24.4 us with 8 and 11, 30.7 with 4 and 8).
#define MOE_GU_WARPS 4
template <typename T, typename TW, int U>
__global__ void __launch_bounds__(MOE_GU_WARPS * 32) moe_gate_up_rows_kernel(
    const T* __restrict__ h, long h_ld, const TW* __restrict__ w_gu, const int* __restrict__ chosen, float* __restrict__ a,
    int width, int ff, int top, FlGate act, int gated, const float* __restrict__ in_weights) {
    pdl_wait();
    pdl_trigger();
    using L = MoeRows<TW>;
    extern __shared__ __align__(16) float moe_x[];      // [width]
    const int pair = blockIdx.x, t = pair / top;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int i = threadIdx.x; i < width; i += blockDim.x) moe_x[i] = to_f32<T>(h[(long)t * h_ld + i]);
    __syncthreads();
    const int f = (blockIdx.y * MOE_GU_WARPS + warp) * L::ROWS + lane / L::LPR, c0 = (lane % L::LPR) * L::V;
    const int fr = min(f, ff - 1);                       // lanes beyond the last feature repeat it and store nothing
    const float win = in_weights != nullptr ? in_weights[pair] : 1.0f;      // what multiplies the expert's input
    if (!gated) {
        float acc[1][L::V] = {};
        moe_rows_dot<1, U>(moe_x + c0, w_gu + ((long)chosen[pair] * ff + fr) * width + c0, 0, width, acc);
        const float x = moe_rows_sum(acc[0]);
        if (c0 == 0 && f < ff) a[(long)pair * ff + f] = fl_gated(x * win, 1.0f, act);
        return;
    }
    float acc[2][L::V] = {};
    moe_rows_dot<2, U>(moe_x + c0, w_gu + ((long)chosen[pair] * 2 * ff + fr) * width + c0, (long)ff * width, width, acc);
    const float g = moe_rows_sum(acc[0]), u = moe_rows_sum(acc[1]);
    if (c0 == 0 && f < ff) a[(long)pair * ff + f] = fl_gated(g * win, u * win, act);
}

// w_down: [experts][width][ff]; a warp takes every eighth choice of the token, the choices are added in order
#define MOE_DOWN_WARPS 8
template <typename T, typename TW, int U>
__global__ void __launch_bounds__(MOE_DOWN_WARPS * 32) moe_down_rows_kernel(
    const float* __restrict__ a, const TW* __restrict__ w_down, const int* __restrict__ chosen, const float* __restrict__ weights,
    T* __restrict__ out, long out_ld, int width, int ff, int top, int accumulate) {
    pdl_wait();
    pdl_trigger();
    using L = MoeRows<TW>;
    __shared__ float y_s[MOE_DOWN_WARPS][L::ROWS];
    const int t = blockIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31, warps = blockDim.x >> 5;
    const int row = lane / L::LPR, c = blockIdx.y * L::ROWS + row, c0 = (lane % L::LPR) * L::V;
    const int cr = min(c, width - 1);
    float sum = 0.0f;
    for (int k0 = 0; k0 < top; k0 += warps) {
        if (k0 + warp < top) {
            const long pair = (long)t * top + k0 + warp;
            float acc[1][L::V] = {};
            moe_rows_dot<1, U>(a + pair * ff + c0, w_down + ((long)chosen[pair] * width + cr) * ff + c0, 0, ff, acc);
            const float y = moe_rows_sum(acc[0]);
            if (c0 == 0) y_s[warp][row] = y;
        }
        __syncthreads();
        if (warp == 0)
            for (int k = 0; k < warps && k0 + k < top; ++k)
                sum += (weights != nullptr ? weights[(long)t * top + k0 + k] : 1.0f) * y_s[k][row];
        __syncthreads();
    }
    if (warp == 0 && c0 == 0 && c < width)
        out[(long)t * out_ld + c] = from_f32<T>(accumulate ? to_f32<T>(out[(long)t * out_ld + c]) + sum : sum);
}

// the same for any sizes
template <typename T, typename TW>
__global__ void __launch_bounds__(256) moe_gate_up_kernel(const T* __restrict__ h, long h_ld, const TW* __restrict__ w_gu,
                                                          const int* __restrict__ chosen, float* __restrict__ a,
                                                          int width, int ff, int top, FlGate act, int gated,
                                                          const float* __restrict__ in_weights) {
    pdl_wait();
    pdl_trigger();
    extern __shared__ __align__(16) float moe_x[];      // [width]
    const int pair = blockIdx.x, t = pair / top;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int i = threadIdx.x; i < width; i += blockDim.x) moe_x[i] = to_f32<T>(h[(long)t * h_ld + i]);
    __syncthreads();
    const int f = blockIdx.y * 8 + warp;
    if (f >= ff) return;
    const float win = in_weights != nullptr ? in_weights[pair] : 1.0f;      // what multiplies the expert's input
    if (!gated) {
        const TW* wx = w_gu + ((long)chosen[pair] * ff + f) * width;
        float x = 0.0f;
        for (int i = lane; i < width; i += 32) x = fmaf(moe_x[i], to_f32<TW>(wx[i]), x);
        x = warp_sum(x);
        if (lane == 0) a[(long)pair * ff + f] = fl_gated(x * win, 1.0f, act);
        return;
    }
    const TW* wg = w_gu + ((long)chosen[pair] * 2 * ff + f) * width;
    const TW* wu = wg + (long)ff * width;
    float g = 0.0f, u = 0.0f;
    for (int i = lane; i < width; i += 32) {
        g = fmaf(moe_x[i], to_f32<TW>(wg[i]), g);
        u = fmaf(moe_x[i], to_f32<TW>(wu[i]), u);
    }
    g = warp_sum(g);
    u = warp_sum(u);
    if (lane == 0) a[(long)pair * ff + f] = fl_gated(g * win, u * win, act);
}

template <typename T, typename TW>
__global__ void __launch_bounds__(256) moe_down_kernel(const float* __restrict__ a, const TW* __restrict__ w_down,
                                                       const int* __restrict__ chosen, const float* __restrict__ weights,
                                                       T* __restrict__ out, long out_ld, int width, int ff, int top,
                                                       int accumulate) {
    pdl_wait();
    pdl_trigger();
    const int t = blockIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int c = blockIdx.y * 8 + warp;
    if (c >= width) return;
    float sum = 0.0f;
    for (int k = 0; k < top; ++k) {
        const long pair = (long)t * top + k;
        const TW* wd = w_down + ((long)chosen[pair] * width + c) * ff;
        const float* ar = a + pair * ff;
        float y = 0.0f;
        for (int i = lane; i < ff; i += 32) y = fmaf(ar[i], to_f32<TW>(wd[i]), y);
        sum += (weights != nullptr ? weights[pair] : 1.0f) * warp_sum(y);
    }
    if (lane == 0) out[(long)t * out_ld + c] = from_f32<T>(accumulate ? to_f32<T>(out[(long)t * out_ld + c]) + sum : sum);
}

FL_API int fl_moe_pick(const float* z, long z_ld, const void* bias, int bias_dtype, int* chosen, float* weights,
                       int n_tokens, int experts, int top, int softmax_scores, int renormalise, int n_groups, int keep,
                       float renorm_eps, int group_top, float weight_scale, cudaStream_t stream) {
    if (n_tokens <= 0) return 0;
    if (n_groups < 1) n_groups = keep = 1;
    const size_t smem = (size_t)(2 * experts + n_groups) * 4 * sizeof(float);
    if (top < 1 || top > experts || smem > 48 * 1024 || experts % n_groups || keep < 1 || keep > n_groups ||
        (long)keep * (experts / n_groups) < top || group_top < 1)
        return (int)cudaErrorInvalidValue;
    FL_DISPATCH(bias_dtype, TW,
        return fl_launch(moe_pick_kernel<TW>, dim3((n_tokens + 3) / 4), dim3(128), smem, stream,
                         z, z_ld, (const TW*)bias, chosen, weights, n_tokens, experts, top, softmax_scores, renormalise,
                         n_groups, keep, renorm_eps, group_top, weight_scale));
    return 0;
}

FL_API int fl_moe_experts(const void* h, int dtype, long h_ld, const void* w_gu, const void* w_down, int w_dtype,
                          const int* chosen, const float* weights, float* a, void* out, long out_ld, int n_tokens,
                          int width, int ff, int top, int act, float act_p0, float act_p1, int gated,
                          int accumulate, int weight_on_input, int num_sms, cudaStream_t stream) {
    if (n_tokens <= 0) return 0;
    if ((size_t)width * sizeof(float) > 48 * 1024 || (ff + 7) / 8 > 65535 || (width + 7) / 8 > 65535 || act < 0 || act >= FL_ACT_COUNT)
        return (int)cudaErrorInvalidValue;
    int rc = 0;
    const FlGate unit{act, act_p0, act_p1};
    const float *in_weights = weight_on_input ? weights : nullptr, *out_weights = weight_on_input ? nullptr : weights;
    const bool few = (long)n_tokens * top * ((ff + 31) / 32) * MOE_GU_WARPS <= 16L * num_sms;    // 16 warps an SM with U = 8
    // Several rows a warp pay once that leaves warps enough.  For the second product, whose warps take a choice each: two
    // choices or more, or 8192 rows' worth of bfloat16 outputs (both products, 1 choice of 32 experts of 2048 x 1408: 1 token
    // 14.6 us a row a warp and 22.7 eight rows a warp, 8 tokens 49 and 36).  For the first: beside such a second one, with a
    // warp an SM (1 token x 4: 24.6 us, 30.6 with a row a warp in the first product, 36.8 in both).
    const bool aligned = width % 32 == 0 && ff % 32 == 0 && (((uintptr_t)w_gu | (uintptr_t)w_down | (uintptr_t)a) % 16) == 0;
    const bool rows_down = aligned && (top > 1 || (long)n_tokens * width * 2 >= 8192L * (w_dtype == FL_F32 ? 4 : 2));
    const bool rows_up = rows_down && (long)n_tokens * top * ((ff + 31) / 32) * MOE_GU_WARPS >= num_sms;
    FL_DISPATCH(dtype, T, FL_DISPATCH(w_dtype, TW, {
        constexpr int PER = MOE_GU_WARPS * MoeRows<TW>::ROWS;
        if (rows_up)
            rc = fl_launch(few ? moe_gate_up_rows_kernel<T, TW, 8> : moe_gate_up_rows_kernel<T, TW, 4>, dim3(n_tokens * top, (ff + PER - 1) / PER), dim3(MOE_GU_WARPS * 32),
                           (size_t)width * sizeof(float), stream, (const T*)h, h_ld, (const TW*)w_gu, chosen, a, width, ff, top,
                           unit, gated, in_weights);
        else
            rc = fl_launch(moe_gate_up_kernel<T, TW>, dim3(n_tokens * top, (ff + 7) / 8), dim3(256), (size_t)width * sizeof(float),
                           stream, (const T*)h, h_ld, (const TW*)w_gu, chosen, a, width, ff, top, unit, gated, in_weights);
    }));
    if (rc) return rc;
    FL_DISPATCH(dtype, T, FL_DISPATCH(w_dtype, TW, {
        constexpr int PER = MoeRows<TW>::ROWS;
        if (rows_down)
            return fl_launch(few ? moe_down_rows_kernel<T, TW, 11> : moe_down_rows_kernel<T, TW, 8>, dim3(n_tokens, (width + PER - 1) / PER),
                             dim3(32 * (top < MOE_DOWN_WARPS ? top : MOE_DOWN_WARPS)), 0, stream, (const float*)a,
                             (const TW*)w_down, chosen, out_weights, (T*)out, out_ld, width, ff, top, accumulate);
        return fl_launch(moe_down_kernel<T, TW>, dim3(n_tokens, (width + 7) / 8), dim3(256), 0, stream, (const float*)a,
                         (const TW*)w_down, chosen, out_weights, (T*)out, out_ld, width, ff, top, accumulate);
    }));
    return 0;
}

// ----------------------------------------------------------------- many tokens: grouped products
// With many tokens the per-token kernels above would read each expert's matrices once per token.  Here
// the (token, choice) pairs are ordered by expert, and two tensor-core products run over tiles of up to 256 pairs
// that share an expert's matrix.
//
//   moe_sort        one block: counts per expert, row -> pair, pair -> row, and the list of tiles: an expert's rows are
//                   cut into as few tiles of at most 256 (of small matrices 128 or 64) as will do, equally wide (a multiple
//                   of 64)
//   moe_gather      the tokens' rows in the order of the pairs
//   moe_group       tcgen05.mma over CTA pairs.  GATED: a pair's 256 weight rows are 128 gate rows and the 128 up rows of
//                   the same features, the epilogue writes f(g, u) (bfloat16, in row order); UP: experts without a gate,
//                   256 up rows, the epilogue writes the unit's f(x, 1); DOWN: A is that buffer and the output
//                   float [rows, width]
//   moe_combine     out[t] = sum_k weight[t, k] * y[row of pair (t, k)], in order of choice
//
// A row's sums do not depend on the other rows of its tile, so the order of rows within an expert (it
// comes from atomics) does not show in the results.
#define MOE_TN 256               // rows (pairs) of a tile at most
// a tile of the list, an int4: expert, first row, rows, rows in the MMA (a multiple of 64)

__global__ void __launch_bounds__(1024) moe_sort_kernel(const int* __restrict__ chosen, int n_pairs, int experts,
                                                       int* __restrict__ row_pair, int* __restrict__ pair_row,
                                                       int4* __restrict__ tiles, int* __restrict__ n_tiles_out, int tile_rows) {
    pdl_wait();
    pdl_trigger();
    extern __shared__ int count[];                       // [experts] counts, then cursors
    for (int e = threadIdx.x; e < experts; e += blockDim.x) count[e] = 0;
    __syncthreads();
    for (int p = threadIdx.x; p < n_pairs; p += blockDim.x) atomicAdd(&count[chosen[p]], 1);
    __syncthreads();
    if (threadIdx.x < 32) {                              // running sums of rows and tiles, 32 experts at a time
        const int lane = threadIdx.x;
        int rows_before = 0, tiles_before = 0;
        for (int e0 = 0; e0 < experts; e0 += 32) {
            const int c = e0 + lane < experts ? count[e0 + lane] : 0, nt = (c + tile_rows - 1) / tile_rows;
            int row = c, tile = nt;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int r = __shfl_up_sync(0xffffffffu, row, o), t = __shfl_up_sync(0xffffffffu, tile, o);
                if (lane >= o) row += r, tile += t;
            }
            const int first = rows_before + row - c, at = tiles_before + tile - nt;
            if (e0 + lane < experts) count[e0 + lane] = first;
            const int n = nt > 0 ? ((c + nt - 1) / nt + 63) / 64 * 64 : 0;
            for (int i = 0; i < nt; ++i) tiles[at + i] = make_int4(e0 + lane, first + i * n, min(n, c - i * n), n);
            rows_before += __shfl_sync(0xffffffffu, row, 31);
            tiles_before += __shfl_sync(0xffffffffu, tile, 31);
        }
        if (lane == 0) *n_tiles_out = tiles_before;
    }
    __syncthreads();
    for (int p = threadIdx.x; p < n_pairs; p += blockDim.x) {
        const int r = atomicAdd(&count[chosen[p]], 1);
        row_pair[r] = p;
        pair_row[p] = r;
    }
}

// a[r] = h[token of row r]: 16 bytes a thread (a pass of its own costs 2 x rows x width bytes, 10 us at 8192 rows of 2048;
// in return the products fetch both operands with plain TMA boxes; measured with its launch: 16 us)
__global__ void __launch_bounds__(256) moe_gather_kernel(const bf16* __restrict__ h, long h_ld, const int* __restrict__ row_pair,
                                                         int n_pairs, int top, bf16* __restrict__ a, int width) {
    pdl_wait();
    pdl_trigger();
    const int per_row = width / 8;
    const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
    const int r = (int)(i / per_row), c = (int)(i - (long)r * per_row) * 8;
    if (r >= n_pairs) return;
    *reinterpret_cast<uint4*>(a + (long)r * width + c) = *reinterpret_cast<const uint4*>(h + (long)(row_pair[r] / top) * h_ld + c);
}

// The CTA-pair product of gemm_tcgen05.cu (see there for the roles, the barriers and why a pair) over the list of tiles:
// a unit of work is (tile, 256 weight rows), weight rows going fastest so that a tile's rows stay in L2 while its
// expert's matrix streams by once; a tile's width is its own, so the MMA's N, the 32-row boxes of A and the bytes of a
// stage are per unit.  64 rows x 128 weight rows a block on mma.sync took 452 + 300 us for 8192 pairs, 32 experts of
// 2048 x 1408 (142 GFLOP: 190 TFLOP/s), its operands fetched six times as often from L2; this takes 119 + 66 us (770
// TFLOP/s).  The accumulator's bits are the same: K in steps of 16 from the first to the last.
enum { MOE_DOWN = 0, MOE_GATED = 1, MOE_UP = 2 };
enum { MOE_ERR_WAIT = 131 };

// g[j] = f(g[j], v[j]) as `fl_gated` has it (the exact exponential and division), the unit chosen once for all N values
template <int N> __device__ __forceinline__ void moe_act(float (&g)[N], const float (&v)[N], const FlGate act) {
#define MOE_ACT(ACT)                                                                                 \
    {                                                                                                \
        _Pragma("unroll") for (int j = 0; j < N; ++j) g[j] = fl_gated(g[j], v[j], FlGate{ACT, act.p0, act.p1}); \
    }
    switch (act.act) {
        case FL_ACT_RELU: MOE_ACT(FL_ACT_RELU) break;
        case FL_ACT_RELU_SQUARED: MOE_ACT(FL_ACT_RELU_SQUARED) break;
        case FL_ACT_GELU_TANH: MOE_ACT(FL_ACT_GELU_TANH) break;
        case FL_ACT_CLAMPED_SWISH: MOE_ACT(FL_ACT_CLAMPED_SWISH) break;
        default: MOE_ACT(FL_ACT_SILU)
    }
#undef MOE_ACT
}

#define MOE_EPILOGUE_BYTES (2 * 32 * 128 * 4)            // GATED: 2 x (32 x 64 up values | 32 x 64 results); else 2 x 32 x 128
#define MOE_SMEM (Tc2<256>::SMEM + MOE_EPILOGUE_BYTES + 2 * 32 * 4)

template <int MODE>
__global__ void __launch_bounds__(TC_THREADS) moe_group_kernel(
    const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_a, const int4* __restrict__ tiles,
    const int* __restrict__ n_tiles, const int* __restrict__ row_pair, int n_out, int K, bf16* __restrict__ act_out,
    float* __restrict__ y_out, FlGate act, const float* __restrict__ in_weights, int* __restrict__ status) {
    using L = Tc2<256>;
    constexpr bool GATED = MODE == MOE_GATED;
    extern __shared__ unsigned char smem_raw[];
    unsigned char* ring = (unsigned char*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    uint64_t* full_bar = (uint64_t*)(ring + L::TILE_BYTES);
    uint64_t* empty_bar = full_bar + L::STAGES;
    uint64_t* acc_full = empty_bar + L::STAGES;
    uint64_t* acc_empty = acc_full + 2;
    uint32_t* tmem_slot = (uint32_t*)(acc_empty + 2);
    volatile int* abort_flag = (volatile int*)(tmem_slot + 1);
    unsigned char* staged = ring + L::TILE_BYTES + 256;
    float* win_s = reinterpret_cast<float*>(staged + MOE_EPILOGUE_BYTES);          // [2][32] what multiplies a row's input

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t rank = cluster_rank();                   // 0: leader
    const int pair = (int)blockIdx.x >> 1, num_pairs = (int)gridDim.x >> 1;
    const int num_kb = (K + TC_BK - 1) / TC_BK;
    constexpr int FEATURES = GATED ? 128 : 256;             // of a unit; half of them are this CTA's
    const int tiles_n = (n_out + FEATURES - 1) / FEATURES;
    const int num_units = *n_tiles * tiles_n;

    if (threadIdx.x == 0) {
        for (int s = 0; s < L::STAGES; ++s) {
            mbar_init(&full_bar[s], 1);
            mbar_init(&empty_bar[s], 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(&acc_full[b], 1);
            mbar_init(&acc_empty[b], 8);                    // four epilogue warps in each of the two CTAs
        }
        *abort_flag = (*(volatile int*)status != 0) ? 1 : 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                     "r"(512u)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync_all();                                     // both CTAs' barriers exist before anyone signals them
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    // (launched in plain stream order, and no pdl_trigger: see the pair kernel of gemm_tcgen05.cu)

    auto give_up = [&]() {
        if (!*abort_flag) { *abort_flag = 1; atomicCAS(status, 0, MOE_ERR_WAIT); }
    };
    int issued = 0;                                         // (thread 0: fills of the ring)
    if (warp == 0) {
        if (lane == 0 && !*abort_flag) {
            // ---- producer (both CTAs): this CTA's 128 weight rows and half of the tile's rows, k-block after k-block
            int s = 0;
            uint32_t ph = 0;
            bool ok = true;
            for (int u = pair; u < num_units && ok; u += num_pairs) {
                const int4 t = tiles[u / tiles_n];
                const int tn = u % tiles_n, half = t.w / 2;
                for (int kb = 0; kb < num_kb; ++kb) {
                    if (!mbar_wait(&empty_bar[s], ph ^ 1u, abort_flag)) {
                        give_up();
                        ok = false;
                        break;
                    }
                    unsigned char* dst = ring + s * L::STAGE_BYTES;
                    if (rank == 0) mbar_expect_tx(&full_bar[s], 2 * (L::W_BYTES + half * TC_BK * 2));
                    if (GATED) {                            // 64 gate rows and the 64 up rows of the same features
                        const int f0 = t.x * 2 * n_out + tn * 128 + (int)rank * 64;
                        tma_load_2d_pair(dst, &map_w, &full_bar[s], kb * TC_BK, f0);
                        tma_load_2d_pair(dst + L::W_BYTES / 2, &map_w, &full_bar[s], kb * TC_BK, f0 + n_out);
                    } else {
                        tma_load_2d_pair(dst, &map_w, &full_bar[s], kb * TC_BK, t.x * n_out + tn * 256 + (int)rank * 128);
                    }
                    for (int r = 0; r < half; r += 32)
                        tma_load_2d_pair(dst + L::W_BYTES + r * TC_BK * 2, &map_a, &full_bar[s], kb * TC_BK,
                                         t.y + (int)rank * half + r);
                    ++issued;
                    if (++s == L::STAGES) { s = 0; ph ^= 1u; }
                }
            }
        }
    } else if (warp == 1) {
        if (lane == 0 && rank == 0) {
            // ---- MMA issuer (leader only): one 256 x n x 16 MMA per 16 columns of K, for both CTAs
            int s = 0, i = 0;
            uint32_t ph = 0;
            bool ok = !*abort_flag;
            for (int u = pair; u < num_units && ok; u += num_pairs, ++i) {
                const uint32_t idesc = instr_desc_bf16(256, tiles[u / tiles_n].w);
                const int buf = i & 1;
                const uint32_t use = (uint32_t)(i >> 1);
                if (!mbar_wait(&acc_empty[buf], (use & 1u) ^ 1u, abort_flag)) {
                    give_up();
                    ok = false;
                    break;
                }
                tc_fence_after();
                const uint32_t tmem_acc = tmem_base + (uint32_t)(buf * 256);
                for (int kb = 0; kb < num_kb; ++kb) {
                    if (!mbar_wait(&full_bar[s], ph, abort_flag)) {
                        give_up();
                        ok = false;
                        break;
                    }
                    tc_fence_after();
                    const uint32_t w_addr = smem_u32(ring + s * L::STAGE_BYTES);
                    const uint64_t adesc = smem_desc_sw128(w_addr);
                    const uint64_t bdesc = smem_desc_sw128(w_addr + L::W_BYTES);
#pragma unroll
                    for (int k = 0; k < TC_BK / 16; ++k)
                        umma_bf16_pair(tmem_acc, adesc + (uint64_t)(2 * k), bdesc + (uint64_t)(2 * k), idesc,
                                       (kb > 0 || k > 0) ? 1u : 0u);
                    umma_commit_pair(&empty_bar[s]);
                    if (++s == L::STAGES) { s = 0; ph ^= 1u; }
                }
                if (ok) umma_commit_pair(&acc_full[buf]);
            }
        }
    } else {
        // ---- epilogue warps 2..5 of both CTAs: this CTA's 128 accumulator rows of the unit, 32 tile rows at a time
        const int quarter = warp & 3, e = quarter * 32 + lane;
        uint32_t rounds_out = 0;                            // picks the staging half
        int i = 0;
        for (int u = pair; u < num_units; u += num_pairs, ++i) {
            const int buf = i & 1;
            const uint32_t use = (uint32_t)(i >> 1);
            if (!mbar_wait(&acc_full[buf], use & 1u, abort_flag)) give_up();
            if (epilogue_any(*abort_flag != 0)) break;      // the four warps decide together (they share barriers below)
            tc_fence_after();
            const int4 t = tiles[u / tiles_n];
            const int f0 = (u % tiles_n) * FEATURES + (int)rank * (FEATURES / 2), cols = n_out - f0;
            const uint32_t t_base = tmem_base + (uint32_t)(buf * 256) + ((uint32_t)(quarter * 32) << 16);
#pragma unroll 1
            for (int c = 0; c < t.z; c += 32) {
                const int rows = min(32, t.z - c);
                uint32_t r[32];
                tmem_ld16(t_base + (uint32_t)c, r);
                tmem_ld16(t_base + (uint32_t)c + 16u, r + 16);
                const uint32_t half = rounds_out++ & 1u;
                float* win = win_s + half * 32;
                if (MODE != MOE_DOWN && in_weights != nullptr && quarter == 0)
                    win[lane] = lane < rows ? in_weights[row_pair[t.y + c + lane]] : 0.0f;
                unsigned char* area = staged + half * (MOE_EPILOGUE_BYTES / 2);
                tmem_ld_wait();
                if constexpr (GATED) {
                    // accumulator lanes 0..63: gate features, 64..127: the same features' up values; the gate warps
                    // finish the even rows, the up warps the odd ones, trading values through shared memory
                    const bool is_up = quarter >= 2;
                    const int mine = is_up ? 1 : 0, col = (quarter & 1) * 32 + lane;
                    float* x = reinterpret_cast<float*>(area);
                    bf16* st = reinterpret_cast<bf16*>(area + 32 * 64 * 4);
#pragma unroll
                    for (int j = 0; j < 16; ++j)
                        x[(2 * j + 1 - mine) * 64 + col] = __uint_as_float(is_up ? r[2 * j] : r[2 * j + 1]);
                    epilogue_sync();
                    float g[16], v[16];                     // rows 2 j + mine
#pragma unroll
                    for (int j = 0; j < 16; ++j) {
                        const float own = __uint_as_float(is_up ? r[2 * j + 1] : r[2 * j]), other = x[(2 * j + mine) * 64 + col];
                        g[j] = is_up ? other : own;
                        v[j] = is_up ? own : other;
                    }
                    if (in_weights != nullptr) {
#pragma unroll
                        for (int j = 0; j < 16; ++j) {
                            const float w = win[2 * j + mine];
                            g[j] *= w;
                            v[j] *= w;
                        }
                    }
                    moe_act(g, v, act);
#pragma unroll
                    for (int j = 0; j < 16; ++j) st[(2 * j + mine) * 64 + col] = __float2bfloat16_rn(g[j]);
                    epilogue_sync();
                    if (cols > 0)
                        tc_copy_rows<bf16, 64>(act_out + (long)(t.y + c) * n_out + f0, n_out, st, rows, min(cols, 64), e, true);
                } else if constexpr (MODE == MOE_UP) {
                    if (in_weights != nullptr) epilogue_sync();
                    float g[32], one[32];
#pragma unroll
                    for (int j = 0; j < 32; ++j) {
                        g[j] = __uint_as_float(r[j]) * (in_weights != nullptr ? win[j] : 1.0f);
                        one[j] = 1.0f;
                    }
                    moe_act(g, one, act);
                    bf16* st = reinterpret_cast<bf16*>(area);
#pragma unroll
                    for (int j = 0; j < 32; ++j) st[j * 128 + e] = __float2bfloat16_rn(g[j]);
                    epilogue_sync();
                    if (cols > 0)
                        tc_copy_rows<bf16, 128>(act_out + (long)(t.y + c) * n_out + f0, n_out, st, rows, min(cols, 128), e, true);
                } else {
                    float* st = reinterpret_cast<float*>(area);
#pragma unroll
                    for (int j = 0; j < 32; ++j) st[j * 128 + e] = __uint_as_float(r[j]);
                    epilogue_sync();
                    if (cols > 0)
                        tc_copy_rows<float, 128>(y_out + (long)(t.y + c) * n_out + f0, n_out, st, rows, min(cols, 128), e, true);
                }
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive_leader(&acc_empty[buf]);
        }
    }
    tc_fence_before();
    __syncthreads();
    if (threadIdx.x == 0 && *abort_flag) tma_drain(full_bar, rank == 0 ? L::STAGES : 0, issued);
    __syncwarp();
    cluster_sync_all();                                     // the peer is done with this CTA's barriers and memory
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512u) : "memory");
    }
    cluster_sync_all();                                     // both have given their tensor memory back before either leaves
}

// Four columns a thread and the rows of all choices asked for at once: one column a thread, each load behind its row's
// index, took 62 us for 2048 tokens x 4 choices of 2048 columns (67 MB); this takes 12.
template <typename T>
__global__ void __launch_bounds__(256) moe_combine_kernel(const float* __restrict__ y, long y_ld, const int* __restrict__ pair_row,
                                                          const float* __restrict__ weights, T* __restrict__ out, long out_ld,
                                                          int width, int top, int accumulate) {
    pdl_wait();
    pdl_trigger();
    const int t = blockIdx.x, c = (blockIdx.y * blockDim.x + threadIdx.x) * 4;
    if (c >= width) return;
    const int* rows = pair_row + (long)t * top;
    const float* w = weights != nullptr ? weights + (long)t * top : nullptr;
    float sum[4] = {};
    for (int k0 = 0; k0 < top; k0 += 4) {                   // (width is a multiple of 32)
        float4 v[4];
        float wk[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            if (k0 + k >= top) continue;
            v[k] = *reinterpret_cast<const float4*>(y + (long)rows[k0 + k] * y_ld + c);
            wk[k] = w != nullptr ? w[k0 + k] : 1.0f;
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            if (k0 + k >= top) continue;
            sum[0] += wk[k] * v[k].x;
            sum[1] += wk[k] * v[k].y;
            sum[2] += wk[k] * v[k].z;
            sum[3] += wk[k] * v[k].w;
        }
    }
    T* o = out + (long)t * out_ld + c;
#pragma unroll
    for (int j = 0; j < 4; ++j) o[j] = from_f32<T>(accumulate ? to_f32<T>(o[j]) + sum[j] : sum[j]);
}

// Rows of the ordered buffers that a step of n_tokens is given: one a pair, and 64 an expert, which the products do not
// need but the list of tiles (one for every 256 pairs and one per expert, 16 bytes each) does.
FL_API long fl_moe_group_rows(int n_tokens, int top, int experts) {
    return (((long)n_tokens * top + 63) / 64 + experts) * 64;
}

// Does the grouped path take this problem?  (bfloat16 everywhere, K of both products a multiple of 32.)
FL_API int fl_moe_group_takes(int dtype, int w_dtype, int width, int ff) {
    return dtype == FL_BF16 && w_dtype == FL_BF16 && width % 32 == 0 && ff % 32 == 0;
}

template <int MODE>
static int moe_group_launch(const void* a, const void* w, long w_rows, int n_pairs, int max_tiles, const int4* tiles, const int* n_tiles,
                            const int* row_pair, int n_out, int K, void* act_out, float* y_out, FlGate act,
                            const float* in_weights, int num_sms, int* status, cudaStream_t stream) {
    auto kernel = moe_group_kernel<MODE>;
    CUtensorMap map_w, map_a;
    int rc = make_map(&map_w, w, w_rows, K, K, MODE == MOE_GATED ? 64 : 128);
    if (rc == 0) rc = make_map(&map_a, a, n_pairs, K, K, 32);
    if (rc == 0) rc = (int)cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, MOE_SMEM);
    if (rc) return rc;
    static_assert(MOE_SMEM <= 232448, "more shared memory than a CTA can have");
    const int features = MODE == MOE_GATED ? 128 : 256;
    const long units = (long)max_tiles * ((n_out + features - 1) / features);
    const int pairs = units < num_sms / 2 ? (int)units : num_sms / 2;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(2 * pairs);
    cfg.blockDim = dim3(TC_THREADS);
    cfg.dynamicSmemBytes = MOE_SMEM;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return (int)cudaLaunchKernelEx(&cfg, kernel, map_w, map_a, tiles, n_tiles, row_pair, n_out, K, (bf16*)act_out, y_out, act,
                                   in_weights, status);
}

// ints: rows + n_tokens * top + rows / 64 + 1 of them, rows = fl_moe_group_rows: row -> pair, pair -> row, the list of tiles
// (from a 16-byte boundary on) and its length, 2 pairs + pairs / 64 + 4 experts + 4 at most with tiles of 256;
// act: bfloat16 [rows, ff], 16-byte aligned; y: float [rows, width], of which the first 16-byte boundary on holds the
// gathered tokens and then the results, a row a pair.
FL_API int fl_moe_experts_grouped(const void* h, long h_ld, const void* w_gu, const void* w_down, const int* chosen,
                                  const float* weights, int* ints, void* act, float* y, void* out, long out_ld,
                                  int n_tokens, int width, int ff, int top, int experts, int act_code, float act_p0, float act_p1,
                                  int gated, int accumulate, int weight_on_input, int num_sms, int* status, cudaStream_t stream) {
    if (n_tokens <= 0) return 0;
    const float* in_weights = weight_on_input ? weights : nullptr;
    if (act_code < 0 || act_code >= FL_ACT_COUNT) return (int)cudaErrorInvalidValue;
    const FlGate gate{act_code, act_p0, act_p1};
    const int n_pairs = n_tokens * top;
    int* row_pair = ints;
    int* pair_row = ints + n_pairs;
    int4* tiles = reinterpret_cast<int4*>(((uintptr_t)(ints + 2L * n_pairs) + 15) & ~(uintptr_t)15);
    y = reinterpret_cast<float*>(((uintptr_t)y + 15) & ~(uintptr_t)15);
    // Tiles of 256 rows, or narrower ones where matrices of few rows would leave most CTA pairs idle (and where the list has
    // room for them): 2048 pairs, 8 experts of 256 x 128, are 8 units of 256 rows.
    const int some = experts < n_pairs ? experts : n_pairs;
    const int n_up = gated ? (ff + 127) / 128 : (ff + 255) / 256, n_down = (width + 255) / 256, n_few = n_up < n_down ? n_up : n_down;
    const long rows = fl_moe_group_rows(n_tokens, top, experts), room = rows + n_pairs + rows / 64 + 1 - (2L * n_pairs + 3) - 1;
    int tile_rows = MOE_TN;
    while (tile_rows > 64 && (long)(n_pairs / tile_rows > some ? n_pairs / tile_rows : some) * n_few < num_sms / 2 &&
           4L * (2 * n_pairs / tile_rows + some) <= room)
        tile_rows /= 2;
    const int max_tiles = n_pairs / tile_rows + some;
    int* n_tiles = reinterpret_cast<int*>(tiles + max_tiles);
    if ((size_t)experts * sizeof(int) > 48 * 1024 || width % 32 || ff % 32 || num_sms < 2 ||
        (((uintptr_t)h | (uintptr_t)act) % 16) || (h_ld % 8))
        return (int)cudaErrorInvalidValue;
    int rc = fl_launch(moe_sort_kernel, dim3(1), dim3(1024), (size_t)experts * sizeof(int), stream, chosen, n_pairs, experts,
                       row_pair, pair_row, tiles, n_tiles, tile_rows);
    if (rc) return rc;
    const long pieces = (long)n_pairs * (width / 8);
    rc = fl_launch(moe_gather_kernel, dim3((unsigned)((pieces + 255) / 256)), dim3(256), 0, stream, (const bf16*)h, h_ld,
                   (const int*)row_pair, n_pairs, top, (bf16*)y, width);
    if (rc) return rc;
    if (gated)
        rc = moe_group_launch<MOE_GATED>(y, w_gu, 2L * experts * ff, n_pairs, max_tiles, tiles, n_tiles, row_pair, ff, width, act,
                                         nullptr, gate, in_weights, num_sms, status, stream);
    else
        rc = moe_group_launch<MOE_UP>(y, w_gu, (long)experts * ff, n_pairs, max_tiles, tiles, n_tiles, row_pair, ff, width, act,
                                      nullptr, gate, in_weights, num_sms, status, stream);
    if (rc) return rc;
    rc = moe_group_launch<MOE_DOWN>(act, w_down, (long)experts * width, n_pairs, max_tiles, tiles, n_tiles, row_pair, width, ff,
                                    nullptr, y, gate, nullptr, num_sms, status, stream);
    if (rc) return rc;
    return fl_launch(moe_combine_kernel<bf16>, dim3(n_tokens, (width + 1023) / 1024), dim3(256), 0, stream, (const float*)y,
                     (long)width, (const int*)pair_row, weight_on_input ? nullptr : weights, (bf16*)out, out_ld, width, top, accumulate);
}
