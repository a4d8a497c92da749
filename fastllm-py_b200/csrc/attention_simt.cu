// Paged causal attention on CUDA cores, for any mix of prompt portions and
// single decoded tokens, in bfloat16 or true 32-bit.
//
// The keys of a token are taken in tiles of 64 that start at multiples of 64 of
// the absolute key position.  A tile has a result of its own (its maximum, the
// sum of exp(score - maximum) and the weighted values, softmax in float with the
// exact expf; a score is summed in four chains over the head's columns, the weighted
// values over the tile's keys in order), and the tiles' results are folded from
// the first to the last.  So the order of every sum depends only on the token's
// own position: the result is the same bit for bit however the sequence was cut
// into steps, whatever else is in the batch and however many CTAs share the
// tiles.  This is the reference kernel of the engine and the 32-bit path's
// attention.
//
// A cluster of CL CTAs serves QT neighbouring tokens of the step and one query
// head.  QT is 8 for prompts (a tile that has been fetched serves 8 tokens; where
// requests meet inside the 8, one request's tokens follow the other's) and 1
// for steps in which every request brings one token.  Prompts are bound by the
// multiply-adds and shared-memory reads, single tokens by latency: with few
// (token, head) pairs in the step the tiles are dealt out to the cluster's CTAs
// (tile t to CTA t mod CL), which hand their results over through distributed
// shared memory.  One block a (token, head) pair, each thread walking a key row
// in global memory, took 91 us for 4 tokens over 700 keys and 16 heads of 128 in
// 32 bits, and 437 us for a prompt of 300 tokens; this takes 25 and 82 (in
// bfloat16 93, 430, 29 and 83; 32 tokens over 700 keys 280 and 178).
//
// fastllm-py's counterparts: `_sdpa` (fastllm_py/model.py:341-353: scores scaled
// by head_dim^-1/2, keys beyond the query masked, softmax and the weighted sum in
// float) and the decode kernels `attn_decode` (fastllm_py/graph_decode.py:378-420)
// and `battn` (fastllm_py/batched.py:48-92).  Grouped heads are index
// arithmetic, h / (H / KVH), never a materialised repeat (model.py:426-428).
#include <cooperative_groups.h>

#include "common.cuh"

#define ATT_THREADS 128
#define ATT_TILE 64              // keys

template <int QT> struct AttHold { static constexpr int TILES = QT == 1 ? 8 : 2; };     // tiles a CTA holds before they are folded

// floats of shared memory of a CTA: queries, keys, values, scores, weights, tile results
__host__ __device__ constexpr int att_pad(int head_dim) { return (head_dim + 3) / 4 * 4; }
__host__ __device__ constexpr int att_floats(int qt, int hold, int dp) {
    return qt * dp + ATT_TILE * (dp + 4) + ATT_TILE * dp + 2 * qt * ATT_TILE + hold * qt * (dp + 2);
}

__device__ __forceinline__ void att_cp16(float* smem, const float* gmem) {
    const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(s), "l"(gmem) : "memory");
}

// NV: value columns a thread (1: heads of up to 128)
template <typename T, int QT, int CL, int NV>
__global__ void __launch_bounds__(ATT_THREADS) paged_attention_simt_kernel(
    const T* __restrict__ q, long q_ld, T* __restrict__ out, long out_ld,
    const T* __restrict__ k_cache, const T* __restrict__ v_cache, long page_stride, int page_size,
    const int* __restrict__ block_table, int bt_stride, const int* __restrict__ tok_req,
    const int* __restrict__ positions, int n_tokens, int n_heads, int n_kv_heads, int head_dim, int window,
    float scale, int vec, int page_shift) {
    pdl_wait();
    pdl_trigger();
    namespace cg = cooperative_groups;
    constexpr int HOLD = AttHold<QT>::TILES;
    extern __shared__ __align__(16) float att_smem[];
    const int dp = att_pad(head_dim), kp = dp + 4;
    float* q_s = att_smem;                              // [QT][dp]
    float* k_s = q_s + QT * dp;                         // [tile][kp]: eight neighbouring rows lie in all 32 banks
    float* v_s = k_s + ATT_TILE * kp;                   // [tile][dp]
    float* s_s = v_s + ATT_TILE * dp;                   // [QT][tile] scores
    float* p_s = s_s + QT * ATT_TILE;                   // [tile][QT] softmax numerators
    float* hold_acc = p_s + QT * ATT_TILE;              // [HOLD][QT][dp]
    float* hold_ml = hold_acc + HOLD * QT * dp;         // [HOLD][QT] maximum, sum

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int rank = CL == 1 ? 0 : (int)(blockIdx.x % CL), h = blockIdx.y;
    const int t_begin = (int)((gridDim.x - 1 - blockIdx.x) / CL) * QT, t_end = min(n_tokens, t_begin + QT);
    const int kvh = h / (n_heads / n_kv_heads);
    const long head_off = (long)kvh * page_size * head_dim;
    const int pieces = vec ? head_dim / (16 / (int)sizeof(T)) : 1;          // 16-byte pieces of a row
    const int row0 = tid / pieces, piece0 = tid - row0 * pieces;            // this thread's first one of a tile

    for (int t0 = t_begin, nq; t0 < t_end; t0 += nq) {  // tokens of one request at a time
        const int req = tok_req[t0];
        nq = 1;
        while (QT > 1 && t0 + nq < t_end && tok_req[t0 + nq] == req) ++nq;
        const int* bt = block_table + (long)req * bt_stride;
        int pos[QT], first = 0x7fffffff, last = -1;
#pragma unroll
        for (int i = 0; i < QT; ++i) {
            pos[i] = i < nq ? positions[t0 + i] : -1;
            if (i < nq) {
                first = min(first, window > 0 ? max(0, pos[i] - window + 1) : 0);
                last = max(last, pos[i]);
            }
        }
        for (int r = QT == 1 ? 0 : warp; r < nq; r += ATT_THREADS / 32)
#pragma unroll 4
            for (int d = QT == 1 ? tid : lane; d < dp; d += QT == 1 ? ATT_THREADS : 32)
                q_s[r * dp + d] = d < head_dim ? to_f32<T>(q[(long)(t0 + r) * q_ld + (long)h * head_dim + d]) : 0.0f;
        float acc[QT][NV] = {}, m[QT], l[QT];
        bool begun[QT];
#pragma unroll
        for (int i = 0; i < QT; ++i) m[i] = -CUDART_INF_F, l[i] = 0.0f, begun[i] = false;
        const int d0 = tid, d1 = tid + ATT_THREADS;                 // (d1: NV 2 only)

        auto lowest = [&](int i) { return window > 0 ? max(0, pos[i] - window + 1) : 0; };
        auto sees = [&](int i, int tile) { return i < nq && pos[i] >= tile * ATT_TILE && lowest(i) < (tile + 1) * ATT_TILE; };

        // The result of one tile: maximum and sum of query i in ml[2 i], ml[2 i + 1], the weighted values in `a`.
        auto do_tile = [&](int tile, float* ml, float (&a)[QT][NV]) {
            const int base = tile * ATT_TILE, keys = min(ATT_TILE, last + 1 - base);
            // keys and values of the tile, rows outside first .. last left as zeros: what lies past the last visible key may
            // hold anything, and the table has -1 for pages that every window in the step has passed
            auto in_sight = [&](int r, long& off) {
                const int j = base + r;
                if (j >= first && r < keys) {
                    const int page = page_shift >= 0 ? j >> page_shift : j / page_size;
                    off = (long)bt[page] * page_stride + head_off + (long)(j - page * page_size) * head_dim;
                    return true;
                }
                return false;
            };
            if (vec) {
                // 16 bytes a thread and step; the next step's piece lies ATT_THREADS pieces on: `rows` rows and `rest` pieces
                constexpr int V = 16 / (int)sizeof(T), BATCH = sizeof(T) == 4 ? 1 : 4;
                const int rows = ATT_THREADS / pieces, rest = ATT_THREADS - rows * pieces;
                int r = row0, c = piece0;
#pragma unroll(sizeof(T) == 4 ? 4 : 1)
                while (r < ATT_TILE) {
                    uint4 kr[BATCH], vr[BATCH];
                    int at_k[BATCH], at_v[BATCH];
#pragma unroll
                    for (int b = 0; b < BATCH; ++b) {
                        long off;
                        at_k[b] = r < ATT_TILE ? r * kp + c * V : -1;
                        at_v[b] = r * dp + c * V;
                        kr[b] = vr[b] = make_uint4(0u, 0u, 0u, 0u);
                        if (r < ATT_TILE && in_sight(r, off)) {
                            if constexpr (sizeof(T) == 4) {
                                att_cp16(k_s + at_k[b], reinterpret_cast<const float*>(k_cache) + off + c * V);
                                att_cp16(v_s + at_v[b], reinterpret_cast<const float*>(v_cache) + off + c * V);
                                at_k[b] = -1;
                            } else {
                                kr[b] = *reinterpret_cast<const uint4*>(k_cache + off + c * V);
                                vr[b] = *reinterpret_cast<const uint4*>(v_cache + off + c * V);
                            }
                        }
                        r += rows;
                        c += rest;
                        if (c >= pieces) c -= pieces, ++r;
                    }
#pragma unroll
                    for (int b = 0; b < BATCH; ++b) {
                        if (at_k[b] < 0) continue;
                        const T *ke = reinterpret_cast<const T*>(&kr[b]), *ve = reinterpret_cast<const T*>(&vr[b]);
#pragma unroll
                        for (int e = 0; e < V; e += 4) {
                            *reinterpret_cast<float4*>(k_s + at_k[b] + e) =
                                make_float4(to_f32<T>(ke[e]), to_f32<T>(ke[e + 1]), to_f32<T>(ke[e + 2]), to_f32<T>(ke[e + 3]));
                            *reinterpret_cast<float4*>(v_s + at_v[b] + e) =
                                make_float4(to_f32<T>(ve[e]), to_f32<T>(ve[e + 1]), to_f32<T>(ve[e + 2]), to_f32<T>(ve[e + 3]));
                        }
                    }
                }
                asm volatile("cp.async.commit_group;" ::: "memory");
                asm volatile("cp.async.wait_group 0;" ::: "memory");
            } else {
#pragma unroll 4
                for (int r = warp; r < ATT_TILE; r += ATT_THREADS / 32) {
                    long off = 0;
                    const bool in = in_sight(r, off);
                    for (int c = lane; c < dp; c += 32) {
                        k_s[r * kp + c] = in && c < head_dim ? to_f32<T>(k_cache[off + c]) : 0.0f;
                        v_s[r * dp + c] = in && c < head_dim ? to_f32<T>(v_cache[off + c]) : 0.0f;
                    }
                }
            }
            __syncthreads();
            if constexpr (QT == 1) {
                // scores: two threads a key, two of its four chains each (one thread a key left half of the block idle: 4 tokens
                // over 500 to 900 keys, 16 heads of 128, 24.3 us and 24.0 now; 32 over 700, 8 heads of 256, 160 and 144)
                const int key = tid >> 1, part = (tid & 1) * 2;
                float2 dot = make_float2(0.0f, 0.0f);
#pragma unroll 8
                for (int d = 0; d < dp; d += 4) {
                    const float2 k2 = *reinterpret_cast<const float2*>(k_s + key * kp + d + part);
                    const float2 q2 = *reinterpret_cast<const float2*>(q_s + d + part);
                    dot.x = fmaf(q2.x, k2.x, dot.x);
                    dot.y = fmaf(q2.y, k2.y, dot.y);
                }
                const float mine = dot.x + dot.y, other = __shfl_xor_sync(0xffffffffu, mine, 1);
                if (part == 0) s_s[key] = (mine + other) * scale;
            } else {
                // scores: a thread takes one key and every other group of queries
                constexpr int HALF = QT / 2;
                const int key = tid & (ATT_TILE - 1), i0 = (tid / ATT_TILE) * HALF;
                float dot[HALF][4] = {};
#pragma unroll 4
                for (int d = 0; d < dp; d += 4) {
                    const float4 k4 = *reinterpret_cast<const float4*>(k_s + key * kp + d);
#pragma unroll
                    for (int i = 0; i < HALF; ++i) {
                        const float4 q4 = *reinterpret_cast<const float4*>(q_s + (i0 + i) * dp + d);
                        dot[i][0] = fmaf(q4.x, k4.x, dot[i][0]);
                        dot[i][1] = fmaf(q4.y, k4.y, dot[i][1]);
                        dot[i][2] = fmaf(q4.z, k4.z, dot[i][2]);
                        dot[i][3] = fmaf(q4.w, k4.w, dot[i][3]);
                    }
                }
#pragma unroll
                for (int i = 0; i < HALF; ++i)
                    s_s[(i0 + i) * ATT_TILE + key] = ((dot[i][0] + dot[i][1]) + (dot[i][2] + dot[i][3])) * scale;
            }
            __syncthreads();
#pragma unroll
            for (int i = 0; i < QT; ++i) {
                if ((i & 3) != warp || !sees(i, tile)) continue;
                const int ja = base + lane, jb = ja + 32;
                const bool va = ja >= lowest(i) && ja <= pos[i], vb = jb >= lowest(i) && jb <= pos[i];
                const float sa = va ? s_s[i * ATT_TILE + lane] : -CUDART_INF_F, sb = vb ? s_s[i * ATT_TILE + lane + 32] : -CUDART_INF_F;
                const float mt = warp_max(fmaxf(sa, sb)), at = mt == -CUDART_INF_F ? 0.0f : mt;     // (scores of -inf: no weight)
                const float pa = va ? expf(sa - at) : 0.0f, pb = vb ? expf(sb - at) : 0.0f;
                p_s[lane * QT + i] = pa;
                p_s[(lane + 32) * QT + i] = pb;
                const float lt = warp_sum(pa + pb);
                if (lane == 0) ml[2 * i] = mt, ml[2 * i + 1] = lt;
            }
            __syncthreads();
            // keys outside a query's range are left out rather than weighted by zero: they may hold infinities
            int from[QT], count[QT];                     // the keys of the tile that query i sees
            int common = nq == QT ? ATT_TILE : 0;        // as many first keys are seen by all
#pragma unroll
            for (int i = 0; i < QT; ++i) {
                from[i] = max(0, lowest(i) - base);
                count[i] = i < nq ? max(0, min(ATT_TILE - 1, pos[i] - base) - from[i] + 1) : 0;
                common = from[i] > 0 ? 0 : min(common, count[i]);
#pragma unroll
                for (int v = 0; v < NV; ++v) a[i][v] = 0.0f;
            }
#pragma unroll 4
            for (int j = 0; j < common; ++j) {
                float v[NV];
                v[0] = d0 < head_dim ? v_s[j * dp + d0] : 0.0f;
                if (NV > 1) v[NV - 1] = d1 < head_dim ? v_s[j * dp + d1] : 0.0f;
#pragma unroll
                for (int i = 0; i < QT; ++i) {
                    const float p = p_s[j * QT + i];
#pragma unroll
                    for (int e = 0; e < NV; ++e) a[i][e] = fmaf(p, v[e], a[i][e]);
                }
            }
            for (int j = common; j < keys; ++j) {
                float v[NV];
                v[0] = d0 < head_dim ? v_s[j * dp + d0] : 0.0f;
                if (NV > 1) v[NV - 1] = d1 < head_dim ? v_s[j * dp + d1] : 0.0f;
#pragma unroll
                for (int i = 0; i < QT; ++i) {
                    if ((unsigned)(j - from[i]) >= (unsigned)count[i]) continue;
                    const float p = p_s[j * QT + i];
#pragma unroll
                    for (int e = 0; e < NV; ++e) a[i][e] = fmaf(p, v[e], a[i][e]);
                }
            }
        };
        auto fold = [&](int i, float mt, float lt, const float (&at)[NV]) {
            if (!begun[i]) {
                begun[i] = true;
                m[i] = mt, l[i] = lt;
#pragma unroll
                for (int e = 0; e < NV; ++e) acc[i][e] = at[e];
                return;
            }
            const float m_new = fmaxf(m[i], mt), at_new = m_new == -CUDART_INF_F ? 0.0f : m_new;
            const float c = expf(m[i] - at_new), ct = expf(mt - at_new);
            m[i] = m_new;
            l[i] = l[i] * c + lt * ct;
#pragma unroll
            for (int e = 0; e < NV; ++e) acc[i][e] = acc[i][e] * c + at[e] * ct;
        };

        const int tile0 = first / ATT_TILE, tile1 = last / ATT_TILE + 1;
        __syncthreads();                                 // the queries are there
        if constexpr (CL == 1) {
            for (int tile = tile0; tile < tile1; ++tile) {
                float a[QT][NV];
                do_tile(tile, hold_ml, a);
#pragma unroll
                for (int i = 0; i < QT; ++i)
                    if (sees(i, tile)) fold(i, hold_ml[2 * i], hold_ml[2 * i + 1], a[i]);
                __syncthreads();                         // the tile's shared memory is read, the next one may come
            }
        } else {
            cg::cluster_group cluster = cg::this_cluster();
            for (int round = tile0; round < tile1; round += CL * HOLD) {
#pragma unroll 1
                for (int slot = 0; slot < HOLD; ++slot) {
                    const int tile = round + slot * CL + rank;
                    if (tile >= tile1) break;
                    float a[QT][NV];
                    do_tile(tile, hold_ml + slot * 2 * QT, a);
#pragma unroll
                    for (int i = 0; i < QT; ++i) {
                        if (d0 < head_dim) hold_acc[(slot * QT + i) * dp + d0] = a[i][0];
                        if (NV > 1 && d1 < head_dim) hold_acc[(slot * QT + i) * dp + d1] = a[i][NV - 1];
                    }
                    __syncthreads();
                }
                cluster.sync();
                // query i is folded by CTA i mod CL
                const int stop = min(tile1, round + CL * HOLD);
#pragma unroll
                for (int i = 0; i < QT; ++i) {
                    if (i % CL != rank || i >= nq) continue;
                    constexpr int BATCH = 8;             // results on their way at once
                    for (int t = round; t < stop; t += BATCH) {
                        float mt[BATCH], lt[BATCH], at[BATCH][NV];
#pragma unroll
                        for (int e = 0; e < BATCH; ++e) {
                            const int n = min(t + e, stop - 1) - round, slot = n / CL;
                            const float* ml = cluster.map_shared_rank(hold_ml, n % CL) + slot * 2 * QT;
                            const float* ha = cluster.map_shared_rank(hold_acc, n % CL) + (slot * QT + i) * dp;
                            mt[e] = ml[2 * i];
                            lt[e] = ml[2 * i + 1];
                            at[e][0] = d0 < head_dim ? ha[d0] : 0.0f;
                            if (NV > 1) at[e][NV - 1] = d1 < head_dim ? ha[d1] : 0.0f;
                        }
#pragma unroll
                        for (int e = 0; e < BATCH; ++e)
                            if (t + e < stop && sees(i, t + e)) fold(i, mt[e], lt[e], at[e]);
                    }
                }
                cluster.sync();
            }
        }
#pragma unroll
        for (int i = 0; i < QT; ++i) {
            if (i >= nq || (CL > 1 && i % CL != rank)) continue;
            T* o = out + (long)(t0 + i) * out_ld + (long)h * head_dim;
            if (d0 < head_dim) o[d0] = from_f32<T>(acc[i][0] / l[i]);
            if (NV > 1 && d1 < head_dim) o[d1] = from_f32<T>(acc[i][NV - 1] / l[i]);
        }
        __syncthreads();                                 // the queries are read, the next request's may come
    }
}

template <typename T, int QT, int CL, int NV>
static int att_launch(const T* q, long q_ld, T* out, long out_ld, const T* k_cache, const T* v_cache, long page_stride,
                      int page_size, const int* block_table, int bt_stride, const int* tok_req, const int* positions,
                      int n_tokens, int n_heads, int n_kv_heads, int head_dim, int window, float scale, cudaStream_t stream) {
    auto kernel = paged_attention_simt_kernel<T, QT, CL, NV>;
    const size_t smem = 4 * (size_t)att_floats(QT, AttHold<QT>::TILES, att_pad(head_dim));
    cudaError_t err = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (err != cudaSuccess) return (int)err;
    constexpr int V = 16 / (int)sizeof(T);
    const int vec = head_dim % V == 0 && page_stride % V == 0 && (((uintptr_t)k_cache | (uintptr_t)v_cache) % 16) == 0;
    int page_shift = -1;
    if ((page_size & (page_size - 1)) == 0)
        for (page_shift = 0; (1 << page_shift) < page_size;) ++page_shift;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)((n_tokens + QT - 1) / QT) * CL, n_heads);
    cfg.blockDim = dim3(ATT_THREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = CL;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = fl_pdl_enabled() ? 2 : 1;
    return (int)cudaLaunchKernelEx(&cfg, kernel, q, q_ld, out, out_ld, k_cache, v_cache, page_stride, page_size, block_table,
                                   bt_stride, tok_req, positions, n_tokens, n_heads, n_kv_heads, head_dim, window, scale, vec, page_shift);
}

// What a launch of groups of `qt` tokens on clusters of `cl` CTAs takes, in microseconds, fitted (on the logarithm, 24 %
// root-mean-square error) to runs of both group sizes over heads of 16 to 256, prompts of 8 to 1024 tokens and portions
// behind up to 2000: rounds of as many CTAs as the SMs hold, in each of which a CTA begins and goes through its share of the
// tiles, one tile taking as long as a CTA alone takes for it or as the SM takes for those of all its CTAs.
static double att_cost(long units, int tiles, int qt, int cl, int head_dim, int sms) {
    const size_t smem = 4 * (size_t)att_floats(qt, qt == 1 ? AttHold<1>::TILES : AttHold<8>::TILES, att_pad(head_dim)) + 1024;
    int places = (int)(228 * 1024 / smem);
    if (places > (qt == 1 ? 4 : 3)) places = qt == 1 ? 4 : 3;
    const double wide = head_dim / 128.0, waves = (double)units * cl / ((double)places * sms);
    const double beside = waves >= 1.0 ? places : ceil(waves * places);
    const double alone = qt == 1 ? 2.7 + 2.3 * wide : 6.8 + 3.1 * wide, shared = (qt == 1 ? 2.0 * wide : 1.0 + 3.0 * wide) * beside;
    const double share = (tiles + cl - 1) / cl;                          // (of the last tokens: earlier ones see fewer tiles)
    return (waves <= 2.0 ? ceil(waves) : waves + 0.5) *
           ((qt == 1 ? 0.0 : 5.4) + (waves <= 1.0 ? share : 0.5 * share + 0.5) * (alone > shared ? alone : shared));
}

// q: [n_tokens, q_ld] with head h at columns [h*head_dim, (h+1)*head_dim);
// out likewise.  tok_req[t] is the row of `block_table` that token t's request
// uses; positions[t] is the token's absolute position, whose key (already in
// the cache) is the last one it sees.  window <= 0 means all keys.  Two hints, on which results do not depend: `single`:
// neighbouring tokens belong to different requests; `longest`: the most keys that a token of the step has (0: not known).
FL_API int fl_paged_attention_simt(const void* q, int dtype, long q_ld, void* out, long out_ld,
                                   const void* k_cache, const void* v_cache, long page_stride,
                                   int page_size, const int* block_table, int bt_stride,
                                   const int* tok_req, const int* positions, int n_tokens,
                                   int n_heads, int n_kv_heads, int head_dim, int window, float scale, int single, int longest,
                                   int sms, cudaStream_t stream) {
    if (n_tokens <= 0) return 0;
    if (head_dim < 1 || head_dim > 2 * ATT_THREADS || n_heads > 65535 || n_heads % n_kv_heads)
        return (int)cudaErrorInvalidValue;
    // As many CTAs a cluster as keep the launch within two CTAs an SM or so: more only wait for one another.
    const long units = (long)((n_tokens + (single ? 0 : 7)) / (single ? 1 : 8)) * n_heads;
    int cl = units * 4 <= 2L * sms ? 8 : units <= sms ? 4 : units <= 2L * sms ? 2 : 1;
    if (longest > 0 && !single) {
        // Where the number of keys is known: groups of eight tokens, or one token a CTA if some cluster makes that cheaper.
        // (Few tokens over few keys wait for one tile, which eight tokens take twice as long for: a prompt of 8 tokens, 16
        // heads of 128, took 12.9 us in groups of eight and takes 5.)  Picks are 3.5 % off the better one on average.
        auto tiles = [&](int qt) {
            int keys = longest;
            if (window > 0 && keys > window + qt + ATT_TILE - 2) keys = window + qt + ATT_TILE - 2;
            return (keys + ATT_TILE - 1) / ATT_TILE;
        };
        const bool two = head_dim > ATT_THREADS;                          // (kernels for clusters of 4 and 1 only)
        double best = att_cost(units, tiles(8), 8, two ? (cl >= 4 ? 4 : 1) : cl, head_dim, sms);
        for (int c = 1; c <= (two ? 4 : 8); c *= two ? 4 : 2) {
            const double t = att_cost((long)n_tokens * n_heads, tiles(1), 1, c, head_dim, sms);
            if (t < best) best = t, single = 1, cl = c;
        }
    }
#define ATT_GO(QT, CL, NV)                                                                                                \
    FL_DISPATCH(dtype, T, return (att_launch<T, QT, CL, NV>((const T*)q, q_ld, (T*)out, out_ld, (const T*)k_cache,        \
                                                            (const T*)v_cache, page_stride, page_size, block_table,      \
                                                            bt_stride, tok_req, positions, n_tokens, n_heads, n_kv_heads, \
                                                            head_dim, window, scale, stream)))
    if (head_dim > ATT_THREADS) {
        if (single) {
            if (cl >= 4) ATT_GO(1, 4, 2);
            ATT_GO(1, 1, 2);
        }
        if (cl >= 4) ATT_GO(8, 4, 2);
        ATT_GO(8, 1, 2);
    }
    if (single) {
        if (cl == 8) ATT_GO(1, 8, 1);
        if (cl == 4) ATT_GO(1, 4, 1);
        if (cl == 2) ATT_GO(1, 2, 1);
        ATT_GO(1, 1, 1);
    }
    if (cl == 8) ATT_GO(8, 8, 1);
    if (cl == 4) ATT_GO(8, 4, 1);
    if (cl == 2) ATT_GO(8, 2, 1);
    ATT_GO(8, 1, 1);
#undef ATT_GO
}
