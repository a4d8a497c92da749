// C[M, N] = A[M, K] * W[N, K]^T on CUDA cores with float accumulation: the
// matrix product of the true 32-bit path (no tensor-core mode drops mantissa
// bits here), and the product for any operand types the tensor-core kernel
// does not take (a weight stored in 32-bit under bfloat16 activations).
//
// fastllm-py calls cuBLAS for `x @ w.T` (fastllm_py/model.py:63).  These kernels
// have one property cuBLAS lacks: the order of every sum depends on K alone,
// whatever M is and whichever kernel runs, so a token's result does not depend
// on how many other tokens share the step.  The order: K is cut into GS_SLICES
// slices of gs_slice(K) inputs, a slice is summed from its first input to its last
// with fused multiply-adds, and the slices' sums are added from the first to
// the last.  (Eight short chains instead of one of K: the rounding error falls
// too, and the slices are what the kernels share out among threads and CTAs.)
//
// Three kernels:
//   gemm_f32_skinny_kernel  float operands, up to 16 rows: bound by streaming W from memory
//   gemm_f32_tile_kernel    float operands, more rows: bound by the multiply-adds
//   gemm_simt_kernel        any operand types, alignments and batches
// The last one served everything before: 350 us a product for 4 rows and 590 us for 300 rows of a layer with 2048 and
// 5504 columns (10 TFLOP/s); the others take 6 to 21 us (2.7 to 4.3 TB/s of W, out of a cold cache) and 67 to 305 us (37
// to 44 TFLOP/s).
#include <cooperative_groups.h>

#include "common.cuh"

#define GS_BM 64
#define GS_BN 64
#define GS_BK 16
#define GS_SLICES 8

// Inputs per slice: a multiple of 32, which every kernel's K step divides.
static inline int gs_slice(int K) { return ((K + GS_SLICES - 1) / GS_SLICES + 31) / 32 * 32; }

template <typename TA, typename TW, typename TC>
__global__ void __launch_bounds__(256, 4) gemm_simt_kernel(const TA* __restrict__ A, long lda,
                                                        const TW* __restrict__ W, long ldw,
                                                        TC* __restrict__ C, long ldc, int M, int N,
                                                        int K, int slice, long a_batch, long w_batch, long c_batch) {
    pdl_wait();
    pdl_trigger();
    A += blockIdx.z * a_batch;                // a batch of products over column blocks of wider buffers
    W += blockIdx.z * w_batch;
    C += blockIdx.z * c_batch;
    __shared__ __align__(16) float As[GS_BK][GS_BM + 4];
    __shared__ __align__(16) float Ws[GS_BK][GS_BN + 4];
    const int tid = threadIdx.x;
    const int tx = tid & 15, ty = tid >> 4;
    const int m0 = blockIdx.y * GS_BM, n0 = blockIdx.x * GS_BN;
    float acc[4][4] = {}, total[4][4] = {};
    // The next 16 inputs are on their way while these are used, and both operands come from shared memory four at a time: 4
    // rows of 2050 x 2050 take 192 us and 300 rows 204 (a value at a time 217 and 277, with the slices' ends looked for in
    // the loop over K and nothing on its way 273 and 291).
    float next_a[4], next_w[4];
    auto fetch = [&](int k0) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int r = (tid >> 4) + i * 16, k = k0 + (tid & 15);
            next_a[i] = (k < K && m0 + r < M) ? to_f32<TA>(A[(long)(m0 + r) * lda + k]) : 0.0f;
            next_w[i] = (k < K && n0 + r < N) ? to_f32<TW>(W[(long)(n0 + r) * ldw + k]) : 0.0f;
        }
    };
    fetch(0);
    for (int begin = 0; begin < K; begin += slice) {
        const int end = min(K, begin + slice);
        for (int k0 = begin; k0 < end; k0 += GS_BK) {
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                As[tid & 15][(tid >> 4) + i * 16] = next_a[i];
                Ws[tid & 15][(tid >> 4) + i * 16] = next_w[i];
            }
            __syncthreads();
            fetch(k0 + GS_BK);
#pragma unroll
            for (int kk = 0; kk < GS_BK; ++kk) {
                const float4 a4 = *reinterpret_cast<const float4*>(&As[kk][ty * 4]), b4 = *reinterpret_cast<const float4*>(&Ws[kk][tx * 4]);
                const float a[4] = {a4.x, a4.y, a4.z, a4.w}, b[4] = {b4.x, b4.y, b4.z, b4.w};
#pragma unroll
                for (int i = 0; i < 4; ++i)
#pragma unroll
                    for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
            }
            __syncthreads();
        }
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                total[i][j] += acc[i][j];
                acc[i][j] = 0.0f;
            }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int m = m0 + ty * 4 + i;
        if (m >= M) continue;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int n = n0 + tx * 4 + j;
            if (n < N) C[(long)m * ldc + n] = from_f32<TC>(total[i][j]);
        }
    }
}

// ------------------------------------------------------------ up to 16 rows
// A CTA of 64 threads serves 8 x RT features: thread (slice s, row r) sums slice s of features r, r + 8, ... for all MT
// rows of A.  W and A pass through a ring of shared-memory stages, 32 inputs of every slice each, filled by 16-byte
// cp.async: what bounds the product is the stream of W, so the ring keeps 2 or 3 stages (16 KB of W each, two or three CTAs an
// SM) in flight, and where the caller says that no kernel writes W (constant_w) its first stages are asked for before the
// preceding kernel has ended.  A staged row of W is padded
// to 36 floats: the eight lanes of a quarter warp, on eight rows, then read all 32 banks.  With RT = 2 a value of A that has been read
// from shared memory serves two features: with one, the reads of A kept more shared memory busy than W did (11008 features
// of 2048, out of a cold cache: 21.7, 22.2, 29.1 and 25.0 us for 1 to 4 rows; 19.1, 20.1, 21.0 and 21.2 now, 4.2 to 4.7 TB/s
// of W; 2048 features 6.1 to 8.0, now 5.6 to 6.4).  A third stage in flight costs four rows 5 to 10 % on many features, as
// one CTA an SM fewer fits, and gains one or two rows up to 7 % on few.  Rows past M are zeroes up to four rows (3 rows took
// longer than 4 when they repeated the last one), and repeat the last one above, where leaving them out costs 2 to 4 % of the
// products that have them all; they are not written.
#define SK_BK 32
#define SK_PITCH 36

template <int MT, int RT_> struct Skinny {
    static constexpr int RT = RT_;
    static constexpr int R = 8 * RT;
    static constexpr int STAGES = RT == 2 && (MT > 8 || MT == 4) ? 3 : 4;
    static constexpr int A_PITCH = MT * SK_BK + 4;                     // floats of a slice's rows of A
    static constexpr int W_FLOATS = GS_SLICES * R * SK_PITCH;
    static constexpr int STAGE_FLOATS = W_FLOATS + GS_SLICES * A_PITCH;
    static constexpr int SMEM = STAGES * STAGE_FLOATS * 4;
};

__device__ __forceinline__ void sk_cp16(float* smem, const float* gmem, bool valid) {
    const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(s), "l"(gmem), "r"(valid ? 16 : 0) : "memory");
}

template <typename TC, int MT, int RT_>
__global__ void __launch_bounds__(64) gemm_f32_skinny_kernel(const float* __restrict__ A, long lda,
                                                             const float* __restrict__ W, long ldw,
                                                             TC* __restrict__ C, long ldc, int M, int N, int K, int slice,
                                                             int constant_w) {
    using L = Skinny<MT, RT_>;
    constexpr int RT = L::RT, R = L::R, STAGES = L::STAGES;
    extern __shared__ __align__(16) float sk_smem[];
    const int tid = threadIdx.x, row = tid & 7, s = tid >> 3;
    const int n0 = blockIdx.x * R;
    const int n_st = slice / SK_BK;
    // this thread copies 16-byte piece `row` of a stage's 32 inputs, of slice `s`, for every row of W and A
    auto load_w = [&](int t) {
        const int k = s * slice + t * SK_BK + row * 4;
        float* dst = sk_smem + (t % STAGES) * L::STAGE_FLOATS + s * R * SK_PITCH + row * 4;
#pragma unroll
        for (int r = 0; r < R; ++r) sk_cp16(dst + r * SK_PITCH, k < K ? W + (long)min(n0 + r, N - 1) * ldw + k : W, k < K);
    };
    auto load_a = [&](int t) {
        const int k = s * slice + t * SK_BK + row * 4;
        float* dst = sk_smem + (t % STAGES) * L::STAGE_FLOATS + L::W_FLOATS + s * L::A_PITCH + row * 4;
#pragma unroll
        for (int m = 0; m < MT; ++m) {
            const bool in = k < K && (MT != 4 || m < M);                // (below, M is MT)
            sk_cp16(dst + m * SK_BK, in ? A + (long)(MT > 4 ? min(m, M - 1) : m) * lda + k : A, in);
        }
    };
    if (constant_w)
        for (int t = 0; t < STAGES - 1 && t < n_st; ++t) load_w(t);
    pdl_wait();
    pdl_trigger();
    for (int t = 0; t < STAGES - 1; ++t) {
        if (t < n_st && !constant_w) load_w(t);
        if (t < n_st) load_a(t);
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
    float acc[RT][MT] = {};
    for (int t = 0; t < n_st; ++t) {
        asm volatile("cp.async.wait_group %0;" ::"n"(STAGES - 2) : "memory");
        __syncthreads();                                               // stage t is there, stage t - 1 has been read
        if (t + STAGES - 1 < n_st) {
            load_w(t + STAGES - 1);
            load_a(t + STAGES - 1);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
        const float* w_s = sk_smem + (t % STAGES) * L::STAGE_FLOATS + (s * R + row) * SK_PITCH;
        const float* a_s = sk_smem + (t % STAGES) * L::STAGE_FLOATS + L::W_FLOATS + s * L::A_PITCH;
#pragma unroll(MT > 8 ? 1 : 4)
        for (int k = 0; k < SK_BK; k += 4) {
            float4 w[RT];
#pragma unroll
            for (int r = 0; r < RT; ++r) w[r] = *reinterpret_cast<const float4*>(w_s + r * 8 * SK_PITCH + k);
#pragma unroll
            for (int m = 0; m < MT; ++m) {
                const float4 a = *reinterpret_cast<const float4*>(a_s + m * SK_BK + k);
#pragma unroll
                for (int r = 0; r < RT; ++r) {
                    acc[r][m] = fmaf(a.x, w[r].x, acc[r][m]);
                    acc[r][m] = fmaf(a.y, w[r].y, acc[r][m]);
                    acc[r][m] = fmaf(a.z, w[r].z, acc[r][m]);
                    acc[r][m] = fmaf(a.w, w[r].w, acc[r][m]);
                }
            }
        }
    }
    __syncthreads();
    float* red = sk_smem;                                              // [slice][row of A][feature]
#pragma unroll
    for (int r = 0; r < RT; ++r)
#pragma unroll
        for (int m = 0; m < MT; ++m) red[(s * MT + m) * R + r * 8 + row] = acc[r][m];
    __syncthreads();
    for (int i = tid; i < MT * R; i += 64) {
        const int m = i / R, n = n0 + i % R;
        float total = 0.0f;
#pragma unroll
        for (int z = 0; z < GS_SLICES; ++z) total += red[z * MT * R + i];
        if (m < M && n < N) C[(long)m * ldc + n] = from_f32<TC>(total);
    }
}

// ------------------------------------------------------------ more rows
// SPLIT: a cluster of GS_SLICES CTAs shares a tile of 64 rows x TL_BN features; each sums one slice, and each adds up an eighth
// of the rows from the others' shared memory, in the order of the slices, so no partial sum goes to global memory.  Else one CTA
// sums the slices of a tile one after the other, which is the faster form where a slice is short (see gs_f32).  Bound by
// the multiply-adds, which are issued in pairs (fma.rn.f32x2, the same rounding), and by what they read from shared memory
// (128 bytes a clock reach the registers, however many lanes want the same): 8 rows x 8 features a thread.  Both operands
// wait in shared memory turned to [input][row], double-buffered; columns are exchanged by a pattern of the input's index, so
// that neither the turned stores nor the 16-byte reads meet in a bank.  The next stage comes by cp.async into slots that only
// the copying thread reads, so it needs no registers meanwhile and four CTAs of a split tile fit an SM.  (300 rows, 11008
// features of 2048: 409 us with the next stage in registers and two CTAs an SM; 305 now, 44 TFLOP/s.  Every value of A twice in shared memory instead of a move for each pair of features, or 64 x 256 tiles:
// 347 and 327 us at best.)
#define TL_BM 64
#define TL_BN 128
#define TL_NH (TL_BN / 64)               // groups of four features a thread
#define TL_BK 16
#define TL_THREADS 128
#define TL_SMEM (3 * TL_BK * (TL_BM + TL_BN) > TL_BM * TL_BN ? 12 * TL_BK * (TL_BM + TL_BN) : 4 * TL_BM * TL_BN)

__device__ __forceinline__ void fma2(float2& d, const float2 a, const float2 b) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;"
        : "+l"(reinterpret_cast<unsigned long long&>(d))
        : "l"(reinterpret_cast<const unsigned long long&>(a)), "l"(reinterpret_cast<const unsigned long long&>(b)));
}

template <typename TC, bool SPLIT>
__device__ __forceinline__ void gemm_f32_tile(const float* __restrict__ A, long lda, const float* __restrict__ W, long ldw,
                                              TC* __restrict__ C, long ldc, int M, int N, int K, int slice) {
    constexpr int A_FLOATS = TL_BK * TL_BM, STAGE = A_FLOATS + TL_BK * TL_BN, PIECES = (TL_BM + TL_BN) / 32;
    extern __shared__ __align__(16) float tl_smem[];                    // two stages and the copies' slots; the tile's sums
    float4(*raw)[TL_THREADS] = reinterpret_cast<float4(*)[TL_THREADS]>(tl_smem + 2 * STAGE);
    const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
    const int m0 = blockIdx.y * TL_BM, n0 = blockIdx.x * TL_BN;
    const int k_begin = SPLIT ? min(K, (int)blockIdx.z * slice) : 0, k_end = SPLIT ? min(K, k_begin + slice) : K;
    // this thread's 16-byte pieces of a stage: rows lr, lr + 32, ... of A (two) and W, inputs 4 lk .. 4 lk + 3
    const int lr = tid >> 2, lk = tid & 3;
    auto fetch = [&](int k0) {
        const int k = k0 + lk * 4;
        const bool in = k < k_end;
#pragma unroll
        for (int i = 0; i < PIECES; ++i) {
            const int row = i < 2 ? m0 + lr + 32 * i : n0 + lr + 32 * (i - 2);
            const bool there = in && row < (i < 2 ? M : N);             // else zeroes, and nothing is read
            const float* src = i < 2 ? A + (long)row * lda : W + (long)row * ldw;
            sk_cp16(reinterpret_cast<float*>(&raw[i][tid]), there ? src + k : A, there);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    auto turn = [&](int buf) {
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        float* a_s = tl_smem + buf * STAGE;
#pragma unroll
        for (int i = 0; i < PIECES; ++i) {
            const float4 v = raw[i][tid];
            const int pitch = i < 2 ? TL_BM : TL_BN;
            float* d = a_s + (i < 2 ? 0 : A_FLOATS) + lk * 4 * pitch + ((lr + 32 * (i < 2 ? i : i - 2)) ^ (lk << 3));
            d[0] = v.x, d[pitch] = v.y, d[2 * pitch] = v.z, d[3 * pitch] = v.w;
        }
    };
    float2 acc[8][2 * TL_NH], total[SPLIT ? 1 : 8][2 * TL_NH];          // 8 rows x pairs of features
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 2 * TL_NH; ++j) {
            acc[i][j] = make_float2(0.0f, 0.0f);
            if (!SPLIT) total[i][j] = make_float2(0.0f, 0.0f);
        }
    if (k_begin < k_end) {
        fetch(k_begin);
        turn(0);
        if (k_begin + TL_BK < k_end) fetch(k_begin + TL_BK);
    }
    __syncthreads();
    int buf = 0, left = slice;
    for (int k0 = k_begin; k0 < k_end; k0 += TL_BK) {
        if (k0 + TL_BK < k_end) {
            turn(buf ^ 1);
            if (k0 + 2 * TL_BK < k_end) fetch(k0 + 2 * TL_BK);          // (its slots have been read: their values are stored)
        }
        const float* a_s = tl_smem + buf * STAGE;
        const float* w_s = a_s + A_FLOATS;
#pragma unroll
        for (int kk = 0; kk < TL_BK; ++kk) {
            const int x = (kk >> 2) << 3;
            float2 b[2 * TL_NH];
#pragma unroll
            for (int h = 0; h < TL_NH; ++h) {
                const float4 v = *reinterpret_cast<const float4*>(w_s + kk * TL_BN + h * 64 + ((tx * 4) ^ x));
                b[2 * h] = make_float2(v.x, v.y), b[2 * h + 1] = make_float2(v.z, v.w);
            }
            const float4 a0 = *reinterpret_cast<const float4*>(a_s + kk * TL_BM + ((ty * 4) ^ x));
            const float4 a1 = *reinterpret_cast<const float4*>(a_s + kk * TL_BM + 32 + ((ty * 4) ^ x));
            const float a[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w};
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const float2 aa = make_float2(a[i], a[i]);
#pragma unroll
                for (int j = 0; j < 2 * TL_NH; ++j) fma2(acc[i][j], aa, b[j]);
            }
        }
        if (!SPLIT) {
            left -= TL_BK;
            if (left == 0 || k0 + TL_BK >= k_end) {                     // the slice is complete
                left = slice;
#pragma unroll
                for (int i = 0; i < 8; ++i)
#pragma unroll
                    for (int j = 0; j < 2 * TL_NH; ++j) {
                        total[i][j].x += acc[i][j].x;
                        total[i][j].y += acc[i][j].y;
                        acc[i][j] = make_float2(0.0f, 0.0f);
                    }
            }
        }
        __syncthreads();
        buf ^= 1;
    }
    auto store = [&](int m, int n, const float (&v)[4]) {               // four features of one row
        if (m >= M) return;
        TC* out = C + (long)m * ldc + n;
        if (sizeof(TC) == 4 && n + 4 <= N && ((uintptr_t)out & 15) == 0) {
            *reinterpret_cast<float4*>(out) = make_float4(v[0], v[1], v[2], v[3]);
        } else {
#pragma unroll
            for (int j = 0; j < 4; ++j)
                if (n + j < N) out[j] = from_f32<TC>(v[j]);
        }
    };
    if constexpr (!SPLIT) {
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
            for (int h = 0; h < TL_NH; ++h) {
                const float v[4] = {total[i][2 * h].x, total[i][2 * h].y, total[i][2 * h + 1].x, total[i][2 * h + 1].y};
                store(m0 + (i >> 2) * 32 + ty * 4 + (i & 3), n0 + h * 64 + tx * 4, v);
            }
    } else {
        namespace cg = cooperative_groups;
        cg::cluster_group cluster = cg::this_cluster();
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
            for (int h = 0; h < TL_NH; ++h)
                *reinterpret_cast<float4*>(tl_smem + ((i >> 2) * 32 + ty * 4 + (i & 3)) * TL_BN + h * 64 + tx * 4) =
                    make_float4(acc[i][2 * h].x, acc[i][2 * h].y, acc[i][2 * h + 1].x, acc[i][2 * h + 1].y);
        cluster.sync();
        // an eighth of the tile's rows are this CTA's to add up: four features a thread
#pragma unroll
        for (int e = tid; e < TL_BM / GS_SLICES * TL_BN / 4; e += TL_THREADS) {
            const int r = (int)blockIdx.z * (TL_BM / GS_SLICES) + e / (TL_BN / 4), c = e % (TL_BN / 4) * 4;
            float sum[4] = {};
#pragma unroll
            for (int z = 0; z < GS_SLICES; ++z) {
                const float4 v = *reinterpret_cast<const float4*>(cluster.map_shared_rank(tl_smem, z) + r * TL_BN + c);
                sum[0] += v.x, sum[1] += v.y, sum[2] += v.z, sum[3] += v.w;
            }
            store(m0 + r, n0 + c, sum);
        }
        cluster.sync();                                                 // no CTA leaves while another reads its sums
    }
}

template <typename TC, int EACH>
__global__ void __cluster_dims__(1, 1, GS_SLICES) __launch_bounds__(TL_THREADS, EACH)
    gemm_f32_tile_kernel(const float* __restrict__ A, long lda, const float* __restrict__ W, long ldw, TC* __restrict__ C,
                         long ldc, int M, int N, int K, int slice) {
    pdl_wait();
    pdl_trigger();
    gemm_f32_tile<TC, true>(A, lda, W, ldw, C, ldc, M, N, K, slice);
}

template <typename TC>
__global__ void __launch_bounds__(TL_THREADS, 2)
    gemm_f32_whole_tile_kernel(const float* __restrict__ A, long lda, const float* __restrict__ W, long ldw, TC* __restrict__ C,
                               long ldc, int M, int N, int K, int slice) {
    pdl_wait();
    pdl_trigger();
    gemm_f32_tile<TC, false>(A, lda, W, ldw, C, ldc, M, N, K, slice);
}

// ------------------------------------------------------------ host side
template <typename TC, int MT, int RT>
static int gs_skinny(const float* A, long lda, const float* W, long ldw, TC* C, long ldc, int M, int N, int K, int constant_w, cudaStream_t stream) {
    using L = Skinny<MT, RT>;
    auto kernel = gemm_f32_skinny_kernel<TC, MT, RT>;
    cudaError_t err = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, L::SMEM);
    if (err != cudaSuccess) return (int)err;
    return fl_launch(kernel, dim3((N + L::R - 1) / L::R), dim3(64), L::SMEM, stream, A, lda, W, ldw, C, ldc, M, N, K, gs_slice(K), constant_w);
}

// Features a CTA: two for a thread (RT = 2, above), but one where that leaves SMs idle or busy unevenly.  What is compared is the
// features that the busiest SM gets.  Up to two rows, out of a cold cache: 256 of 2048 inputs 3.6 us with one and 4.2 with two,
// 5504 11.6 and 12.4, 2048 6.2 and 5.5, 32256 60.8 and 48.7.  From three rows on two are the better ones as soon as every SM
// has some (1024 of 2048 4.8 and 5.7 us, 2048 6.7 and 6.4, 5504 15.5 and 12.9).
template <typename TC, int MT>
static int gs_few_rows(const float* A, long lda, const float* W, long ldw, TC* C, long ldc, int M, int N, int K, int sms, int constant_w,
                       cudaStream_t stream) {
    const int one = ((N + 7) / 8 + sms - 1) / sms, two = 2 * (((N + 15) / 16 + sms - 1) / sms);
    if (one < two && (MT <= 2 || one == 1)) return gs_skinny<TC, MT, 1>(A, lda, W, ldw, C, ldc, M, N, K, constant_w, stream);
    return gs_skinny<TC, MT, 2>(A, lda, W, ldw, C, ldc, M, N, K, constant_w, stream);
}

template <typename TC, int EACH>
static int gs_split(dim3 grid, int smem, const float* A, long lda, const float* W, long ldw, TC* C, long ldc, int M, int N, int K, int slice,
                    cudaStream_t stream) {
    auto kernel = gemm_f32_tile_kernel<TC, EACH>;
    cudaError_t err = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 116 * 1024);
    if (err != cudaSuccess) return (int)err;
    return fl_launch(kernel, grid, dim3(TL_THREADS), smem, stream, A, lda, W, ldw, C, ldc, M, N, K, slice);
}

// The time of a product in whole and in split tiles, microseconds, fitted to 220 products of 17 to 2048 rows, 64 to 32000
// features and 16 to 5504 inputs.  Whole tiles, two an SM: 0.094 us an input for a round of them (0.06 where there is one an
// SM).  Split ones, four CTAs an SM: 0.19 us an input of a slice, and 6 us for a round's start and exchange, which is what a
// slice of 32 inputs costs too: 2048 x 2048 x 64 takes 60 us split and 15 whole, 500 x 2048 x 128 19 and 9.6, 1024 x 32000 x 256
// 469 and 349; 300 x 2048 x 256 14 and 18, 300 x 5504 x 2048 162 and 201.  The choice is right or within 3 %.
static double gs_whole_us(long tiles, int K, int sms) {
    const long rest = tiles % (2 * sms);
    const double round = 3.0 + 0.0935 * K;
    return tiles / (2 * sms) * round + (rest == 0 ? 0.0 : rest <= sms ? 1.7 + 0.06 * K : round);
}
static double gs_split_us(long tiles, int slice, int sms) {
    const long ctas = tiles * GS_SLICES, rest = ctas % (4 * sms);
    if (ctas <= sms * 7 / 4) return 1.5 + 0.011 * ctas + 0.098 * slice;          // all at once, two an SM at most
    return 3.0 + (2.9 + 0.188 * slice) * (ctas / (4 * sms) + (rest + sms - 1) / sms * 0.25);
}

// Float operands that 16-byte loads can read.  Up to 16 rows W's bytes decide and the skinny kernel streams them; above,
// the multiply-adds do (17 rows, 2048 x 2048: 31 us in tiles; the skinny kernel takes 14.5 for each 16 rows).
template <typename TC>
static int gs_f32(const float* A, long lda, const float* W, long ldw, TC* C, long ldc, int M, int N, int K, int sms,
                  int constant_w, cudaStream_t stream) {
    if (M <= 1) return gs_few_rows<TC, 1>(A, lda, W, ldw, C, ldc, M, N, K, sms, constant_w, stream);
    if (M <= 2) return gs_few_rows<TC, 2>(A, lda, W, ldw, C, ldc, M, N, K, sms, constant_w, stream);
    if (M <= 4) return gs_few_rows<TC, 4>(A, lda, W, ldw, C, ldc, M, N, K, sms, constant_w, stream);
    if (M <= 8) return gs_skinny<TC, 8, 2>(A, lda, W, ldw, C, ldc, M, N, K, constant_w, stream);
    if (M <= 16) return gs_skinny<TC, 16, 2>(A, lda, W, ldw, C, ldc, M, N, K, constant_w, stream);
    dim3 grid((N + TL_BN - 1) / TL_BN, (M + TL_BM - 1) / TL_BM, GS_SLICES);
    if (grid.y > 65535) return (int)cudaErrorInvalidValue;
    const int slice = gs_slice(K);
    if (gs_whole_us((long)grid.x * grid.y, K, sms) < gs_split_us((long)grid.x * grid.y, slice, sms)) {
        grid.z = 1;
        return fl_launch(gemm_f32_whole_tile_kernel<TC>, grid, dim3(TL_THREADS), TL_SMEM, stream, A, lda, W, ldw, C, ldc, M, N, K, slice);
    }
    // Four CTAs fit an SM, and the clusters of a product of few tiles would be packed so, beside idle SMs: more shared memory
    // than they use keeps one, two or three an SM where that many hold all tiles (100 x 2048 x 2048: 36.4 us so packed, 31.8
    // two an SM), and there they may use more registers (29.8).  A cluster lies within a GPC: at one CTA an SM they reach 3 of 4
    // SMs (of 16 tiles one waits for another to end: 17 x 2048 x 2048 took 39.6 us), at two or three 7 of 8.
    for (int each = 1; each < 4; ++each)
        if ((long)grid.x * grid.y * GS_SLICES <= (each == 1 ? sms * 3L / 4 : (long)sms * each * 7 / 8))
            return gs_split<TC, 3>(grid, 228 * 1024 / (each + 1) - 1024 + 128, A, lda, W, ldw, C, ldc, M, N, K, slice, stream);
    return gs_split<TC, 4>(grid, TL_SMEM, A, lda, W, ldw, C, ldc, M, N, K, slice, stream);      // (a CTA takes 1 KB more than it asks for)
}

// constant_w: no kernel that may still run when this one is launched writes W (which is then read ahead of it).
FL_API int fl_gemm_simt(const void* A, int a_dtype, long lda, const void* W, int w_dtype, long ldw,
                        void* C, int c_dtype, long ldc, int M, int N, int K, int sms, int constant_w, cudaStream_t stream) {
    if (M <= 0 || N <= 0) return 0;
    if (a_dtype == FL_F32 && w_dtype == FL_F32 && K > 0 && K % 4 == 0 && lda % 4 == 0 && ldw % 4 == 0 &&
        ((uintptr_t)A | (uintptr_t)W) % 16 == 0) {
        FL_DISPATCH(c_dtype, TC, return gs_f32<TC>((const float*)A, lda, (const float*)W, ldw, (TC*)C, ldc, M, N, K, sms, constant_w, stream));
    }
    dim3 grid((N + GS_BN - 1) / GS_BN, (M + GS_BM - 1) / GS_BM);
    if (grid.y > 65535) return (int)cudaErrorInvalidValue;
    FL_DISPATCH(a_dtype, TA, FL_DISPATCH(w_dtype, TW, FL_DISPATCH(c_dtype, TC,
        return fl_launch(gemm_simt_kernel<TA, TW, TC>, grid, dim3(256), 0, stream, (const TA*)A, lda,
                         (const TW*)W, ldw, (TC*)C, ldc, M, N, K, gs_slice(K), 0L, 0L, 0L))));
    return 0;
}

// `batch` products of one shape in one launch: product b reads A + b * a_batch and W + b * w_batch and
// writes C + b * c_batch (strides in elements).  With a_batch and c_batch smaller than a row this is a
// product per head over the column blocks of [M, heads x K] and [M, heads x N] buffers.
FL_API int fl_gemm_simt_batched(const void* A, int a_dtype, long lda, long a_batch, const void* W, int w_dtype,
                                long ldw, long w_batch, void* C, int c_dtype, long ldc, long c_batch, int M, int N,
                                int K, int batch, cudaStream_t stream) {
    if (M <= 0 || N <= 0 || batch <= 0) return 0;
    dim3 grid((N + GS_BN - 1) / GS_BN, (M + GS_BM - 1) / GS_BM, batch);
    if (grid.y > 65535 || batch > 65535) return (int)cudaErrorInvalidValue;
    FL_DISPATCH(a_dtype, TA, FL_DISPATCH(w_dtype, TW, FL_DISPATCH(c_dtype, TC,
        return fl_launch(gemm_simt_kernel<TA, TW, TC>, grid, dim3(256), 0, stream, (const TA*)A, lda,
                         (const TW*)W, ldw, (TC*)C, ldc, M, N, K, gs_slice(K), a_batch, w_batch, c_batch))));
    return 0;
}
