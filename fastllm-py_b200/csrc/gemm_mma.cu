// Batched bfloat16 product on tensor cores (mma.sync m16n8k16, float accumulation):
//     C_b[M, N] = A_b[M, K] * W_b[N, K]^T   for b = 0 .. batch - 1
// where A_b and C_b are column blocks of wider row-major buffers (A + b * a_batch, C + b * c_batch, in
// elements) and W is [batch][N][K].  This is the product per head that stands on either side of latent
// attention (a head's query block through its own small matrix), for steps of any size: a block takes 64
// rows x 128 columns (32 where there are no more than 64 rows: a step of few tokens is bound by the way of W's rows through
// a few blocks, and the more blocks share it the better) of one batch entry, K in steps of 32 through a cp.async ring of 3
// (6) stages with one barrier a step.  The tile leaves by way of shared memory, 16 bytes a thread and whole rows of it side by
// side where C's rows allow: element by element the stores of 2048 rows x 16 x 512 columns took most of the time.  Bound by its stores (33 MB), else by
// one block's serial way through K: 16 products of K = 128 and N = 512 took 3.5 us for 4 rows, 17.2 for 300 and 55.7 for 2048
// in blocks of 64 x 64 and a ring of 3 stages, and take 2.5, 6.0 and 23.7; of K = 512 and N = 128 8.1, 11.6 and 33.6, now 4.2,
// 7.7 and 22.2.
// With `gate` (laid out like C: gate + b * g_batch, ldg between rows) the epilogue writes C * sigmoid(gate): the
// product is rounded to C's type first, as a gate applied by a kernel of its own would have read it.
// K must be a multiple of 32 and every A row 16-byte aligned; other shapes go to gemm_simt's batched form.
#include "common.cuh"

#define GM_BM 64
#define GM_BK 32
#define GM_PITCH 40              // bfloat16 elements between staged rows: ldmatrix without bank conflicts

template <int BN> struct GmTile {
    static constexpr int STAGES = BN == 128 ? 3 : 6;
    static constexpr int STAGE = (GM_BM + BN) * GM_PITCH;               // elements: rows of A, then rows of W
    static constexpr int WN = BN / 4, NT = WN / 8;                      // columns of a warp, in eights
    static constexpr int OUT_PITCH = BN + 8;                            // of the tile on its way out
    static constexpr int BYTES = STAGES * STAGE * 2 > GM_BM * OUT_PITCH * 4 ? STAGES * STAGE * 2 : GM_BM * OUT_PITCH * 4;
};

// `there` false: zeroes, and nothing is read.  (Rows past M that all read the last row again meet in the same few sectors of
// L2: 8 rows x 16 heads x 512 columns took 7.1 us, 2.5 with zeroes.)
__device__ __forceinline__ void gm_cp16(void* smem, const void* gmem, bool there) {
    const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(s), "l"(gmem), "r"(there ? 16 : 0));
}

// wide: C's rows (and the gate's) are whole and aligned pieces of 16 bytes
template <typename TC, int BN>
__global__ void __launch_bounds__(256) gemm_mma_batched_kernel(const bf16* __restrict__ A, long lda, long a_batch,
                                                               const bf16* __restrict__ W, TC* __restrict__ C, long ldc,
                                                               long c_batch, int M, int N, int K,
                                                               const TC* __restrict__ gate, long ldg, long g_batch, int wide) {
    using L = GmTile<BN>;
    pdl_wait();
    pdl_trigger();
    __shared__ __align__(16) unsigned char gm_raw[L::BYTES];
    bf16* ring = reinterpret_cast<bf16*>(gm_raw);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int wm = warp >> 2, wn = warp & 3;                    // 2 x 4 warps, 32 rows x WN columns each
    const int m0 = blockIdx.x * GM_BM, n0 = blockIdx.y * BN, b = blockIdx.z;
    const int ar = tid >> 2, ac = (tid & 3) * 8;                // this thread's 16-byte pieces of a stage
    const bf16* a_src = A + b * a_batch + (long)min(m0 + ar, M - 1) * lda + ac;
    constexpr int W_PIECES = (BN + 63) / 64;
    const bf16* w_src[W_PIECES];
#pragma unroll
    for (int i = 0; i < W_PIECES; ++i) w_src[i] = W + ((long)b * N + min(n0 + ar + i * 64, N - 1)) * K + ac;
    const int n_k = K / GM_BK;
    auto stage = [&](int kb) {                                  // (also past the last one: the ring counts groups of copies)
        if (kb < n_k) {
            bf16* dst = ring + kb % L::STAGES * L::STAGE + ar * GM_PITCH + ac;
            gm_cp16(dst, a_src + kb * GM_BK, m0 + ar < M);
#pragma unroll
            for (int i = 0; i < W_PIECES; ++i)
                if (BN >= 64 || ar < BN) gm_cp16(dst + (GM_BM + i * 64) * GM_PITCH, w_src[i] + kb * GM_BK, n0 + ar + i * 64 < N);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    float acc[2][L::NT][4];
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < L::NT; ++j) acc[i][j][0] = acc[i][j][1] = acc[i][j][2] = acc[i][j][3] = 0.0f;
#pragma unroll
    for (int kb = 0; kb < L::STAGES - 1; ++kb) stage(kb);
    for (int kb = 0; kb < n_k; ++kb) {
        asm volatile("cp.async.wait_group %0;" ::"n"(L::STAGES - 2) : "memory");
        __syncthreads();                                        // stage kb is there, stage kb - 1 has been read
        stage(kb + L::STAGES - 1);
        const bf16* a_s = ring + kb % L::STAGES * L::STAGE;
        const bf16* w_s = a_s + GM_BM * GM_PITCH;
#pragma unroll
        for (int ks = 0; ks < GM_BK; ks += 16) {
            unsigned af[2][4], bfr[L::NT][2];
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const unsigned s = (unsigned)__cvta_generic_to_shared(a_s + (wm * 32 + i * 16 + (lane & 15)) * GM_PITCH + ks + (lane >> 4) * 8);
                asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
                             : "=r"(af[i][0]), "=r"(af[i][1]), "=r"(af[i][2]), "=r"(af[i][3]) : "r"(s));
            }
            if constexpr (L::NT == 1) {
                const unsigned s = (unsigned)__cvta_generic_to_shared(w_s + (wn * 8 + (lane & 7)) * GM_PITCH + ks + ((lane >> 3) & 1) * 8);
                asm volatile("ldmatrix.sync.aligned.m8n8.x2.shared.b16 {%0,%1}, [%2];" : "=r"(bfr[0][0]), "=r"(bfr[0][1]) : "r"(s));
            } else {
#pragma unroll
                for (int j2 = 0; j2 < L::NT / 2; ++j2) {
                    const unsigned s = (unsigned)__cvta_generic_to_shared(
                        w_s + (wn * L::WN + j2 * 16 + (lane & 7) + (lane >> 4) * 8) * GM_PITCH + ks + ((lane >> 3) & 1) * 8);
                    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
                                 : "=r"(bfr[j2 * 2][0]), "=r"(bfr[j2 * 2][1]), "=r"(bfr[j2 * 2 + 1][0]), "=r"(bfr[j2 * 2 + 1][1])
                                 : "r"(s));
                }
            }
#pragma unroll
            for (int i = 0; i < 2; ++i)
#pragma unroll
                for (int j = 0; j < L::NT; ++j)
                    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                                 : "+f"(acc[i][j][0]), "+f"(acc[i][j][1]), "+f"(acc[i][j][2]), "+f"(acc[i][j][3])
                                 : "r"(af[i][0]), "r"(af[i][1]), "r"(af[i][2]), "r"(af[i][3]), "r"(bfr[j][0]), "r"(bfr[j][1]));
        }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();                                            // the ring has been read: the tile takes its place
    TC* tile = reinterpret_cast<TC*>(gm_raw);
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int half = 0; half < 2; ++half)
#pragma unroll
            for (int j = 0; j < L::NT; ++j)
#pragma unroll
                for (int c = 0; c < 2; ++c)
                    tile[(wm * 32 + i * 16 + (lane >> 2) + half * 8) * L::OUT_PITCH + wn * L::WN + j * 8 + (lane & 3) * 2 + c] =
                        from_f32<TC>(acc[i][j][half * 2 + c]);
    __syncthreads();
    TC* c_base = C + b * c_batch;
    const TC* g_base = gate != nullptr ? gate + b * g_batch : nullptr;
    constexpr int V = 16 / (int)sizeof(TC), PIECES = BN / V;
    for (int e = tid; e < GM_BM * PIECES; e += 256) {
        const int r = e / PIECES, m = m0 + r, n = n0 + (e - r * PIECES) * V;
        if (m >= M || n >= N) continue;
        __align__(16) TC v[V];
        *reinterpret_cast<uint4*>(v) = *reinterpret_cast<const uint4*>(tile + r * L::OUT_PITCH + n - n0);
        if (wide) {
            if (g_base != nullptr) {
                __align__(16) TC g[V];
                *reinterpret_cast<uint4*>(g) = *reinterpret_cast<const uint4*>(g_base + (long)m * ldg + n);
#pragma unroll
                for (int c = 0; c < V; ++c) v[c] = from_f32<TC>(to_f32<TC>(v[c]) / (1.0f + expf(-to_f32<TC>(g[c]))));
            }
            *reinterpret_cast<uint4*>(c_base + (long)m * ldc + n) = *reinterpret_cast<const uint4*>(v);
        } else {
#pragma unroll
            for (int c = 0; c < V; ++c) {
                if (n + c >= N) break;
                TC x = v[c];
                if (g_base != nullptr) x = from_f32<TC>(to_f32<TC>(x) / (1.0f + expf(-to_f32<TC>(g_base[(long)m * ldg + n + c]))));
                c_base[(long)m * ldc + n + c] = x;
            }
        }
    }
}

template <typename TC, int BN>
static int gm_launch(const void* A, long lda, long a_batch, const void* W, void* C, long ldc, long c_batch, int M, int N, int K,
                     int batch, const void* gate, long ldg, long g_batch, cudaStream_t stream) {
    constexpr int V = 16 / (int)sizeof(TC);
    const bool wide = N % V == 0 && ldc % V == 0 && c_batch % V == 0 && ((uintptr_t)C % 16) == 0 &&
                      (gate == nullptr || (ldg % V == 0 && g_batch % V == 0 && ((uintptr_t)gate % 16) == 0));
    return fl_launch(gemm_mma_batched_kernel<TC, BN>, dim3((M + GM_BM - 1) / GM_BM, (N + BN - 1) / BN, batch), dim3(256), 0, stream,
                     (const bf16*)A, lda, a_batch, (const bf16*)W, (TC*)C, ldc, c_batch, M, N, K, (const TC*)gate, ldg, g_batch,
                     (int)wide);
}

FL_API int fl_gemm_mma_batched_takes(long lda, long a_batch, int K, const void* A) {
    return K % GM_BK == 0 && lda % 8 == 0 && a_batch % 8 == 0 && ((uintptr_t)A % 16) == 0;
}

FL_API int fl_gemm_mma_batched(const void* A, long lda, long a_batch, const void* W, void* C, int c_dtype, long ldc,
                               long c_batch, int M, int N, int K, int batch, const void* gate, long ldg, long g_batch,
                               cudaStream_t stream) {
    if (M <= 0 || N <= 0 || batch <= 0) return 0;
    if (!fl_gemm_mma_batched_takes(lda, a_batch, K, A) || ((uintptr_t)W % 16) || batch > 65535 || (N + 127) / 128 > 65535)
        return (int)cudaErrorInvalidValue;
    FL_DISPATCH(c_dtype, TC, {
        if (M <= GM_BM && (N + 31) / 32 <= 65535)
            return (gm_launch<TC, 32>(A, lda, a_batch, W, C, ldc, c_batch, M, N, K, batch, gate, ldg, g_batch, stream));
        return (gm_launch<TC, 128>(A, lda, a_batch, W, C, ldc, c_batch, M, N, K, batch, gate, ldg, g_batch, stream));
    });
    return 0;
}
