// Latent attention on tensor cores, one build per (LAT_RANK, LAT_ROT): a kernel for any step on bfloat16 mma.sync m16n8k16
// with its merge of splits, and one for steps of prompts on tcgen05 (see the second half of the file), which gives the first
// one's bits.
//
// The same computation as latent_attention.cu's kernel: per token and head, softmax over the visible
// cache rows of q~ . [c | rotated part] * scale, then the weighted sum of the rows' first LAT_RANK
// elements.  All heads share a token's rows, so a block takes one token and 16 heads as the 16 rows of
// the MMA's A operand: decode steps use the tensor cores at full width, and a cache row that a block
// stages in shared memory serves 16 heads.
//
// A block has 4 warps and walks the keys in tiles of 32 (aligned to absolute positions), two tiles in
// flight through cp.async.  Per tile: warp w computes the scores of keys 8w..8w+7 (q~ from shared
// memory, the rows as the col-major B operand), the row maxima and sums cross the warps through shared
// memory, the probabilities go to shared memory in bfloat16, and warp w accumulates its quarter of the
// value columns over all 32 keys (the staged rows read through ldmatrix.trans).  Scores, maxima, sums and
// the output accumulator are float; the accumulator is rescaled at every tile.
#include "common.cuh"

#ifndef LAT_RANK
#error "build with -DLAT_RANK=<latent size> -DLAT_ROT=<rotated key size>"
#endif
#define LT_WIDTH (LAT_RANK + LAT_ROT)
#define LT_PITCH (LT_WIDTH + 8)          // bfloat16 elements between staged rows (ldmatrix without bank conflicts)
#define LT_KEYS 32
#define LT_WARPS 4
#define LT_VCOLS (LAT_RANK / LT_WARPS)   // value columns of a warp
#define LT_NT (LT_VCOLS / 8)
#define LT_PPITCH (LT_KEYS + 8)
static_assert(LAT_RANK % 32 == 0 && LT_WIDTH % 16 == 0, "latent size must be a multiple of 32, row width of 16");

__device__ __forceinline__ void lt_cp16(void* smem, const void* gmem, int bytes) {
    const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(s), "l"(gmem), "r"(bytes));
}

#define LT_SMEM ((16 * LT_PITCH + 2 * LT_KEYS * LT_PITCH + 16 * LT_PPITCH) * 2 + 2 * LT_WARPS * 16 * 4)

// Among the threads of `latent_token`: the whole block, or the first four warps of a larger one.
template <bool WHOLE> __device__ __forceinline__ void lt_sync() {
    if (WHOLE) __syncthreads();
    else asm volatile("bar.sync 1, %0;" ::"n"(LT_WARPS * 32) : "memory");
}

// One token and 16 heads, by threads 0 .. LT_WARPS * 32 - 1 of the block (WHOLE: it has no others) with LT_SMEM bytes at
// lt_smem.  q, out: the token's rows; bt: its request's row of the block table; partial: where the token's splits go.
template <typename TO, bool WHOLE>
__device__ __forceinline__ void latent_token(unsigned char* lt_smem, const bf16* __restrict__ q, TO* __restrict__ out,
                                             const bf16* __restrict__ cache, int page_size, const int* __restrict__ bt, int pos,
                                             int heads, int head0, int window, float scale, int split_keys, int split, int n_splits,
                                             float* __restrict__ partial, const float* __restrict__ sink) {
    bf16* q_s = reinterpret_cast<bf16*>(lt_smem);                         // [16][LT_PITCH]
    bf16* k_s = q_s + 16 * LT_PITCH;                                      // [2][LT_KEYS][LT_PITCH]
    bf16* p_s = k_s + 2 * LT_KEYS * LT_PITCH;                             // [16][LT_PPITCH]
    float* red_max = reinterpret_cast<float*>(p_s + 16 * LT_PPITCH);      // [LT_WARPS][16]
    float* red_sum = red_max + LT_WARPS * 16;                             // [LT_WARPS][16]
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int lo = window > 0 ? max(0, pos - window + 1) : 0;

    auto stage = [&](int buf, int tile) {
        bf16* dst = k_s + (long)buf * LT_KEYS * LT_PITCH;
        constexpr int CHUNKS = LT_WIDTH / 8;
        for (int c = tid; c < LT_KEYS * CHUNKS; c += LT_WARPS * 32) {
            const int r = c / CHUNKS, piece = c % CHUNKS;
            const int j = tile + r;
            const bool valid = j >= lo && j <= pos;
            const bf16* src = cache;
            if (valid) src = cache + ((long)bt[j / page_size] * page_size + j % page_size) * LT_WIDTH + piece * 8;
            lt_cp16(dst + r * LT_PITCH + piece * 8, src, valid ? 16 : 0);     // rows out of sight are zeros
        }
        asm volatile("cp.async.commit_group;");
    };
    // with split_keys (a multiple of LT_KEYS) the block takes only the keys of split `split`, counted from
    // the multiple of split_keys at or below the first visible key, and leaves (accumulator, maximum, sum)
    // in `partial` for the merge kernel; the splits' borders depend on the token's own position only
    int first_tile = (lo / LT_KEYS) * LT_KEYS, last = pos;
    if (split_keys > 0) {
        first_tile = (lo / split_keys + split) * split_keys;
        last = min(pos, first_tile + split_keys - 1);
        first_tile = max(first_tile, (lo / LT_KEYS) * LT_KEYS);      // (no tile wholly out of sight: its maximum would be -inf)
    }
    float* part_row = nullptr;
    if (split_keys > 0) {
        part_row = partial + (long)split * (LAT_RANK + 2);   // + head * n_splits * (rank + 2)
        if (first_tile > pos) {                              // nothing of this split is in sight
            for (int r = tid; r < 16 && head0 + r < heads; r += LT_WARPS * 32) {
                float* pr = part_row + (long)(head0 + r) * n_splits * (LAT_RANK + 2);
                pr[LAT_RANK] = -CUDART_INF_F;
                pr[LAT_RANK + 1] = 0.0f;
            }
            return;
        }
    }
    stage(0, first_tile);
    for (int c = tid; c < 16 * (LT_WIDTH / 8); c += LT_WARPS * 32) {     // the 16 heads' q~
        const int r = c / (LT_WIDTH / 8), piece = c % (LT_WIDTH / 8);
        uint4 v = make_uint4(0, 0, 0, 0);
        if (head0 + r < heads) v = *reinterpret_cast<const uint4*>(q + (long)(head0 + r) * LT_WIDTH + piece * 8);
        *reinterpret_cast<uint4*>(q_s + r * LT_PITCH + piece * 8) = v;
    }
    float acc[LT_NT][4];
#pragma unroll
    for (int n = 0; n < LT_NT; ++n) acc[n][0] = acc[n][1] = acc[n][2] = acc[n][3] = 0.0f;
    float m_run[2] = {-CUDART_INF_F, -CUDART_INF_F}, l_run[2] = {0.0f, 0.0f};   // rows lane / 4 and lane / 4 + 8
    const int row0 = lane >> 2;
    if (sink != nullptr && split_keys == 0) {                // the running maximum and sum start from the sink's term
#pragma unroll
        for (int h = 0; h < 2; ++h)
            if (head0 + row0 + h * 8 < heads) {
                m_run[h] = sink[head0 + row0 + h * 8];
                l_run[h] = 1.0f;
            }
    }
    int buf = 0;
    for (int tile = first_tile; tile <= last; tile += LT_KEYS, buf ^= 1) {
        if (tile + LT_KEYS <= last) {
            stage(buf ^ 1, tile + LT_KEYS);
            asm volatile("cp.async.wait_group 1;");
        } else {
            asm volatile("cp.async.wait_group 0;");
        }
        lt_sync<WHOLE>();
        const bf16* ks = k_s + (long)buf * LT_KEYS * LT_PITCH;
        // ---- scores of this warp's 8 keys
        float s[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll 4
        for (int kk = 0; kk < LT_WIDTH; kk += 16) {
            unsigned a[4], b[2];
            const unsigned qa = (unsigned)__cvta_generic_to_shared(q_s + (lane & 15) * LT_PITCH + kk + (lane >> 4) * 8);
            asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
                         : "=r"(a[0]), "=r"(a[1]), "=r"(a[2]), "=r"(a[3]) : "r"(qa));
            const unsigned ka = (unsigned)__cvta_generic_to_shared(ks + (warp * 8 + (lane & 7)) * LT_PITCH + kk + ((lane >> 3) & 1) * 8);
            asm volatile("ldmatrix.sync.aligned.m8n8.x2.shared.b16 {%0,%1}, [%2];" : "=r"(b[0]), "=r"(b[1]) : "r"(ka));
            asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                         : "+f"(s[0]), "+f"(s[1]), "+f"(s[2]), "+f"(s[3])
                         : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
        }
        const int j0 = tile + warp * 8 + (lane & 3) * 2;
        float mx[2];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                const int j = j0 + c;
                s[h * 2 + c] = (j >= lo && j <= pos) ? s[h * 2 + c] * scale : -CUDART_INF_F;
            }
            mx[h] = fmaxf(s[h * 2], s[h * 2 + 1]);
            mx[h] = fmaxf(mx[h], __shfl_xor_sync(0xffffffffu, mx[h], 1));
            mx[h] = fmaxf(mx[h], __shfl_xor_sync(0xffffffffu, mx[h], 2));
        }
        if ((lane & 3) == 0) {
            red_max[warp * 16 + row0] = mx[0];
            red_max[warp * 16 + row0 + 8] = mx[1];
        }
        lt_sync<WHOLE>();
        float corr[2];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int r = row0 + h * 8;
            float m_new = m_run[h];
#pragma unroll
            for (int w = 0; w < LT_WARPS; ++w) m_new = fmaxf(m_new, red_max[w * 16 + r]);
            corr[h] = expf(m_run[h] - m_new);               // 0 at the first tile without a sink
            m_run[h] = m_new;
            const float p0 = expf(s[h * 2] - m_new), p1 = expf(s[h * 2 + 1] - m_new);   // exp(-inf) = 0 out of sight
            float sum = p0 + p1;
            sum += __shfl_xor_sync(0xffffffffu, sum, 1);
            sum += __shfl_xor_sync(0xffffffffu, sum, 2);
            if ((lane & 3) == 0) red_sum[warp * 16 + r] = sum;
            *reinterpret_cast<__nv_bfloat162*>(p_s + r * LT_PPITCH + warp * 8 + (lane & 3) * 2) = __floats2bfloat162_rn(p0, p1);
        }
        lt_sync<WHOLE>();
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            float sum = 0.0f;
#pragma unroll
            for (int w = 0; w < LT_WARPS; ++w) sum += red_sum[w * 16 + row0 + h * 8];
            l_run[h] = l_run[h] * corr[h] + sum;
        }
#pragma unroll
        for (int n = 0; n < LT_NT; ++n) {
            acc[n][0] *= corr[0]; acc[n][1] *= corr[0];
            acc[n][2] *= corr[1]; acc[n][3] *= corr[1];
        }
        // ---- this warp's value columns over the tile's 32 keys
#pragma unroll
        for (int kk = 0; kk < LT_KEYS; kk += 16) {
            unsigned a[4];
            const unsigned pa = (unsigned)__cvta_generic_to_shared(p_s + (lane & 15) * LT_PPITCH + kk + (lane >> 4) * 8);
            asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
                         : "=r"(a[0]), "=r"(a[1]), "=r"(a[2]), "=r"(a[3]) : "r"(pa));
#pragma unroll
            for (int n = 0; n < LT_NT; ++n) {
                unsigned b[2];
                const unsigned va = (unsigned)__cvta_generic_to_shared(ks + (kk + (lane & 15)) * LT_PITCH + warp * LT_VCOLS + n * 8);
                asm volatile("ldmatrix.sync.aligned.m8n8.x2.trans.shared.b16 {%0,%1}, [%2];" : "=r"(b[0]), "=r"(b[1]) : "r"(va));
                asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                             : "+f"(acc[n][0]), "+f"(acc[n][1]), "+f"(acc[n][2]), "+f"(acc[n][3])
                             : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
            }
        }
        lt_sync<WHOLE>();                                     // the tile, p_s and the reductions are rewritten next
    }
    if (split_keys > 0) {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int head = head0 + row0 + h * 8;
            if (head >= heads) continue;
            float* pr = part_row + (long)head * n_splits * (LAT_RANK + 2);
            float* o = pr + warp * LT_VCOLS + (lane & 3) * 2;
#pragma unroll
            for (int n = 0; n < LT_NT; ++n) {
                o[n * 8] = acc[n][h * 2];
                o[n * 8 + 1] = acc[n][h * 2 + 1];
            }
            if (warp == 0 && (lane & 3) == 0) {
                pr[LAT_RANK] = m_run[h];
                pr[LAT_RANK + 1] = l_run[h];
            }
        }
        return;
    }
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const int head = head0 + row0 + h * 8;
        if (head >= heads) continue;
        TO* o = out + (long)head * LAT_RANK + warp * LT_VCOLS + (lane & 3) * 2;
        const float inv = 1.0f / l_run[h];
#pragma unroll
        for (int n = 0; n < LT_NT; ++n) {
            o[n * 8] = from_f32<TO>(acc[n][h * 2] * inv);
            o[n * 8 + 1] = from_f32<TO>(acc[n][h * 2 + 1] * inv);
        }
    }
}

template <typename TO>
__global__ void __launch_bounds__(LT_WARPS * 32) latent_attention_tc_kernel(
    const bf16* __restrict__ q, long q_ld, TO* __restrict__ out, long out_ld, const bf16* __restrict__ cache,
    int page_size, const int* __restrict__ block_table, int bt_stride, const int* __restrict__ tok_req,
    const int* __restrict__ positions, int heads, int window, float scale, int split_keys, float* __restrict__ partial, const float* __restrict__ sink) {
    pdl_wait();
    pdl_trigger();
    extern __shared__ __align__(16) unsigned char lt_smem[];
    const int t = blockIdx.x;
    latent_token<TO, true>(lt_smem, q + (long)t * q_ld, out + (long)t * out_ld, cache, page_size,
                           block_table + (long)tok_req[t] * bt_stride, positions[t], heads, blockIdx.y * 16, window, scale,
                           split_keys, blockIdx.z, gridDim.z,
                           split_keys > 0 ? partial + (long)t * heads * gridDim.z * (LAT_RANK + 2) : nullptr, sink);
}

// out[t, head] = sum_z acc_z e^(m_z - M) / ([e^(sink - M) +] sum_z l_z e^(m_z - M)), splits in order; one block per (token, head).
template <typename TO>
__global__ void __launch_bounds__(128) latent_merge_kernel(const float* __restrict__ partial, TO* __restrict__ out,
                                                           long out_ld, int heads, int n_splits, const float* __restrict__ sink) {
    pdl_wait();
    pdl_trigger();
    const int t = blockIdx.x, head = blockIdx.y;
    const float* pr = partial + ((long)t * heads + head) * n_splits * (LAT_RANK + 2);
    float mx = sink != nullptr ? sink[head] : -CUDART_INF_F;
    for (int z = 0; z < n_splits; ++z) mx = fmaxf(mx, pr[(long)z * (LAT_RANK + 2) + LAT_RANK]);
    float l = sink != nullptr ? expf(sink[head] - mx) : 0.0f;
    for (int z = 0; z < n_splits; ++z) {
        const float* p = pr + (long)z * (LAT_RANK + 2);
        if (p[LAT_RANK + 1] > 0.0f) l += p[LAT_RANK + 1] * expf(p[LAT_RANK] - mx);
    }
    for (int c = threadIdx.x; c < LAT_RANK; c += blockDim.x) {
        float sum = 0.0f;
        for (int z = 0; z < n_splits; ++z) {
            const float* p = pr + (long)z * (LAT_RANK + 2);
            if (p[LAT_RANK + 1] > 0.0f) sum += p[c] * expf(p[LAT_RANK] - mx);
        }
        out[(long)t * out_ld + (long)head * LAT_RANK + c] = from_f32<TO>(sum / l);
    }
}

FL_API int fl_latent_attention_tc_rank() { return LAT_RANK; }
FL_API int fl_latent_attention_tc_rot() { return LAT_ROT; }

// q: bfloat16 [n_tokens, heads x (rank + rot)], rows 16-byte aligned; out: float or bfloat16 [n_tokens, heads x rank];
// cache: bfloat16 [pages][page_size][rank + rot].  window <= 0: all earlier tokens.
// split_keys > 0 (a multiple of 32): the keys are shared out over n_splits blocks per token (decode steps,
// where tokens are too few to fill the GPU); `partial` then holds n_tokens * heads * n_splits * (rank + 2)
// floats and a merge kernel follows.  n_splits must reach the last key of every token:
// (longest visible span - 1) / split_keys + 2 does.  sink: [heads] float, a term exp(sink) of each head's denominator, or
// null.
FL_API int fl_latent_attention_tc(const void* q, long q_ld, void* out, int out_dtype, long out_ld, const void* cache, int page_size,
                                  const int* block_table, int bt_stride, const int* tok_req, const int* positions,
                                  int n_tokens, int heads, int window, float scale, int split_keys, int n_splits,
                                  float* partial, const float* sink, cudaStream_t stream) {
    if (n_tokens <= 0) return 0;
    if (split_keys < 0 || split_keys % LT_KEYS || (split_keys > 0 && (n_splits < 1 || n_splits > 65535 || partial == nullptr)))
        return (int)cudaErrorInvalidValue;
    if (((uintptr_t)q % 16) || (q_ld % 8) || ((uintptr_t)cache % 16) || (heads + 15) / 16 > 65535)
        return (int)cudaErrorInvalidValue;
    const size_t smem = LT_SMEM;
    static bool raised = false;
    if (!raised && smem > 48 * 1024) {
        cudaError_t rc = cudaFuncSetAttribute(latent_attention_tc_kernel<float>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (rc == cudaSuccess)
            rc = cudaFuncSetAttribute(latent_attention_tc_kernel<bf16>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (rc != cudaSuccess) return (int)rc;
        raised = true;
    }
    int rc = 0;
    FL_DISPATCH(out_dtype, TO,
        rc = fl_launch(latent_attention_tc_kernel<TO>, dim3(n_tokens, (heads + 15) / 16, split_keys > 0 ? n_splits : 1),
                       dim3(LT_WARPS * 32), smem, stream, (const bf16*)q, q_ld, (TO*)out, out_ld, (const bf16*)cache,
                       page_size, block_table, bt_stride, tok_req, positions, heads, window, scale, split_keys, partial, sink));
    if (rc || split_keys == 0) return rc;
    FL_DISPATCH(out_dtype, TO,
        return fl_launch(latent_merge_kernel<TO>, dim3(n_tokens, heads), dim3(128), 0, stream, (const float*)partial,
                         (TO*)out, out_ld, heads, n_splits, sink));
    return 0;
}

// ----------------------------------------------------------------- prompts: tcgen05
// Eight neighbouring tokens of a request x 16 heads are the 128 rows of tcgen05.mma, where the kernel above has 16 rows of
// mma.sync: a cache row that has been fetched serves 8 tokens.  (Prompt of 2048 tokens, 16 heads, rank 512, window 1024:
// 971 us with mma.sync, which fetched 1.8 GB of rows from L2 and kept its tensor cores 4 % busy, 224 us so.)  The sums are the other
// kernel's, one by one: the same tiles of 32 keys, scores and value sums in K steps of 16 from the first to the last, the
// weights' sums in the same tree, a rescaling at every tile where the maximum moved (where it did not, the other kernel
// multiplies by one), so results are the same bit for bit.
//
// A tile serves tokens that do not see all of its keys, with weights of zero, and zero times a value that is not finite is
// NaN, where the other kernel never reads keys out of a token's sight.  Such a key shows in its scores (a sum with a term
// that is not finite is not finite): where a score out of a token's sight is not finite, the CTA's tokens are done again
// token by token, by the other kernel's code.  Only tiles at a border of what the tokens see are looked at.
//
// Tensor memory holds 512 columns, so a CTA accumulates LP_VC = 256 value columns at most, and the CTAs of a tile's two
// halves both compute its scores.  Roles in a CTA of 320 threads:
//   warps 0-3  a row's weights: scores from tensor memory, maximum, exponentials, the weights as bfloat16 back into tensor
//              memory (the A operand of the second product)
//   warps 4-7  the same rows' accumulators: rescaled (read, multiplied, written) while the exponentials are made; output
//   warp 8     TMA: queries once, then the keys' pages, LP_STAGES tiles ahead; a page that no row sees is fetched from
//              beyond the tensor, which gives zeros
//   warp 9     the MMAs: scores of tile i + 1, then values of tile i
// Two thirds of the queries are kept in tensor memory (written there once by warps 0-7): the score MMAs that take them from
// there do not read 4 KB of shared memory each, and four tiles of keys find room instead of two, so that a tile's way through
// L2 is hidden.  (With all of the queries in shared memory that way showed between any two tiles: a tile's stage is free only
// after its values, which come after the next tile's scores.  The 2048 tokens took 413 us, 243 without the copies.)
#if LT_WIDTH % 64 == 0 && LAT_RANK % 64 == 0 && LT_WIDTH <= 576 && (LAT_RANK <= 256 || LAT_RANK == 512)
#define LP_BUILT 1
#include "tcgen05.cuh"

#define LP_VC (LAT_RANK <= 256 ? LAT_RANK : 256)         // value columns of a CTA
#define LP_HALVES (LAT_RANK / LP_VC)
#define LP_ATOMS (LT_WIDTH / 64)                          // 64-column swizzle atoms of a row
#define LP_Q_ATOM (128 * 128)                             // bytes of an atom of the 128 query rows
#define LP_K_ATOM (LT_KEYS * 128)
#define LP_STAGE_BYTES (LP_ATOMS * LP_K_ATOM)
// Queries in tensor memory, beside 256 columns of accumulators and two score buffers: the first six atoms (192 columns); the
// other atoms' rows are in shared memory.
#define LP_TQ (LP_ATOMS < 6 ? LP_ATOMS : 6)
#define LP_SQ (LP_ATOMS - LP_TQ)
#define LP_STAGES 4
#define LP_TOKENS 8
#define LP_THREADS 320
// They come by TMA too: into the stages of the second to fourth tile, which are filled when the queries have left, where that
// is room enough (rows of 512 and more elements), else into memory of their own.  (Read row by row from global memory, 16 of
// every 1152 bytes a lane, they took 2 us more: 20 prompts of 20 tokens, 16 heads, 14.5 us.)
#define LP_TQ_BYTES (LP_TQ * LP_Q_ATOM)
#define LP_TQ_LENT (LP_TQ_BYTES <= 3 * LP_STAGE_BYTES)
#define LP_TILES (LP_SQ * LP_Q_ATOM + LP_STAGES * LP_STAGE_BYTES + (LP_TQ_LENT ? 0 : LP_TQ_BYTES))
#define LP_SMEM (LP_TILES + 256 + 3 * 128 * 4 + 1024)
// Asked for: more than half of an SM's.  A second CTA would only wait there for tensor memory, while another SM may have none
// (2048 tokens, 16 heads, a latent of 128: 151 us with two on an SM, 106 with one).
#define LP_SMEM_ASKED (LP_SMEM > 116 * 1024 ? LP_SMEM : 116 * 1024)
enum { LP_ERR_WAIT = 141 };
static_assert(LP_SMEM <= 232448, "more shared memory than a CTA can have");
static_assert(LT_SMEM <= LP_SQ * LP_Q_ATOM + LP_STAGES * LP_STAGE_BYTES, "tokens done again find room in the tiles' place");

__device__ __forceinline__ void lp_arrive(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ bool lp_warp_wait(uint64_t* bar, uint32_t parity, volatile int* abort_flag) {
    uint32_t ok = 1;
    if ((threadIdx.x & 31) == 0) ok = mbar_wait(bar, parity, abort_flag) ? 1u : 0u;
    return __shfl_sync(0xffffffffu, ok, 0) != 0;
}
__device__ __forceinline__ void lp_warp_arrive(uint64_t* bar) {
    __syncwarp();
    if ((threadIdx.x & 31) == 0) lp_arrive(bar);
}
__device__ __forceinline__ void lp_tma_3d(void* dst, const CUtensorMap* map, uint64_t* bar, int x, int y, int z) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes"
        " [%0], [%1, {%3, %4, %5}], [%2];" ::"r"(smem_u32(dst)),
        "l"((uint64_t)map), "r"(smem_u32(bar)), "r"(x), "r"(y), "r"(z)
        : "memory");
}
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t* r) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
        "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};" ::"r"(taddr),
        "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
        "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
        : "memory");
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
// D[tmem] (+)= A[tmem] * B[smem]
__device__ __forceinline__ void umma_bf16_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}" ::"r"(tmem_d),
        "r"(tmem_a), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}
// the staged rows as the second product's B operand, the contiguous axis being its N: 64-column blocks of N an atom apart
__device__ __forceinline__ uint64_t lp_desc_values(uint32_t saddr) {
    return (uint64_t)((saddr & 0x3FFFFu) >> 4) | ((uint64_t)(LP_K_ATOM >> 4) << 16) | ((uint64_t)(1024 >> 4) << 32) |
           ((uint64_t)1 << 46) | ((uint64_t)2 << 61);
}

// The tokens of a CTA one by one (a function of its own, so that the kernel's warps keep their registers).
template <typename TO>
__device__ __noinline__ void lp_again(unsigned char* smem, const bf16* q, long q_ld, TO* out, long out_ld, const bf16* cache,
                                      int page_size, const int* bt, int pos, int tokens, int heads, int head0, int window,
                                      float scale, const float* sink) {
    for (int k = 0; k < tokens; ++k)
        latent_token<TO, false>(smem, q + k * q_ld, out + k * out_ld, cache, page_size, bt, pos + k, heads, head0, window, scale, 0,
                                0, 1, nullptr, sink);
}

template <typename TO>
__global__ void __launch_bounds__(LP_THREADS, 1) latent_prompt_kernel(
    const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k, const bf16* __restrict__ q, long q_ld,
    TO* __restrict__ out, long out_ld, const bf16* __restrict__ cache, int heads, int page_size, int cache_rows,
    const int* __restrict__ block_table, int bt_stride, const int* __restrict__ req_start, const int* __restrict__ req_ctx,
    const int* __restrict__ req_qlen, int n_requests, int window, float scale, const float* __restrict__ sink,
    int* __restrict__ status) {
    extern __shared__ unsigned char lp_raw[];
    unsigned char* q_s = (unsigned char*)(((uintptr_t)lp_raw + 1023) & ~(uintptr_t)1023);
    unsigned char* k_s = q_s + LP_SQ * LP_Q_ATOM;
    unsigned char* t_s = k_s + (LP_TQ_LENT ? LP_STAGE_BYTES : LP_STAGES * LP_STAGE_BYTES);     // queries on their way to tensor memory
    uint64_t* bars = (uint64_t*)(q_s + LP_TILES);
    uint64_t* q_full = bars;
    uint64_t* k_full = bars + 1;                          // [LP_STAGES]
    uint64_t* k_empty = k_full + LP_STAGES;
    uint64_t* s_full = k_empty + LP_STAGES;               // [2]
    uint64_t* c_full = s_full + 2;                        // [2] the rows' rescaling factors are there
    uint64_t* p_full = c_full + 2;                        // [2] weights written and accumulators rescaled
    uint64_t* o_done = p_full + 2;                        // [2] values of tile i are added up: barrier i & 1, phase i >> 1
    uint64_t* t_full = o_done + 2;                        // the queries in tensor memory are there
    uint64_t* t_sent = t_full + 1;                        // and in shared memory before that
    uint32_t* tmem_slot = (uint32_t*)(t_sent + 1);
    volatile int* abort_flag = (volatile int*)(tmem_slot + 1);
    volatile int* never = abort_flag + 1;                 // stays 0: for waits that must not be cut short
    volatile int* again = never + 1;                      // the tokens are done again
    float* corr_s = reinterpret_cast<float*>((unsigned char*)bars + 256);                // [2][128]
    float* inv_s = corr_s + 2 * 128;                                                     // [128]

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    int req = -1, tile = 0;                               // a request's last (longest) tile first
    for (int r = 0, acc = 0; r < n_requests; ++r) {
        const int nt = (req_qlen[r] + LP_TOKENS - 1) / LP_TOKENS;
        if ((int)blockIdx.x < acc + nt) {
            req = r;
            tile = nt - 1 - ((int)blockIdx.x - acc);
            break;
        }
        acc += nt;
    }
    if (req < 0) return;
    const int head0 = (int)(blockIdx.y / LP_HALVES) * 16, half = (int)(blockIdx.y % LP_HALVES);
    const int ctx = req_ctx[req], tok0 = req_start[req] + tile * LP_TOKENS;
    const int tokens = min(LP_TOKENS, req_qlen[req] - tile * LP_TOKENS);
    const int pos_first = ctx + tile * LP_TOKENS, pos_last = pos_first + tokens - 1;
    const int lo_first = window > 0 ? max(0, pos_first - window + 1) : 0;
    const int t_begin = lo_first / LT_KEYS, n_tiles = pos_last / LT_KEYS + 1 - t_begin;

    if (threadIdx.x == 0) {
        mbar_init(q_full, 1);
        mbar_init(t_full, 8);
        mbar_init(t_sent, 1);
        for (int s = 0; s < LP_STAGES; ++s) {
            mbar_init(&k_full[s], 1);
            mbar_init(&k_empty[s], 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(&s_full[b], 1);
            mbar_init(&c_full[b], 4);
            mbar_init(&p_full[b], 8);
            mbar_init(&o_done[b], 1);
        }
        *abort_flag = (*(volatile int*)status != 0) ? 1 : 0;
        *never = 0;
        *again = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (warp == 9) {
        tmem_alloc(tmem_slot, 512u);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_o = *tmem_slot, tmem_s = tmem_o + 256;          // two score buffers of 32 columns
    const uint32_t tmem_q = tmem_s + 2 * LT_KEYS;                       // 32 columns an atom
    auto give_up = [&]() {
        if (!*abort_flag) { *abort_flag = 1; atomicCAS(status, 0, LP_ERR_WAIT); }
    };
    if (warp < 8) {
        // a row's queries for tensor memory, pairs of elements a column, every other atom by warps 4-7
        if (lp_warp_wait(t_sent, 0, abort_flag)) {
            const int r = threadIdx.x & 127;
            const uint32_t dst = tmem_q + ((uint32_t)((warp & 3) * 32) << 16);
#pragma unroll
            for (int i = 0; i < (LP_TQ + 1) / 2; ++i) {
                const int a = (warp >> 2) + 2 * i;
                if (a >= LP_TQ) continue;
                uint4 w[8];
#pragma unroll
                for (int j = 0; j < 8; ++j)               // (the pieces of a row lie in the swizzle's order)
                    w[j] = *reinterpret_cast<const uint4*>(t_s + a * LP_Q_ATOM + r * 128 + ((j ^ (r & 7)) << 4));
                tmem_st16(dst + (uint32_t)(a * 32), reinterpret_cast<const uint32_t*>(w));
                tmem_st16(dst + (uint32_t)(a * 32 + 16), reinterpret_cast<const uint32_t*>(w + 4));
            }
            tmem_st_wait();
            tc_fence_before();
            lp_warp_arrive(t_full);
        } else if (lane == 0) {
            give_up();
        }
    }

    if (warp == 8) {
        // ---- producer: a lane issues one box, the part of a page that lies in the tile x 64 columns
        const int* bt = block_table + (long)req * bt_stride;
        const int box = min(page_size, LT_KEYS), boxes = LT_KEYS / box;
        const bool sent = __shfl_sync(0xffffffffu, *abort_flag, 0) == 0;
        if (lane == 0 && sent) {
            mbar_expect_tx(t_sent, LP_TQ_BYTES);
            for (int a = 0; a < LP_TQ; ++a) lp_tma_3d(t_s + a * LP_Q_ATOM, &map_q, t_sent, a * 64, head0, tok0);
            mbar_expect_tx(q_full, LP_SQ * LP_Q_ATOM);
            for (int a = 0; a < LP_SQ; ++a) lp_tma_3d(q_s + a * LP_Q_ATOM, &map_q, q_full, (LP_TQ + a) * 64, head0, tok0);
        }
        __syncwarp();
        int i = 0;
        for (; i < n_tiles && !*abort_flag; ++i) {
            const int s = i % LP_STAGES;
            const bool lent = LP_TQ_LENT && i == 1;       // (the queries must have left this stage and the next two)
            if ((lent && !lp_warp_wait(t_full, 0, abort_flag)) || !lp_warp_wait(&k_empty[s], ((uint32_t)(i / LP_STAGES) & 1u) ^ 1u, abort_flag)) {
                if (lane == 0) give_up();
                break;
            }
            if (lane == 0) mbar_expect_tx(&k_full[s], LP_STAGE_BYTES);
            __syncwarp();
            for (int op = lane; op < boxes * LP_ATOMS; op += 32) {
                const int b = op / LP_ATOMS, a = op - b * LP_ATOMS;
                const int key = (t_begin + i) * LT_KEYS + b * box;
                int row = cache_rows;
                if (key <= pos_last && key + box > lo_first) row = bt[key / page_size] * page_size + key % page_size;
                tma_load_2d(k_s + s * LP_STAGE_BYTES + a * LP_K_ATOM + b * box * 128, &map_k, &k_full[s], a * 64, row);
            }
        }
        if (*abort_flag) {                                // copies on their way land before the memory goes to another CTA
            for (int k = max(0, i - LP_STAGES); k < i; ++k) lp_warp_wait(&k_full[k % LP_STAGES], (uint32_t)(k / LP_STAGES) & 1u, never);
            if (sent) lp_warp_wait(q_full, 0, never);
            if (sent) lp_warp_wait(t_sent, 0, never);
        }
    } else if (warp == 9) {
        // ---- MMA issuer
        constexpr uint32_t idesc_s = instr_desc_bf16(128, LT_KEYS);
        constexpr uint32_t idesc_o = instr_desc_bf16(128, LP_VC) | (1u << 16);          // B: the contiguous axis is N
        bool ok = !*abort_flag;
        auto scores = [&](int i) -> bool {
            const int s = i % LP_STAGES, b = i & 1;
            if (!lp_warp_wait(&k_full[s], (uint32_t)(i / LP_STAGES) & 1u, abort_flag)) return false;
            __syncwarp();
            const int here = pos_last + 1 - (t_begin + i) * LT_KEYS;                     // rows that are keys of the request
            if (here < LT_KEYS) {                         // the last tile: rows never written may hold anything, also NaN
                for (int p = here * 8 + lane; p < LT_KEYS * 8; p += 32)
                    for (int a = 0; a < LP_ATOMS; ++a)
                        *reinterpret_cast<uint4*>(k_s + s * LP_STAGE_BYTES + a * LP_K_ATOM + p * 16) = make_uint4(0, 0, 0, 0);
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                __syncwarp();
            }
            tc_fence_after();
            if (lane == 0) {
                // (a descriptor's address counts 16 bytes)
                const uint64_t qd = smem_desc_sw128(smem_u32(q_s)), kd = smem_desc_sw128(smem_u32(k_s + s * LP_STAGE_BYTES));
                const uint32_t d = tmem_s + (uint32_t)(b * LT_KEYS);
#pragma unroll
                for (int k = 0; k < LP_TQ * 4; ++k)
                    umma_bf16_ts(d, tmem_q + (uint32_t)(k * 8), kd + (uint64_t)(((k >> 2) * LP_K_ATOM + (k & 3) * 32) >> 4), idesc_s, k > 0 ? 1u : 0u);
#pragma unroll
                for (int k = LP_TQ * 4; k < LP_ATOMS * 4; ++k)
                    umma_bf16(d, qd + (uint64_t)((((k >> 2) - LP_TQ) * LP_Q_ATOM + (k & 3) * 32) >> 4),
                              kd + (uint64_t)(((k >> 2) * LP_K_ATOM + (k & 3) * 32) >> 4), idesc_s, 1u);
                umma_commit(&s_full[b]);
            }
            __syncwarp();
            return true;
        };
        if (ok) ok = lp_warp_wait(t_full, 0, abort_flag) && lp_warp_wait(q_full, 0, abort_flag);
        if (ok) ok = scores(0);
        for (int i = 0; i < n_tiles && ok; ++i) {
            // the scores of tile i + 1 go where those of tile i - 1 and then its weights were: the values of tile i - 1 were
            // issued before, and the tensor cores work in order
            if (i + 1 < n_tiles && !scores(i + 1)) { ok = false; break; }
            const int b = i & 1, s = i % LP_STAGES;
            if (!lp_warp_wait(&p_full[b], (uint32_t)(i >> 1) & 1u, abort_flag)) { ok = false; break; }
            tc_fence_after();
            if (lane == 0) {
                const uint32_t va = smem_u32(k_s + s * LP_STAGE_BYTES + half * (LP_VC / 64) * LP_K_ATOM);
#pragma unroll
                for (int k = 0; k < LT_KEYS / 16; ++k)
                    umma_bf16_ts(tmem_o, tmem_s + (uint32_t)(b * LT_KEYS + k * 8), lp_desc_values(va + (uint32_t)(k * 16 * 128)), idesc_o,
                                 (i > 0 || k > 0) ? 1u : 0u);
                umma_commit(&k_empty[s]);
                umma_commit(&o_done[b]);                  // the accumulators hold the tiles up to i
            }
            __syncwarp();
        }
        if (!ok && lane == 0) give_up();
    } else if (warp < 4) {
        // ---- weights of row r: token r / 16, head head0 + r % 16
        const int r = threadIdx.x, token = r >> 4;
        const uint32_t lanes = (uint32_t)(warp * 32) << 16;
        const int pos = token < tokens ? pos_first + token : -1;
        const int lo = window > 0 ? max(0, pos - window + 1) : 0;
        const int lo_last = window > 0 ? max(0, pos_last - window + 1) : 0;
        float m = -CUDART_INF_F, l = 0.0f;
        if (sink != nullptr) {
            m = sink[head0 + (r & 15)];
            l = 1.0f;
        }
        bool ok = !*abort_flag;
        for (int i = 0; i < n_tiles; ++i) {
            const int b = i & 1;
            if (!lp_warp_wait(&s_full[b], (uint32_t)(i >> 1) & 1u, abort_flag)) {
                if (lane == 0) give_up();
                ok = false;
                break;
            }
            tc_fence_after();
            uint32_t v[32];
            tmem_ld16(tmem_s + (uint32_t)(b * LT_KEYS) + lanes, v);
            tmem_ld16(tmem_s + (uint32_t)(b * LT_KEYS) + 16u + lanes, v + 16);
            tmem_ld_wait();
            const int key0 = (t_begin + i) * LT_KEYS;
            if (key0 + LT_KEYS - 1 > pos_first || key0 < lo_last) {       // some token does not see all of the tile
                bool odd = false;
#pragma unroll
                for (int j = 0; j < 32; ++j)
                    odd |= (key0 + j < lo || key0 + j > pos) && !(fabsf(__uint_as_float(v[j])) < CUDART_INF_F);
                if (odd && token < tokens) *again = 1;
            }
            float p[32], mx[4];
#pragma unroll
            for (int j = 0; j < 32; ++j) {
                p[j] = key0 + j >= lo && key0 + j <= pos ? __fmul_rn(__uint_as_float(v[j]), scale) : -CUDART_INF_F;
                mx[j & 3] = j < 4 ? p[j] : fmaxf(mx[j & 3], p[j]);
            }
            const float m_new = fmaxf(m, fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3])));
            const bool out_of_sight = pos < key0 || lo >= key0 + LT_KEYS;
            const float corr = out_of_sight ? 1.0f : expf(m - m_new);     // 0 at a row's first tile without a sink
            corr_s[b * 128 + r] = m == -CUDART_INF_F ? 1.0f : corr;       // (nothing has been added up yet)
            lp_warp_arrive(&c_full[b]);
            uint32_t w[16];
            if (out_of_sight) {
#pragma unroll
                for (int j = 0; j < 16; ++j) w[j] = 0u;
            } else {
                float sum = 0.0f;
#pragma unroll
                for (int g = 0; g < 4; ++g) {
                    float e[8];
#pragma unroll
                    for (int j = 0; j < 8; ++j) e[j] = expf(__fsub_rn(p[g * 8 + j], m_new));
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        const __nv_bfloat162 pair = __floats2bfloat162_rn(e[2 * j], e[2 * j + 1]);
                        w[g * 4 + j] = *reinterpret_cast<const uint32_t*>(&pair);
                    }
                    sum += ((e[0] + e[1]) + (e[2] + e[3])) + ((e[4] + e[5]) + (e[6] + e[7]));
                }
                m = m_new;
                l = l * corr + sum;
            }
            tmem_st16(tmem_s + (uint32_t)(b * LT_KEYS) + lanes, w);
            tmem_st_wait();
            tc_fence_before();
            lp_warp_arrive(&p_full[b]);
        }
        inv_s[r] = ok ? 1.0f / l : 0.0f;
        lp_warp_arrive(&c_full[n_tiles & 1]);             // (one phase more than tiles: the sums are there)
    } else {
        // ---- accumulators of row r.  A wait on o_done tells a phase from the one before it only, so no barrier of the two
        // may get two phases ahead of these warps: they wait for the values of tile i - 2 before they let those of tile i
        // go (the scores of tile i came after them: this wait is over at once), and for tile i - 1 where they rescale.
        const int r = threadIdx.x - 128, token = r >> 4;
        const uint32_t o_addr = tmem_o + ((uint32_t)((warp - 4) * 32) << 16);
        bool ok = !*abort_flag;
        for (int i = 0; i < n_tiles && ok; ++i) {
            const int b = i & 1;
            ok = lp_warp_wait(&c_full[b], (uint32_t)(i >> 1) & 1u, abort_flag);
            if (!ok) break;
            if (i > 1) ok = lp_warp_wait(&o_done[i & 1], (uint32_t)((i - 2) >> 1) & 1u, abort_flag);
            if (!ok) break;
            const float corr = corr_s[b * 128 + r];
            if (i > 0 && __any_sync(0xffffffffu, corr != 1.0f)) {
                ok = lp_warp_wait(&o_done[(i - 1) & 1], (uint32_t)((i - 1) >> 1) & 1u, abort_flag);
                if (!ok) break;
                tc_fence_after();
#pragma unroll 2
                for (int c = 0; c < LP_VC; c += 32) {
                    uint32_t v[32];
                    tmem_ld16(o_addr + (uint32_t)c, v);
                    tmem_ld16(o_addr + (uint32_t)c + 16u, v + 16);
                    tmem_ld_wait();
#pragma unroll
                    for (int j = 0; j < 32; ++j) v[j] = __float_as_uint(__uint_as_float(v[j]) * corr);
                    tmem_st16(o_addr + (uint32_t)c, v);
                    tmem_st16(o_addr + (uint32_t)c + 16u, v + 16);
                }
                tmem_st_wait();
                tc_fence_before();
            }
            lp_warp_arrive(&p_full[b]);
        }
        if (ok) ok = lp_warp_wait(&c_full[n_tiles & 1], (uint32_t)(n_tiles >> 1) & 1u, abort_flag);
        if (ok) ok = lp_warp_wait(&o_done[(n_tiles - 1) & 1], (uint32_t)((n_tiles - 1) >> 1) & 1u, abort_flag);
        if (!ok && lane == 0) give_up();
        ok = __all_sync(0xffffffffu, ok) && !*abort_flag;
        ok = __all_sync(0xffffffffu, ok);
        tc_fence_after();
        if (ok && !*again) {
            const float inv = inv_s[r];
            TO* dst = out + (long)(tok0 + token) * out_ld + (long)(head0 + (r & 15)) * LAT_RANK + half * LP_VC;
#pragma unroll 1
            for (int c = 0; c < LP_VC; c += 32) {
                uint32_t v[32];
                tmem_ld16(o_addr + (uint32_t)c, v);       // all lanes of the warp take part
                tmem_ld16(o_addr + (uint32_t)c + 16u, v + 16);
                tmem_ld_wait();
                if (token >= tokens) continue;
                __align__(16) TO o[32];
#pragma unroll
                for (int j = 0; j < 32; ++j) o[j] = from_f32<TO>(__uint_as_float(v[j]) * inv);
#pragma unroll
                for (int j = 0; j < 32 * (int)sizeof(TO) / 16; ++j)
                    reinterpret_cast<uint4*>(dst + c)[j] = reinterpret_cast<const uint4*>(o)[j];
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 9) {
        tc_fence_after();
        tmem_dealloc(tmem_o, 512u);
    }
    if (*again && !*abort_flag && half == 0 && warp < LT_WARPS)           // (all columns: the halves agree, their scores are the same)
        lp_again<TO>(q_s, q + (long)tok0 * q_ld, q_ld, out + (long)tok0 * out_ld, out_ld, cache, page_size, block_table + (long)req * bt_stride,
                     pos_first, tokens, heads, head0, window, scale, sink);
}

// What the prompt kernel takes beyond what latent_attention_tc_kernel does: whole groups of 16 heads, 16-byte aligned rows
// of the output, and pages that tiles of 32 keys consist of or lie in, in whole groups of eight rows (the swizzle's unit).
FL_API int fl_latent_prompt_takes(int heads, int page_size) {
    return heads % 16 == 0 && (page_size % 32 == 0 || page_size == 8 || page_size == 16);
}

// As fl_latent_attention_tc without splits, for steps of prompts; cache: [cache_rows][rank + rot], cache_rows = pages x page_size.
FL_API int fl_latent_prompt(const void* q, long q_ld, void* out, int out_dtype, long out_ld, const void* cache, long cache_rows,
                            int page_size, const int* block_table, int bt_stride, const int* req_start, const int* req_ctx,
                            const int* req_qlen, int n_requests, int n_tokens, int heads, int window, float scale,
                            const float* sink, int* status, cudaStream_t stream) {
    if (n_tokens <= 0 || n_requests <= 0) return 0;
    if (!fl_latent_prompt_takes(heads, page_size) || cache_rows >= (1l << 31) || heads / 16 * LP_HALVES > 65535)
        return (int)cudaErrorInvalidValue;
    if (((uintptr_t)q % 16) || (q_ld % 8) || ((uintptr_t)cache % 16) || ((uintptr_t)out % 16) || out_ld % 8)
        return (int)cudaErrorMisalignedAddress;
    EncodeTiledFn encode = encode_tiled_fn();
    if (!encode) return (int)cudaErrorNotSupported;
    CUtensorMap map_q, map_k;
    {
        // the queries as [tokens][heads][width]: a box is 8 tokens x 16 heads x 64 columns, 128 rows in that order
        cuuint64_t dims[3] = {LT_WIDTH, (cuuint64_t)heads, (cuuint64_t)n_tokens};
        cuuint64_t strides[2] = {LT_WIDTH * 2, (cuuint64_t)q_ld * 2};
        cuuint32_t box[3] = {64, 16, LP_TOKENS}, elem[3] = {1, 1, 1};
        if (encode(&map_q, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(q), dims, strides, box, elem,
                   CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                   CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
            return (int)cudaErrorInvalidValue;
    }
    int rc = make_map(&map_k, cache, cache_rows, LT_WIDTH, LT_WIDTH, page_size < LT_KEYS ? page_size : LT_KEYS);
    if (rc) return rc;
    // plain stream order (no programmatic overlap): this kernel takes all of an SM's tensor memory
    const dim3 grid(n_tokens / LP_TOKENS + n_requests, heads / 16 * LP_HALVES);
    FL_DISPATCH(out_dtype, TO, {
        rc = (int)cudaFuncSetAttribute(latent_prompt_kernel<TO>, cudaFuncAttributeMaxDynamicSharedMemorySize, LP_SMEM_ASKED);
        if (rc) return rc;
        latent_prompt_kernel<TO><<<grid, LP_THREADS, LP_SMEM_ASKED, stream>>>(map_q, map_k, (const bf16*)q, q_ld, (TO*)out, out_ld,
                                                                        (const bf16*)cache, heads, page_size, (int)cache_rows,
                                                                        block_table, bt_stride, req_start, req_ctx, req_qlen,
                                                                        n_requests, window, scale, sink, status);
        return fl_launch_status();
    });
    return 0;
}
#else
FL_API int fl_latent_prompt_takes(int heads, int page_size) { (void)heads; (void)page_size; return 0; }
#endif
