// Paged causal attention for prompt portions on the Blackwell tensor cores:
// both products (Q K^T and P V) are tcgen05.mma with the accumulators in tensor
// memory; keys, values and queries arrive by TMA; the softmax runs in float on
// FT_PARTS threads per query row.
//
// A CTA takes 128 consecutive query rows of one request and one query head and
// walks the request's keys in blocks of 128 (starting at multiples of 128 of the
// absolute position, so a row's sequence of partial maxima does not depend on
// how the prompt was cut).  Per block:
//   producer warps  TMA: the block's pages of this head's keys (one warp) and values
//                   (another) into two-stage rings (one box of page_size x 64
//                   per page and 64 columns, each issued by a lane of its own;
//                   pages that do not exist are fetched from beyond the tensor,
//                   which fills zeros);
//   MMA warp        S = Q K^T into one of two S buffers in tensor memory (so the
//                   next block's scores are computed while this block's are
//                   being exponentiated), then O_blk = P V;
//   softmax warps   FT_PARTS threads share query row r: each reads its part of the row of S
//                   (tcgen05.ld), masks, exchanges the part's maximum with its
//                   partners, keeps the running maximum and sum in float, writes
//                   its part of P as bfloat16 into shared memory in the swizzled
//                   K-major layout the second MMA reads, and adds its columns
//                   of O_blk into its part of the output row, which it holds in
//                   registers (rescaled when the maximum moves).
// Every wait on an mbarrier is bounded; a give-up sets an error word and all
// roles leave.
//
// fastllm-py's counterpart is `_sdpa` (fastllm_py/model.py:341-353).  The
// mma.sync kernel in attention_prefill.cu computes the same thing and serves the
// head sizes and page sizes this one does not take (HEAD_DIM 64 or 128; page
// sizes that are multiples of 8 and divide 128).
#include <cuda.h>

#include "common.cuh"

#ifndef HEAD_DIM
#define HEAD_DIM 128
#endif
static_assert(HEAD_DIM == 64 || HEAD_DIM == 128, "the tcgen05 prefill kernel takes head sizes 64 and 128");

#define FT_BM 128                          // query rows per CTA
#define FT_BN 128                          // keys per block
#ifndef FT_STAGES
#define FT_STAGES 3                        // key and value ring depth (each)
#endif
#ifndef FT_PARTS
#define FT_PARTS 2                         // softmax threads per query row
#endif
#define FT_ATOMS (HEAD_DIM / 64)           // 64-column swizzle atoms per row
#define FT_ATOM_BYTES (128 * 128)          // 128 rows x 128 bytes
#define FT_WAIT_LIMIT_NS 2000000000ull

enum { FT_ERR_WAIT = 301, FT_ERR_SMEM = 302 };

// ------------------------------------------------------------------ PTX wraps
__device__ __forceinline__ uint32_t ft_smem(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void ft_bar_init(uint64_t* bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(ft_smem(bar)), "r"(count));
}
__device__ __forceinline__ void ft_bar_arrive(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(ft_smem(bar)) : "memory");
}
__device__ __forceinline__ void ft_bar_expect(uint64_t* bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(ft_smem(bar)), "r"(bytes)
                 : "memory");
}
__device__ __forceinline__ uint64_t ft_now() {
    uint64_t t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}
__device__ __forceinline__ bool ft_wait(uint64_t* bar, uint32_t parity, volatile int* abort_flag) {
    uint32_t ok = 0, spins = 0;
    uint64_t t0 = 0;
    while (true) {
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(ok)
            : "r"(ft_smem(bar)), "r"(parity)
            : "memory");
        if (ok) return true;
        if ((++spins & 127u) == 0) {
            if (*abort_flag) return false;
            if (t0 == 0) t0 = ft_now();
            else if (ft_now() - t0 > FT_WAIT_LIMIT_NS) return false;
        }
    }
}
// A warp waits through its first lane and arrives through it (after __syncwarp, which orders
// the other lanes' writes before the arrival): a barrier then sees 8 arrivals per phase from the
// softmax warps instead of 256, and one thread polls instead of 32.
__device__ __forceinline__ bool ft_warp_wait(uint64_t* bar, uint32_t parity, volatile int* abort_flag) {
    uint32_t ok = 1;
    if ((threadIdx.x & 31) == 0) ok = ft_wait(bar, parity, abort_flag) ? 1u : 0u;
    return __shfl_sync(0xffffffffu, ok, 0) != 0;
}
__device__ __forceinline__ void ft_warp_arrive(uint64_t* bar) {
    __syncwarp();
    if ((threadIdx.x & 31) == 0) ft_bar_arrive(bar);
}
__device__ __forceinline__ void ft_tma_2d(void* dst, const CUtensorMap* map, uint64_t* bar, int x, int y) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes"
        " [%0], [%1, {%3, %4}], [%2];" ::"r"(ft_smem(dst)),
        "l"((uint64_t)map), "r"(ft_smem(bar)), "r"(x), "r"(y)
        : "memory");
}
__device__ __forceinline__ void ft_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void ft_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void ft_mma(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                       uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem_d),
        "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}
__device__ __forceinline__ void ft_commit(uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(ft_smem(bar))
                 : "memory");
}
__device__ __forceinline__ void ft_ld32(uint32_t taddr, uint32_t* r) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, %17, %18, %19, %20, %21, "
        "%22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
          "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]),
          "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]),
          "=r"(r[30]), "=r"(r[31])
        : "r"(taddr)
        : "memory");
}
__device__ __forceinline__ void ft_ld4(uint32_t taddr, uint32_t* r) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(taddr) : "memory");
}
__device__ __forceinline__ void ft_ld2(uint32_t taddr, uint32_t* r) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x2.b32 {%0, %1}, [%2];" : "=r"(r[0]), "=r"(r[1]) : "r"(taddr) : "memory");
}
__device__ __forceinline__ void ft_st1(uint32_t taddr, uint32_t a) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x1.b32 [%0], {%1};" ::"r"(taddr), "r"(a) : "memory");
}
__device__ __forceinline__ void ft_st2(uint32_t taddr, uint32_t a, uint32_t b) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x2.b32 [%0], {%1, %2};" ::"r"(taddr), "r"(a), "r"(b) : "memory");
}
__device__ __forceinline__ void ft_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void ft_st32(uint32_t taddr, const uint32_t* r) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
        "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, %17, %18, %19, %20, %21, %22, "
        "%23, %24, %25, %26, %27, %28, %29, %30, %31, %32};" ::"r"(taddr),
        "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]),
        "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]),
        "r"(r[18]), "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]),
        "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31])
        : "memory");
}
__device__ __forceinline__ void ft_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
// D[tmem] (+)= A[tmem] * B[smem]: the A operand (128 rows in the lanes, 16 bfloat16 of K as 8 columns) comes
// from tensor memory
__device__ __forceinline__ void ft_mma_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t bdesc, uint32_t idesc,
                                          uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}" ::"r"(tmem_d),
        "r"(tmem_a), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}

// K-major operand, rows of 128 bytes in the 128-byte swizzle, 8-row groups 1024 bytes apart.
__device__ __forceinline__ uint64_t ft_desc_kmajor(uint32_t saddr) {
    return (uint64_t)((saddr & 0x3FFFFu) >> 4) | ((uint64_t)1 << 16) | ((uint64_t)(1024 >> 4) << 32) |
           ((uint64_t)1 << 46) | ((uint64_t)2 << 61);
}
// MN-major operand (the contiguous axis is N): 64-element blocks of N are `atom` bytes apart
// (leading offset), groups of 8 K rows 1024 bytes apart (stride offset).
__device__ __forceinline__ uint64_t ft_desc_mnmajor(uint32_t saddr, uint32_t atom) {
    return (uint64_t)((saddr & 0x3FFFFu) >> 4) | ((uint64_t)(atom >> 4) << 16) |
           ((uint64_t)(1024 >> 4) << 32) | ((uint64_t)1 << 46) | ((uint64_t)2 << 61);
}
// float accumulator, bfloat16 operands; b_mn: B is MN-major
__host__ __device__ constexpr uint32_t ft_idesc(int m, int n, int b_mn) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)b_mn << 16) | ((uint32_t)(n >> 3) << 17) |
           ((uint32_t)(m >> 4) << 24);
}
// 2^x by the special-function unit (relative error about 2^-22; -inf gives 0)
__device__ __forceinline__ float ft_ex2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float ft_weight(float a, float b) { return (a == -CUDART_INF_F) ? 0.0f : exp2f(a - b); }

// ROWS (see the kernel): blocks of 64 keys, and stages for as much of the SM's shared memory as leaves room for one CTA.
template <bool ROWS> struct FtSmem {
    static constexpr int BN = ROWS ? 64 : FT_BN;                       // keys of a block
    static constexpr int PARTS = ROWS && HEAD_DIM == 128 ? 4 : FT_PARTS;   // softmax threads per query row
    static constexpr int SOFTMAX_WARPS = 4 * PARTS, THREADS = (SOFTMAX_WARPS + 3) * 32;
    static constexpr int STAGES = ROWS ? (HEAD_DIM == 128 ? 5 : 6) : FT_STAGES;
    static constexpr int ATOM = BN * 128;                              // bytes of 64 columns of a block
    static constexpr int Q_BYTES = FT_ATOMS * FT_ATOM_BYTES;
    static constexpr int KV_BYTES = FT_ATOMS * ATOM;                   // one of K or V, one stage
    static constexpr int TILES = Q_BYTES + 2 * STAGES * KV_BYTES;
    static constexpr int BAR_SLOTS = 24 + 4 * STAGES;                  // 8-byte slots: barriers and the like
    static constexpr int BARS = BAR_SLOTS * 8 + (ROWS ? 4 : 2) * PARTS * 128 * 4;   // ... then the parts' maxima (two rounds; ROWS: and sums)
    // The tiles want a 1024-byte boundary.  Where they fill the SM's shared memory to within a KB
    // there is no room to round up to one: the kernel then counts on the dynamic shared memory
    // starting on such a boundary (it has no static shared memory) and reports FT_ERR_SMEM instead
    // of running if it does not.
    static constexpr int SLACK = (TILES + BARS + 1024 <= 232448) ? 1024 : 0;
    static constexpr int TOTAL = TILES + BARS + SLACK;
};

// ROWS: a cache row holds a token's key and its value (k | v, pages [n_kv_heads][page_size][2 HEAD_DIM]); `sink` ([heads], or
// null) is a term exp(sink) of each head's denominator, and `gate` (or null) multiplies a row's result by the sigmoid of its
// gate, `gate_cols` numbers a head (one, or one a channel), before it is rounded.  Such layers are served by two kernels, by
// the lengths of a step, so this one makes the sums of the other (sink_attention_tc.cu), one by one: blocks of 64 keys at
// multiples of 64 of the absolute position, a rescaling at every block where a row's maximum moved, scores scaled and weights
// made by the same instructions, four partial sums of a row's weights (keys 2c and 2c + 1 of every eight), values in K steps
// of 16 from the first to the last.  The results are the same bit for bit, and a row is written before the values of blocks that
// it does not see are added.  Bound by what a block of 64 keys takes the softmax warps one after the other: scores, maximum,
// weights, then the accumulators, which at nearly every block some row of a warp rescales: 1.9 us (2.1 with two threads a row
// instead of four; 2048 tokens x 16 heads of 128 75 us, on mma.sync 217; 38 with a maximum that is renewed only after it has
// grown by 2^8, which rounds otherwise).
template <bool ROWS>
__global__ void __launch_bounds__(FtSmem<ROWS>::THREADS, 1) attention_prefill_tc_kernel(
    const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_kv,
    bf16* __restrict__ out, long out_ld, int page_size, int kv_rows_total, const int* __restrict__ block_table,
    int bt_stride, const int* __restrict__ req_start, const int* __restrict__ req_ctx,
    const int* __restrict__ req_qlen, int n_requests, int include_single, int n_heads, int n_kv_heads,
    int window, float scale, int* __restrict__ status, const float* __restrict__ sink, const bf16* __restrict__ gate,
    long gate_ld, int gate_cols) {
    using L = FtSmem<ROWS>;
    constexpr int BN = L::BN, STAGES = L::STAGES, PARTS = L::PARTS;
    constexpr int KP = BN / PARTS, OD = HEAD_DIM / PARTS;              // a softmax thread's keys of a block, and output columns
    static_assert(OD % 32 == 0 && (ROWS || KP % 32 == 0), "multiples of 32 columns; of 32 keys, where these are neighbours");
    constexpr int PRODUCER_WARP = L::SOFTMAX_WARPS;                    // queries and keys
    constexpr int MMA_WARP = PRODUCER_WARP + 1, VPRODUCER_WARP = PRODUCER_WARP + 2;   // (VPRODUCER: values)
    const float scale_log2e = scale * 1.4426950408889634f;
    extern __shared__ __align__(1024) unsigned char ft_raw[];
    unsigned char* base = (unsigned char*)(((uintptr_t)ft_raw + 1023) & ~(uintptr_t)1023);
    if (base + L::TILES + L::BARS > ft_raw + L::TOTAL) {       // uniform over the CTA
        if (threadIdx.x == 0) atomicCAS(status, 0, FT_ERR_SMEM);
        return;
    }
    unsigned char* q_s = base;
    unsigned char* k_s = q_s + L::Q_BYTES;                        // [stage][atom][128 rows][128 B]
    unsigned char* v_s = k_s + STAGES * L::KV_BYTES;
    uint64_t* bars = (uint64_t*)(base + L::TILES);
    uint64_t* q_full = bars + 0;
    uint64_t* k_full = bars + 24;                                      // [STAGES]
    uint64_t* k_empty = k_full + STAGES;
    uint64_t* s_full = bars + 5;                                       // [2]
    uint64_t* p_full = bars + 9;                                       // [2]
    uint64_t* o_done = bars + 11;                                      // [2] P V of block i is done: barrier i & 1, phase i >> 1
    uint32_t* tmem_slot = (uint32_t*)(bars + 13);
    uint64_t* x_bar = bars + 14;                                       // the softmax threads' exchange point
    uint64_t* z_full = bars + 16;                                      // the last block's values are cleared behind the last key
    uint64_t* v_full = k_empty + STAGES;
    uint64_t* v_empty = v_full + STAGES;
    volatile int* abort_flag = (volatile int*)(tmem_slot + 1);
    volatile int* never = (volatile int*)(bars + 15);                  // stays 0: for waits that must not be cut short

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const bool producer = warp == PRODUCER_WARP || warp == VPRODUCER_WARP;
    if (producer && lane == 0) {
        // the copies' descriptors are wanted first thing: ask for them while the tile is being worked out
        if (warp == PRODUCER_WARP) asm volatile("prefetch.tensormap [%0];" ::"l"((uint64_t)&map_q) : "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"((uint64_t)&map_kv) : "memory");
    }
    // which request and which 128-row tile: blockIdx.y counts tiles, a request's last (longest) tile first
    int req = -1, tile = 0;
    {
        int acc = 0;
        for (int r = 0; r < n_requests; ++r) {
            const int ql = req_qlen[r];
            const int nt = (ql > 1 || include_single) ? (ql + FT_BM - 1) / FT_BM : 0;
            if ((int)blockIdx.y < acc + nt) { req = r; tile = nt - 1 - ((int)blockIdx.y - acc); break; }
            acc += nt;
        }
    }
    if (req < 0) return;
    const int h = blockIdx.x;
    const int kvh = h / (n_heads / n_kv_heads);
    const int q_len = req_qlen[req], ctx = req_ctx[req], row0 = tile * FT_BM;
    const int tok0 = req_start[req] + row0;
    const int rows_here = min(FT_BM, q_len - row0);
    const int pos_first = ctx + row0, pos_last = ctx + row0 + rows_here - 1;
    const int lo_tile = window > 0 ? max(0, pos_first - window + 1) : 0;
    const int kb_begin = lo_tile / BN, kb_end = pos_last / BN + 1;
    const int n_blocks = kb_end - kb_begin;
    // ROWS: what the last page holds behind the tile's last key may be anything, and a weight of zero does not make a value that is
    // not finite vanish: the values' producer warp clears rows clear_from .. clear_to - 1 of the last block
    const int page_box = min(page_size, BN), clear_from = pos_last + 1 - (kb_end - 1) * BN;
    const int clear_to = (clear_from + page_box - 1) / page_box * page_box;
    const bool clears = ROWS && clear_from < clear_to;

    // ---- the producers' side of a block: one box of a page and 64 columns per lane.  A block of 128 keys is
    // pages x atoms boxes of a few KB; one lane issues one box (looking up its page itself), so a block's
    // copies leave together.
    const int is_v = warp == VPRODUCER_WARP ? 1 : 0;
    uint64_t* full = is_v ? v_full : k_full;
    uint64_t* empty = is_v ? v_empty : k_empty;
    auto issue_block = [&](int i) {
        unsigned char* ring = is_v ? v_s : k_s;
        const int* bt = block_table + (long)req * bt_stride;
        const int n_ops = (BN / page_box) * FT_ATOMS;
        const int s = i % STAGES;
        if (lane == 0) ft_bar_expect(&full[s], L::KV_BYTES);
        __syncwarp();
        const int key0 = (kb_begin + i) * BN;
        for (int op = lane; op < n_ops; op += 32) {
            const int p = op / FT_ATOMS, a = op % FT_ATOMS;
            const int first_key = key0 + p * page_box;
            const int last_key = first_key + page_box - 1;
            // a page (or the part of one that lies in the block) wholly outside what this tile may see is fetched from beyond the tensor: zeros
            int row = kv_rows_total;
            if (first_key <= pos_last && last_key >= lo_tile) {
                const long pg = bt[first_key / page_size];
                row = (int)((ROWS ? pg * n_kv_heads + kvh : (pg * 2 + is_v) * n_kv_heads + kvh) * page_size) + (ROWS ? first_key % page_size : 0);
            }
            const int off = s * L::KV_BYTES + a * L::ATOM + p * page_box * 128;
            ft_tma_2d(ring + off, &map_kv, &full[s], a * 64 + (ROWS ? is_v * HEAD_DIM : 0), row);
        }
    };
    // The producer warps set up their own barriers and send for the queries and the first block (the rings are
    // empty: nothing to wait for) before the CTA meets for the rest of its set-up, which the copies' way through
    // memory then hides: tensor memory, the other barriers, a look at the error word.  A tile with many blocks
    // sends for a whole ring at once; for a short one that only put the queries, which are wanted first, behind
    // three blocks of keys and values (measured: 2048 tokens 76 us against 70, 8192 tokens 693 against 744).
    const int early = n_blocks * BN > 32 * FT_BN ? STAGES : FT_BN / BN;
    int issued = 0;
    if (producer) {
        if (lane == 0) {
            if (!is_v) ft_bar_init(q_full, 1);
            for (int s = 0; s < STAGES; ++s) {
                ft_bar_init(&full[s], 1);
                ft_bar_init(&empty[s], 1);
            }
            asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            if (!is_v) {
                ft_bar_expect(q_full, L::Q_BYTES);
                for (int a = 0; a < FT_ATOMS; ++a)
                    ft_tma_2d(q_s + a * FT_ATOM_BYTES, &map_q, q_full, h * HEAD_DIM + a * 64, tok0);
            }
        }
        __syncwarp();
        for (; issued < n_blocks && issued < early; ++issued) issue_block(issued);
    }
    if (threadIdx.x == 0) {
        for (int s = 0; s < 2; ++s) {
            ft_bar_init(&s_full[s], 1);
            ft_bar_init(&p_full[s], L::SOFTMAX_WARPS);
            ft_bar_init(&o_done[s], 1);
        }
        ft_bar_init(x_bar, L::SOFTMAX_WARPS);
        ft_bar_init(z_full, 1);
        *abort_flag = (*(volatile int*)status != 0) ? 1 : 0;
        *never = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (warp == MMA_WARP) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(ft_smem(tmem_slot)),
                     "r"(512u)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    ft_fence_before();
    __syncthreads();
    ft_fence_after();
    const uint32_t tmem = *tmem_slot;
    const uint32_t tmem_s = tmem;                                      // two S buffers: columns 0 and BN
    const uint32_t tmem_o = tmem + 256;                                // O: HEAD_DIM columns, accumulated over the blocks

#define FT_GIVE_UP()                                                             \
    {                                                                            \
        if (!*abort_flag) { *abort_flag = 1; atomicCAS(status, 0, FT_ERR_WAIT); } \
        break;                                                                   \
    }

    if (producer) {
        // ---- producers: one warp for the queries and the keys, one for the values, each with a ring of its
        // own.  A key stage is free again as soon as S of its block is computed, which is a whole block
        // earlier than P V; with keys and values in one ring the next keys could only be asked for after
        // P V, and their way through TMA showed.
        int i = issued;
        for (; i < n_blocks && !*abort_flag; ++i) {
            if (!ft_warp_wait(&empty[i % STAGES], ((uint32_t)(i / STAGES) & 1u) ^ 1u, abort_flag)) FT_GIVE_UP();
            issue_block(i);
        }
        if (clears && is_v && i == n_blocks) {
            const int s = (n_blocks - 1) % STAGES;
            if (ft_warp_wait(&full[s], (uint32_t)((n_blocks - 1) / STAGES) & 1u, abort_flag)) {
                for (int a = 0; a < FT_ATOMS; ++a)
                    for (int o = clear_from * 128 + lane * 16; o < clear_to * 128; o += 512)
                        *reinterpret_cast<uint4*>(v_s + s * L::KV_BYTES + a * L::ATOM + o) = make_uint4(0u, 0u, 0u, 0u);
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                ft_warp_arrive(z_full);
            } else if (!*abort_flag) {
                *abort_flag = 1;
                atomicCAS(status, 0, FT_ERR_WAIT);
            }
        }
        if (*abort_flag) {
            // leaving early: the copies still on their way must land before the shared memory goes to
            // another CTA (the wait is bounded like every other)
            for (int k = max(0, i - STAGES); k < i; ++k)
                ft_warp_wait(&full[k % STAGES], (uint32_t)(k / STAGES) & 1u, never);
            if (!is_v && lane == 0) ft_wait(q_full, 0, never);
        }
    } else if (warp == MMA_WARP) {
        if (lane == 0 && !*abort_flag) {
            // ---- MMA issuer.  The tensor core runs what this thread issues in order, so S(i + 2),
            // which goes where S(i) and then P(i) were, follows P V of block i without a barrier.
            constexpr uint32_t idesc_s = ft_idesc(FT_BM, BN, 0);
            constexpr uint32_t idesc_o = ft_idesc(FT_BM, HEAD_DIM, 1);
            auto issue_s = [&](int i) -> bool {                        // S(i) = Q K(i)^T into S buffer i & 1
                const int s = i & 1, ks = i % STAGES;
                if (!ft_wait(&k_full[ks], (uint32_t)(i / STAGES) & 1u, abort_flag)) return false;
                ft_fence_after();
                const uint32_t qa = ft_smem(q_s), ka = ft_smem(k_s + ks * L::KV_BYTES);
#pragma unroll
                for (int k = 0; k < HEAD_DIM / 16; ++k) {
                    const uint32_t off = (uint32_t)((k & 3) * 32), atom = (uint32_t)(k >> 2);
                    ft_mma(tmem_s + (uint32_t)(s * BN), ft_desc_kmajor(qa + atom * FT_ATOM_BYTES + off),
                           ft_desc_kmajor(ka + atom * L::ATOM + off), idesc_s, k > 0 ? 1u : 0u);
                }
                ft_commit(&k_empty[ks]);            // the key stage is free once these MMAs have read it
                ft_commit(&s_full[s]);
                return true;
            };
            bool ok = ft_wait(q_full, 0, abort_flag);
            if (ok) ok = issue_s(0);
            for (int i = 0; i < n_blocks && ok; ++i) {
                // S(i + 1) overwrites buffer (i + 1) & 1, which held S(i - 1) and P(i - 1): the wait on
                // p_full of block i - 1 (a round ago) says the softmax has read that S, and P V of block
                // i - 1 was issued before this
                if (i + 1 < n_blocks && !issue_s(i + 1)) { ok = false; break; }
                const int b = i & 1, vs = i % STAGES;
                if (!ft_wait(&v_full[vs], (uint32_t)(i / STAGES) & 1u, abort_flag)) { ok = false; break; }
                if (clears && i == n_blocks - 1 && !ft_wait(z_full, 0, abort_flag)) { ok = false; break; }
                if (!ft_wait(&p_full[b], (uint32_t)(i >> 1) & 1u, abort_flag)) { ok = false; break; }
                ft_fence_after();
                // O (+)= P(i) V(i): A = P from tensor memory (rows in the lanes, 16 keys = 8 columns of
                // bfloat16 pairs, at the start of S buffer b); B = V: MN-major, 16 keys = two 8-row groups
                const uint32_t pa = tmem_s + (uint32_t)(b * BN), va = ft_smem(v_s + vs * L::KV_BYTES);
#pragma unroll
                for (int k = 0; k < BN / 16; ++k)
                    ft_mma_ts(tmem_o, pa + (uint32_t)(k * 8), ft_desc_mnmajor(va + (uint32_t)(k * 16 * 128), L::ATOM), idesc_o,
                              (i > 0 || k > 0) ? 1u : 0u);
                ft_commit(&v_empty[vs]);
                ft_commit(&o_done[b]);              // O holds the blocks up to i
            }
            if (!ok && !*abort_flag) { *abort_flag = 1; atomicCAS(status, 0, FT_ERR_WAIT); }
        }
    } else {
        // ---- softmax: PARTS threads (r, r + 128, ...) share query row r; `part` says which
        // KP keys of a block and which OD output columns a thread owns.  P goes back into
        // tensor memory, over the first half of the S it was made from, as the A operand of P V,
        // and O stays in tensor memory, where P V accumulates; it is rescaled (read, multiplied,
        // written back by these threads) only when a row's maximum has grown by more than 2^8
        // since the scale in use was set: until then the exponentials simply use the older maximum
        // (they stay below 2^8, well inside bfloat16 and float), and no thread waits for the last P V.
        const int r = threadIdx.x & 127;
        const int part = threadIdx.x >> 7;
        const int pos_r = ctx + row0 + r;
        const uint32_t lane_base = (uint32_t)((warp & 3) * 32) << 16;
        // [round parity][part][row]: a round's values stay untouched while the next round's are written
        float* part_max_all = reinterpret_cast<float*>(bars + L::BAR_SLOTS);
        float m_run = -CUDART_INF_F, l_run = 0.0f;           // m_run: the maximum the scale in use is based on
        if (ROWS && sink != nullptr) {                       // the running maximum and sum start from the sink's term
            m_run = sink[h] * 1.4426950408889634f;
            l_run = part == 0 ? 1.0f : 0.0f;
        }
        float l_odd = 0.0f;                                  // ROWS: l_run is for keys 0 and 1 of the thread's fours, this for the others
        auto row_sum = [&](const float* sums) -> float {     // ROWS: pairs first, as the other kernel's lanes add them
            if (PARTS == 4) return (sums[r] + sums[128 + r]) + (sums[2 * 128 + r] + sums[3 * 128 + r]);
            return sums[r] + sums[128 + r];
        };
        // 32 columns of this thread's part of the row, from column c, with the row's sum
        auto write_row = [&](const uint32_t (&w)[32], int c, float l_row) {
            const float inv = 1.0f / l_row;
            const bool by_channel = gate_cols > 1;            // else one number for the head
            const bf16* gate_row = nullptr;
            if (ROWS && gate != nullptr)
                gate_row = gate + (long)(tok0 + r) * gate_ld + (long)h * gate_cols + (by_channel ? part * OD : 0);
            bf16* dst = out + (long)(tok0 + r) * out_ld + (long)h * HEAD_DIM + part * OD;
#pragma unroll
            for (int d = 0; d < 32; d += 8) {
                uint4 o4;
                __nv_bfloat162* wp = reinterpret_cast<__nv_bfloat162*>(&o4);
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    float f0 = __uint_as_float(w[d + 2 * e]) * inv, f1 = __uint_as_float(w[d + 2 * e + 1]) * inv;
                    if (ROWS && gate_row != nullptr) {
                        const int at = by_channel ? c + d + 2 * e : 0;
                        f0 = f0 / (1.0f + expf(-__bfloat162float(gate_row[at])));
                        f1 = f1 / (1.0f + expf(-__bfloat162float(gate_row[by_channel ? at + 1 : 0])));
                    }
                    wp[e] = __floats2bfloat162_rn(f0, f1);
                }
                *reinterpret_cast<uint4*>(dst + c + d) = o4;
            }
        };
        bool ok = !*abort_flag;
        for (int i = 0; i < n_blocks && ok; ++i) {
            const int sb = i & 1;
            // A wait on o_done tells a phase from the one before it only, so neither of the two barriers may get two phases
            // ahead of this warp: P(i), which it sends below, lets P V of block i go, so that of block i - 2 is waited for
            // here (S(i) came after it: where S(i) is there, this wait is over at once).
            if (i > 1 && !ft_warp_wait(&o_done[i & 1], (uint32_t)((i - 2) >> 1) & 1u, abort_flag)) FT_GIVE_UP();
            if (!ft_warp_wait(&s_full[sb], (uint32_t)(i >> 1) & 1u, abort_flag)) FT_GIVE_UP();
            ft_fence_after();
            // O holds blocks 0 .. i - 1 once P V of block i - 1 is complete.  The whole warp reads,
            // scales and writes its rows back (rows that keep their scale by 1): the loads and
            // stores of tensor memory are warp-wide instructions.  Rows that are `over` have seen their last block and are written.
            auto rescale_o = [&](float corr, bool over, float l_row) -> bool {
                if (!ft_warp_wait(&o_done[(i - 1) & 1], (uint32_t)((i - 1) >> 1) & 1u, abort_flag)) return false;
                ft_fence_after();
                const uint32_t o_addr = tmem_o + lane_base + (uint32_t)(part * OD);
                uint32_t w[OD / 32][32];
#pragma unroll
                for (int c = 0; c < OD / 32; ++c) ft_ld32(o_addr + (uint32_t)(c * 32), w[c]);
                ft_ld_wait();
#pragma unroll
                for (int c = 0; c < OD / 32; ++c) {
                    if (ROWS && over) write_row(w[c], c * 32, l_row);
#pragma unroll
                    for (int j = 0; j < 32; ++j) w[c][j] = __float_as_uint(__uint_as_float(w[c][j]) * corr);
                    ft_st32(o_addr + (uint32_t)(c * 32), w[c]);
                }
                return true;
            };
            if constexpr (ROWS) {
                // of every eight keys E (neighbours) are this thread's, so that a row's partial sums are those of the other kernel
                constexpr int E = 8 / PARTS;
                uint32_t w[KP];
#pragma unroll
                for (int g = 0; g < 8; ++g) {
                    const uint32_t s_addr = tmem_s + (uint32_t)(sb * BN + g * 8 + part * E) + lane_base;
                    if constexpr (E == 4) ft_ld4(s_addr, w + g * E);
                    else ft_ld2(s_addr, w + g * E);
                }
                ft_ld_wait();
                const int key0 = i * BN + part * E;
                float x[KP], mx4[4] = {-CUDART_INF_F, -CUDART_INF_F, -CUDART_INF_F, -CUDART_INF_F};
#pragma unroll
                for (int j = 0; j < KP; ++j) x[j] = __fmul_rn(__fmul_rn(__uint_as_float(w[j]), scale), 1.4426950408889634f);
                if (i * BN + BN - 1 > pos_r) {
#pragma unroll
                    for (int j = 0; j < KP; ++j)
                        if (key0 + j / E * 8 + j % E > pos_r) x[j] = -CUDART_INF_F;
                }
#pragma unroll
                for (int j = 0; j < KP; ++j) mx4[j & 3] = fmaxf(mx4[j & 3], x[j]);
                const float mx = fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3]));
                float* part_max = part_max_all + sb * (PARTS * 128);
                float* part_l = part_max + 2 * PARTS * 128;
                part_max[part * 128 + r] = mx;
                part_l[part * 128 + r] = l_run + l_odd;
                ft_warp_arrive(x_bar);                                    // past it S may be overwritten by P
                if (!ft_warp_wait(x_bar, (uint32_t)i & 1u, abort_flag)) FT_GIVE_UP();
                float m_new = fmaxf(m_run, part_max[r]);
#pragma unroll
                for (int q = 1; q < PARTS; ++q) m_new = fmaxf(m_new, part_max[q * 128 + r]);
                const float corr = ft_weight(m_run, m_new);
                m_run = m_new;
                l_run *= corr;
                l_odd *= corr;
                uint32_t packed[KP / 2];
#pragma unroll
                for (int c = 0; c < KP / 2; ++c) {
                    const float p0 = ft_weight(x[2 * c], m_new), p1 = ft_weight(x[2 * c + 1], m_new);
                    float& l = E == 4 && (c & 1) ? l_odd : l_run;
                    l += p0;
                    l += p1;
                    const __nv_bfloat162 b = __floats2bfloat162_rn(p0, p1);
                    packed[c] = *reinterpret_cast<const uint32_t*>(&b);
                }
#pragma unroll
                for (int g = 0; g < 8; ++g) {
                    const uint32_t p_addr = tmem_s + (uint32_t)(sb * BN + g * 4 + part * E / 2) + lane_base;
                    if constexpr (E == 4) ft_st2(p_addr, packed[2 * g], packed[2 * g + 1]);
                    else ft_st1(p_addr, packed[g]);
                }
                // A row that sees no key of this block or of later ones is done here, before their values are added: a weight of
                // zero does not make a value that is not finite vanish.
                const bool over = i > 0 && r < rows_here && pos_r / BN + 1 == i;
                if (i > 0 && __any_sync(0xffffffffu, corr != 1.0f || over) &&
                    !rescale_o(corr, over, row_sum(part_l))) FT_GIVE_UP();
                ft_st_wait();
                ft_fence_before();
                ft_warp_arrive(&p_full[sb]);
                continue;
            }
            const int key0 = (kb_begin + i) * FT_BN + part * KP;      // first key of this thread's part
            const uint32_t s_addr = tmem_s + (uint32_t)(sb * FT_BN + part * KP) + lane_base;
            const bool all_seen = (key0 + KP - 1 <= pos_r) && (window <= 0 || key0 > pos_r - window);
            uint32_t v[KP];
#pragma unroll
            for (int c = 0; c < KP; c += 32) ft_ld32(s_addr + (uint32_t)c, v + c);
            ft_ld_wait();
            if (!all_seen) {
#pragma unroll
                for (int j = 0; j < KP; ++j) {
                    const int key = key0 + j;
                    if (!(key <= pos_r && (window <= 0 || key > pos_r - window))) v[j] = 0xff800000u;   // -inf
                }
            }
            float mx4[4] = {-CUDART_INF_F, -CUDART_INF_F, -CUDART_INF_F, -CUDART_INF_F};
#pragma unroll
            for (int j = 0; j < KP; j += 4) {
#pragma unroll
                for (int e = 0; e < 4; ++e) mx4[e] = fmaxf(mx4[e], __uint_as_float(v[j + e]));
            }
            const float mx = fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3]));
            // exchange the parts' maxima (one barrier among the softmax warps per block); past it
            // every softmax thread has its S in registers, so the S buffer may take P
            float* part_max = part_max_all + (i & 1) * (PARTS * 128);
            part_max[part * 128 + r] = mx;
            ft_warp_arrive(x_bar);                                        // (an mbarrier: its wait can give up)
            if (!ft_warp_wait(x_bar, (uint32_t)i & 1u, abort_flag)) FT_GIVE_UP();
            float mx_row = part_max[r];
#pragma unroll
            for (int q = 1; q < PARTS; ++q) mx_row = fmaxf(mx_row, part_max[q * 128 + r]);
            const float m_new = fmaxf(m_run, mx_row * scale_log2e);
            // the row's threads decide alike: they see the same maxima
            const bool rescale = m_new > m_run + 8.0f || (m_run == -CUDART_INF_F && m_new != -CUDART_INF_F);
            const bool any_rescale = __any_sync(0xffffffffu, rescale);
            float corr = 1.0f;
            if (rescale) {
                corr = ft_weight(m_run, m_new);
                l_run *= corr;
                m_run = m_new;
            }
            if (any_rescale && i > 0 && !rescale_o(corr, false, 0.0f)) FT_GIVE_UP();
            const float neg_m = (m_run == -CUDART_INF_F) ? 0.0f : -m_run;      // an empty row: every p below is 0
            float l4[4] = {0.0f, 0.0f, 0.0f, 0.0f};
            uint32_t packed[KP / 2];
#pragma unroll
            for (int c = 0; c < KP / 2; ++c) {
                const float p0 = ft_ex2(fmaf(__uint_as_float(v[2 * c]), scale_log2e, neg_m));
                const float p1 = ft_ex2(fmaf(__uint_as_float(v[2 * c + 1]), scale_log2e, neg_m));
                l4[c & 3] += p0 + p1;
                const __nv_bfloat162 b = __floats2bfloat162_rn(p0, p1);
                packed[c] = *reinterpret_cast<const uint32_t*>(&b);
            }
            l_run += (l4[0] + l4[1]) + (l4[2] + l4[3]);
            // P(i): this thread's KP keys as KP / 2 columns of bfloat16 pairs
#pragma unroll
            for (int c = 0; c < KP / 2; c += 32)
                ft_st32(tmem_s + (uint32_t)(sb * FT_BN + part * (KP / 2) + c) + lane_base, packed + c);
            ft_st_wait();
            ft_fence_before();
            ft_warp_arrive(&p_full[sb]);
        }
        // the whole of O, then the row's sum: the parts' sums (all relative to the same maximum)
        if (ok && n_blocks > 0) {
            ok = ft_warp_wait(&o_done[(n_blocks - 1) & 1], (uint32_t)((n_blocks - 1) >> 1) & 1u, abort_flag);
            if (!ok && !*abort_flag) { *abort_flag = 1; atomicCAS(status, 0, FT_ERR_WAIT); }
            ft_fence_after();
        }
        float* part_sum = part_max_all + (n_blocks & 1) * (PARTS * 128);
        part_sum[part * 128 + r] = ROWS ? l_run + l_odd : l_run;
        ft_warp_arrive(x_bar);
        const bool met = ft_warp_wait(x_bar, (uint32_t)n_blocks & 1u, abort_flag);
        const float l_row = row_sum(part_sum);
        if (met && ok && !*abort_flag && n_blocks > 0) {
            const bool mine = r < rows_here && (!ROWS || pos_r / BN + 1 == n_blocks);
#pragma unroll
            for (int c = 0; c < OD; c += 32) {
                uint32_t w[32];
                ft_ld32(tmem_o + lane_base + (uint32_t)(part * OD + c), w);      // all lanes of the warp take part
                ft_ld_wait();
                if (mine) write_row(w, c, l_row);
            }
        }
    }
#undef FT_GIVE_UP
    ft_fence_before();
    __syncthreads();
    if (warp == MMA_WARP) {
        ft_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
    }
}

// ----------------------------------------------------------------- host side
typedef CUresult (*FtEncodeFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                               const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                               CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
static FtEncodeFn ft_encode_fn() {
    static FtEncodeFn fn = nullptr;
    if (!fn) {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = (FtEncodeFn)p;
    }
    return fn;
}
static int ft_make_map(CUtensorMap* map, const void* base, long rows, long cols, long ld, int box_rows) {
    FtEncodeFn fn = ft_encode_fn();
    if (!fn) return (int)cudaErrorNotSupported;
    if (((uintptr_t)base & 15) || ((ld * 2) & 15)) return (int)cudaErrorMisalignedAddress;
    cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
    cuuint64_t strides[1] = {(cuuint64_t)ld * 2};
    cuuint32_t box[2] = {64, (cuuint32_t)box_rows};
    cuuint32_t elem[2] = {1, 1};
    CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides, box, elem,
                    CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                    CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? 0 : (int)cudaErrorInvalidValue;
}

FL_API int fl_attention_prefill_tc_head_dim() { return HEAD_DIM; }
FL_API int fl_attention_prefill_tc_takes(int page_size) {
    return page_size >= 8 && page_size <= FT_BN && page_size % 8 == 0 && FT_BN % page_size == 0;
}

template <bool ROWS>
static int ft_launch(const void* q, long q_ld, void* out, long out_ld, const void* cache, long n_pages, int page_size,
                     const int* block_table, int bt_stride, const int* req_start, const int* req_ctx, const int* req_qlen,
                     int n_requests, int n_tokens, int include_single, int n_heads, int n_kv_heads, int window, float scale,
                     const float* sink, const void* gate, long gate_ld, int gate_cols, int* status, cudaStream_t stream) {
    if (n_requests <= 0 || n_tokens <= 0) return 0;
    if (!fl_attention_prefill_tc_takes(page_size) || n_heads > 65535 || n_heads % n_kv_heads)
        return (int)cudaErrorInvalidValue;
    if ((q_ld % 8) || (out_ld % 8)) return (int)cudaErrorMisalignedAddress;
    const long kv_rows = n_pages * (ROWS ? 1 : 2) * n_kv_heads * page_size;
    if (kv_rows >= (1l << 31)) return (int)cudaErrorInvalidValue;
    CUtensorMap map_q, map_kv;
    int rc = ft_make_map(&map_q, q, n_tokens, (long)n_heads * HEAD_DIM, q_ld, FT_BM);
    if (rc) return rc;
    rc = ft_make_map(&map_kv, cache, kv_rows, ROWS ? 2 * HEAD_DIM : HEAD_DIM, ROWS ? 2 * HEAD_DIM : HEAD_DIM,
                     page_size < FtSmem<ROWS>::BN ? page_size : FtSmem<ROWS>::BN);
    if (rc) return rc;
    static bool configured = false;
    if (!configured) {
        cudaError_t e = cudaFuncSetAttribute(attention_prefill_tc_kernel<ROWS>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             FtSmem<ROWS>::TOTAL);
        if (e != cudaSuccess) return (int)e;
        configured = true;
    }
    const int max_tiles = n_tokens / FT_BM + n_requests;
    if (max_tiles > 65535) return (int)cudaErrorInvalidValue;
    dim3 grid(n_heads, max_tiles);                 // heads fastest: every head's late (long) tiles start first
    // plain stream order (no programmatic overlap): this kernel takes all of an SM's tensor memory
    attention_prefill_tc_kernel<ROWS><<<grid, FtSmem<ROWS>::THREADS, FtSmem<ROWS>::TOTAL, stream>>>(
        map_q, map_kv, (bf16*)out, out_ld, page_size, (int)kv_rows, block_table, bt_stride, req_start, req_ctx,
        req_qlen, n_requests, include_single, n_heads, n_kv_heads, window, scale, status, sink,
        (const bf16*)gate, gate_ld, gate_cols);
    return fl_launch_status();
}

// The arguments of fl_attention_prefill (attention_prefill.cu) with the cache given
// as one tensor [n_pages, 2, n_kv_heads, page_size, HEAD_DIM] and a status word.
FL_API int fl_attention_prefill_tc(const void* q, long q_ld, void* out, long out_ld, const void* cache,
                                   long n_pages, int page_size, const int* block_table, int bt_stride,
                                   const int* req_start, const int* req_ctx, const int* req_qlen,
                                   int n_requests, int n_tokens, int include_single, int n_heads,
                                   int n_kv_heads, int window, float scale, int* status, cudaStream_t stream) {
    return ft_launch<false>(q, q_ld, out, out_ld, cache, n_pages, page_size, block_table, bt_stride, req_start, req_ctx,
                            req_qlen, n_requests, n_tokens, include_single, n_heads, n_kv_heads, window, scale, nullptr,
                            nullptr, 0, 0, status, stream);
}

// The same over a cache of rows k | v, [n_pages, n_kv_heads, page_size, 2 HEAD_DIM], every earlier token seen, with a sink
// and a gate (see the kernel; either may be null).
FL_API int fl_attention_prefill_rows(const void* q, long q_ld, void* out, long out_ld, const void* cache, long n_pages,
                                     int page_size, const int* block_table, int bt_stride, const int* req_start,
                                     const int* req_ctx, const int* req_qlen, int n_requests, int n_tokens,
                                     int include_single, int n_heads, int n_kv_heads, float scale, const float* sink,
                                     const void* gate, long gate_ld, int gate_cols, int* status, cudaStream_t stream) {
    return ft_launch<true>(q, q_ld, out, out_ld, cache, n_pages, page_size, block_table, bt_stride, req_start, req_ctx,
                           req_qlen, n_requests, n_tokens, include_single, n_heads, n_kv_heads, 0, scale, sink, gate,
                           gate_ld, gate_cols, status, stream);
}
