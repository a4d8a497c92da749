// Shared by the products on the Blackwell tensor cores (gemm_tcgen05.cu, moe.cu) and the latent attention of prompts
// (latent_attention_tc.cu): tile sizes, the PTX that TMA loads, mbarriers, tensor memory and tcgen05.mma take, the gated units
// of the products' epilogues and how their warps give up, and the tensor maps.
#pragma once

#include <cuda.h>

#include "common.cuh"

#define TC_BM 128            // weight rows (output features) per CTA tile
#define TC_BK 64             // K elements per stage: 128 bytes of bfloat16, one swizzle row
#define TC_THREADS 192
#define TC_WAIT_LIMIT_NS 2000000000ull

enum { TC_ERR_FULL_WAIT = 101, TC_ERR_EMPTY_WAIT = 102, TC_ERR_ACC_WAIT = 103 };

// ------------------------------------------------------------------ PTX wraps
__device__ __forceinline__ uint32_t smem_u32(const void* p) {
    return (uint32_t)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)),
                 "r"(bytes)
                 : "memory");
}
__device__ __forceinline__ uint32_t mbar_try_wait(uint64_t* bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok;
}
__device__ __forceinline__ uint64_t global_ns() {
    uint64_t t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}
// Waits for the barrier's phase `parity` to complete.  Gives up (returns false)
// when another role has already given up or after TC_WAIT_LIMIT_NS.
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, volatile int* abort_flag) {
    if (mbar_try_wait(bar, parity)) return true;
    const uint64_t t0 = global_ns();
    uint32_t spins = 0;
    while (!mbar_try_wait(bar, parity)) {
        if ((++spins & 255u) == 0) {
            if (*abort_flag) return false;
            if (global_ns() - t0 > TC_WAIT_LIMIT_NS) return false;
        }
    }
    return true;
}
// For a CTA that gives up: the copies on their way must land before its shared memory goes to another CTA.  Called by the
// thread that issued `issued` fills of a ring of `stages`: waits for the last of them, up to the first that does not land
// within the limit, and a millisecond more (the fills of a pair's other CTA signal the leader's barriers only, which take no
// notice of them before the leader's own).
__device__ __forceinline__ void tma_drain(uint64_t* full_bar, int stages, int issued) {
    bool landed = true;
    for (int k = issued > stages ? issued - stages : 0; k < issued && landed; ++k) {
        const uint64_t t0 = global_ns();
        while (landed && !mbar_try_wait(&full_bar[k % stages], (uint32_t)(k / stages) & 1u)) landed = global_ns() - t0 <= TC_WAIT_LIMIT_NS;
    }
    const uint64_t t0 = global_ns();
    while (issued > 0 && global_ns() - t0 < 1000000ull) {}
}
__device__ __forceinline__ void tma_load_2d(void* dst, const CUtensorMap* map, uint64_t* bar, int x,
                                            int y) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes"
        " [%0], [%1, {%3, %4}], [%2];" ::"r"(smem_u32(dst)),
        "l"((uint64_t)map), "r"(smem_u32(bar)), "r"(x), "r"(y)
        : "memory");
}
__device__ __forceinline__ void tmem_alloc(uint32_t* dst_smem, uint32_t cols) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_u32(dst_smem)),
                 "r"(cols)
                 : "memory");
}
__device__ __forceinline__ void tmem_relinquish() {
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t cols) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(cols)
                 : "memory");
}
__device__ __forceinline__ void tc_fence_before() {
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_after() {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void umma_bf16(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc,
                                          uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem_d),
        "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}
__device__ __forceinline__ void umma_commit(uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                     smem_u32(bar))
                 : "memory");
}
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t* r) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
          "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
          "=r"(r[14]), "=r"(r[15])
        : "r"(taddr)
        : "memory");
}
__device__ __forceinline__ void tmem_ld_wait() {
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

// silu(g) * u with the fast exponential and division: the epilogue has a fixed budget per tile (the
// next tile's MMAs), and the exact forms cost five times the instructions for digits that a
// bfloat16 result cannot hold (relative error about 1e-6 against bfloat16's 4e-3).
// `ACT` is an FlAct (common.cuh): silu, relu, gelu in its tanh form, or the clamped swish unit with its two constants.
template <int ACT> __device__ __forceinline__ float gated_one(float g, float u, const FlGate act) {
    if (ACT == FL_ACT_RELU) return fmaxf(g, 0.0f) * u;
    if (ACT == FL_ACT_RELU_SQUARED) return fmaxf(g, 0.0f) * fmaxf(g, 0.0f) * u;
    if (ACT == FL_ACT_GELU_TANH) return 0.5f * g * (1.0f + tanhf(0.7978845608028654f * (g + 0.044715f * g * g * g))) * u;
    if (ACT == FL_ACT_CLAMPED_SWISH) {
        g = fminf(g, act.p0);
        u = fminf(fmaxf(u, -act.p0), act.p0);
        return __fdividef(g, 1.0f + __expf(-act.p1 * g)) * (u + 1.0f);
    }
    return __fdividef(g, 1.0f + __expf(-g)) * u;
}
// g[j] = f(g[j], u[j]) for the launch's unit.  The unit is chosen once for all N values and not per value: a warp is
// alone on its scheduler here, so its speed is how many of the N chains of dependent instructions are in flight, and a
// choice per value put them one behind another: the 256 x 256 tile's epilogue then took 25 to 30 us, three times its MMAs
// at K = 2048.  The pair kernel's gated product of 2048 tokens, K = 4096, 2 x 11008 features took 413 us and takes 240
// (1540 TFLOP/s), of 1310 tokens, K = 2048, 2 x 5504 features 128 and 54.
template <int ACT, int N> __device__ __forceinline__ void gated_all(float (&g)[N], const float (&u)[N], const FlGate act) {
#pragma unroll
    for (int j = 0; j < N; ++j) g[j] = gated_one<ACT>(g[j], u[j], act);
}
template <int N> __device__ __forceinline__ void gated_act(float (&g)[N], const float (&u)[N], const FlGate act) {
    switch (act.act) {
        case FL_ACT_RELU: gated_all<FL_ACT_RELU>(g, u, act); break;
        case FL_ACT_RELU_SQUARED: gated_all<FL_ACT_RELU_SQUARED>(g, u, act); break;
        case FL_ACT_GELU_TANH: gated_all<FL_ACT_GELU_TANH>(g, u, act); break;
        case FL_ACT_CLAMPED_SWISH: gated_all<FL_ACT_CLAMPED_SWISH>(g, u, act); break;
        default: gated_all<FL_ACT_SILU>(g, u, act);
    }
}

// A product that is not gated may pass an activation of one argument on its way out: f(v, 1), or FL_ACT_NONE.
template <int N> __device__ __forceinline__ void unary_act(uint32_t (&r)[N], const FlGate act) {
    if (act.act == FL_ACT_NONE) return;
    float g[N], one[N];
#pragma unroll
    for (int j = 0; j < N; ++j) g[j] = __uint_as_float(r[j]), one[j] = 1.0f;
    gated_act(g, one, act);
#pragma unroll
    for (int j = 0; j < N; ++j) r[j] = __float_as_uint(g[j]);
}

// A barrier among the four epilogue warps only (hardware barrier 1; barrier 0 is __syncthreads).
__device__ __forceinline__ void epilogue_sync() { asm volatile("bar.sync 1, 128;" ::: "memory"); }
// The same, and whether any of the 128 threads came with `flag`: how they decide to give up.  After a plain barrier each
// would read the abort flag for itself, and one that another role sets between two of these reads would leave some warps at
// a barrier that the others never come to.
__device__ __forceinline__ bool epilogue_any(bool flag) {
    uint32_t any;
    __syncwarp();
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t"
        "setp.ne.u32 p, %1, 0;\n\t"
        "bar.red.or.pred q, 1, 128, p;\n\t"
        "selp.u32 %0, 1, 0, q;\n\t}"
        : "=r"(any)
        : "r"((uint32_t)flag)
        : "memory");
    return any != 0;
}

// Shared-memory matrix descriptor of a K-major tile whose rows are 128 bytes
// (64 bfloat16) in the 128-byte swizzle: 8-row groups are 1024 bytes apart.
__device__ __forceinline__ uint64_t smem_desc_sw128(uint32_t saddr) {
    uint64_t d = 0;
    d |= (uint64_t)((saddr & 0x3FFFFu) >> 4);   // start address, 16-byte units
    d |= (uint64_t)1 << 16;                     // leading byte offset (unused with swizzle)
    d |= (uint64_t)(1024 >> 4) << 32;           // stride byte offset between 8-row groups
    d |= (uint64_t)1 << 46;                     // descriptor version of sm_100
    d |= (uint64_t)2 << 61;                     // SWIZZLE_128B
    return d;
}

// kind::f16 instruction descriptor: float accumulator, bfloat16 A and B, both K-major.
__host__ __device__ constexpr uint32_t instr_desc_bf16(int m, int n) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) |
           ((uint32_t)(m >> 4) << 24);
}

// Rows of 128 (or fewer) values from the epilogue's staging area to global memory, 16 bytes per
// thread where the destination allows it: `e` is the thread's index among the 128 epilogue threads,
// `cols` how many of the 128 columns exist.  Written this way a warp stores whole rows of 256 or 512
// bytes; one value per lane and row (what the accumulator's layout gives) took 40 ns per token.
template <typename T, int WIDTH, int ROWS = 32>
__device__ __forceinline__ void tc_copy_rows(T* __restrict__ dst, long ld, const T* __restrict__ src, int rows,
                                             int cols, int e, bool vec_ok) {
    constexpr int V = 16 / (int)sizeof(T);                  // values per 16 bytes
    constexpr int TPR = WIDTH / V;                          // threads per row
    constexpr int RPP = 128 / TPR;                          // rows per pass
    const int rr = e / TPR, cc = (e % TPR) * V;
#pragma unroll
    for (int p = 0; p < (ROWS + RPP - 1) / RPP; ++p) {
        const int row = p * RPP + rr;
        if (row >= rows || cc >= cols) continue;
        T* d = dst + (long)row * ld + cc;
        const T* s_ = src + row * WIDTH + cc;
        if (vec_ok && cc + V <= cols) {
            *reinterpret_cast<uint4*>(d) = *reinterpret_cast<const uint4*>(s_);
        } else {
            for (int v = 0; v < V && cc + v < cols; ++v) d[v] = s_[v];
        }
    }
}

#define TC2_PEER_MASK 0xFEFFFFFFu                          // clears the CTA-rank bit of a shared::cluster address

// ------------------------------------------------------------ CTA pairs
// A stage of the CTA-pair kernels (see gemm_tcgen05.cu).
template <int BNT>
struct Tc2 {
    static constexpr int W_BYTES = TC_BM * TC_BK * 2;              // 128 weight rows of a stage
    static constexpr int A_BYTES = (BNT / 2) * TC_BK * 2;          // this CTA's half of the token rows
    static constexpr int STAGE_BYTES = W_BYTES + A_BYTES;
    static constexpr int STAGES = BNT == 256 ? 6 : (BNT == 128 ? 8 : 9);
    static constexpr int TILE_BYTES = STAGES * STAGE_BYTES;
    static constexpr int SMEM = TILE_BYTES + 256 + 1024;        // + the epilogue's area below
};

__device__ __forceinline__ uint32_t cluster_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void cluster_sync_all() {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ void tma_load_2d_pair(void* dst, const CUtensorMap* map, uint64_t* leader_bar, int x,
                                                 int y) {
    asm volatile(
        "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes"
        " [%0], [%1, {%3, %4}], [%2];" ::"r"(smem_u32(dst)),
        "l"((uint64_t)map), "r"(smem_u32(leader_bar) & TC2_PEER_MASK), "r"(x), "r"(y)
        : "memory");
}
__device__ __forceinline__ void umma_bf16_pair(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                               uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem_d),
        "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}
__device__ __forceinline__ void umma_commit_pair(uint64_t* bar) {      // arrives on this barrier in both CTAs
    asm volatile(
        "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(
            smem_u32(bar)),
        "h"((uint16_t)3)
        : "memory");
}
__device__ __forceinline__ void mbar_arrive_leader(uint64_t* bar) {    // arrive on the even CTA's copy of `bar`
    asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(smem_u32(bar) & TC2_PEER_MASK) : "memory");
}

// ------------------------------------------------------------ tensor maps
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*,
                                  const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                                  const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeTiledFn encode_tiled_fn() {
    static EncodeTiledFn fn = nullptr;
    if (!fn) {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = (EncodeTiledFn)p;
    }
    return fn;
}

// A [rows, cols] bfloat16 matrix with `ld` elements between rows, read in boxes
// of box_rows x 64 elements with the 128-byte swizzle; out-of-range reads give zeros.
static int make_map(CUtensorMap* map, const void* base, long rows, long cols, long ld, int box_rows) {
    EncodeTiledFn fn = encode_tiled_fn();
    if (!fn) return (int)cudaErrorNotSupported;
    if (((uintptr_t)base & 15) || ((ld * 2) & 15)) return (int)cudaErrorMisalignedAddress;
    cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
    cuuint64_t strides[1] = {(cuuint64_t)ld * 2};
    cuuint32_t box[2] = {TC_BK, (cuuint32_t)box_rows};
    cuuint32_t elem[2] = {1, 1};
    CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides,
                    box, elem, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                    CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? 0 : (int)cudaErrorInvalidValue;
}
