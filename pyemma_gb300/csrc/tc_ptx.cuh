// tc_ptx.cuh -- what the tensor-core assignment kernels share: PTX wrappers
// (mbarriers, TMA, tcgen05, TMEM), operand descriptors, the acceptance window
// of their error bound and the driver's tensor-map encoder.
#pragma once

#include <cuda.h>

#include <mutex>

#include "km_common.cuh"

namespace km {

namespace {

// Scalars shared by the prep kernels and the main kernel (uint32 words).
// kCmax, kHcMax: the largest bounds over the centers of ||c'|| and of the
// operands' rounding error, for each form of the operands.
enum ScalarSlot {
    kScale = 0, kInvScale2 = 1, kScaleMax = 2, kCmax = 3, kHcMax = 4, kSmallCmax = 5, kSmallHcMax = 6, kNumScalars = 8
};

// ---------------------------------------------------------------------------
// PTX wrappers
// ---------------------------------------------------------------------------
__device__ __forceinline__ uint32_t smem_u32(const void *p) {
    return (uint32_t)__cvta_generic_to_shared(p);
}

__device__ __forceinline__ void mbar_init(uint64_t *bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}

__device__ __forceinline__ void fence_mbar_init() {
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

__device__ __forceinline__ void mbar_arrive_expect_tx(uint64_t *bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
                 : "memory");
}

__device__ __forceinline__ void mbar_arrive(uint64_t *bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(uint64_t *bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}

// One lane of the converged warp (the same lane every time).
__device__ __forceinline__ bool elect_one() {
    uint32_t pred = 0;
    asm volatile(
        "{\n\t.reg .pred P;\n\t"
        "elect.sync _|P, 0xffffffff;\n\t"
        "selp.u32 %0, 1, 0, P;\n\t}"
        : "=r"(pred));
    return pred != 0;
}

// Waits for the phase of the given parity; false after kWaitLimitNs.
__device__ __forceinline__ bool mbar_wait(uint64_t *bar, uint32_t parity) {
    if (mbar_try_wait(bar, parity)) return true;
    const uint64_t t0 = globaltimer_ns();
    for (uint32_t spin = 1;; ++spin) {
        if (mbar_try_wait(bar, parity)) return true;
        if ((spin & 255u) == 0 && globaltimer_ns() - t0 > kWaitLimitNs) return false;
    }
}

// mbar_wait that adds the cycles it spent to *acc when acc is non-null.
__device__ __forceinline__ bool mbar_wait_timed(uint64_t *bar, uint32_t parity, unsigned long long *acc) {
    if (!acc) return mbar_wait(bar, parity);
    const long long t0 = clock64();
    const bool ok = mbar_wait(bar, parity);
    *acc += (unsigned long long)(clock64() - t0);
    return ok;
}

__device__ __forceinline__ void tma_load_2d(void *dst, const CUtensorMap *tm, int x, int y,
                                            uint64_t *bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], "
        "[%4];" ::"r"(smem_u32(dst)),
        "l"(reinterpret_cast<uint64_t>(tm)), "r"(x), "r"(y), "r"(smem_u32(bar))
        : "memory");
}

__device__ __forceinline__ void tmem_alloc(uint32_t *holder, uint32_t ncols) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(holder)),
                 "r"(ncols)
                 : "memory");
}

__device__ __forceinline__ void tmem_relinquish() {
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}

__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}

__device__ __forceinline__ void tc_fence_before() {
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}

__device__ __forceinline__ void tc_fence_after() {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}

__device__ __forceinline__ void mma_f16(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                         uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
        "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}

// FP8 (e4m3 x e4m3 -> F32): the same operand layout, 32 elements (32 bytes)
// per K step.
__device__ __forceinline__ void mma_f8(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                        uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f8f6f4 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
        "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}

__device__ __forceinline__ void mma_commit(uint64_t *bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                     smem_u32(bar))
                 : "memory");
}

// ---- CTA pairs (cluster of 2, tcgen05 cta_group::2) ----
__device__ __forceinline__ uint32_t cluster_ctarank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}

// Address of the same shared-memory offset in CTA `rank` of the cluster.
__device__ __forceinline__ uint32_t mapa_shared(uint32_t addr, uint32_t rank) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}

// Every thread of both CTAs.
__device__ __forceinline__ void cluster_sync_all() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// Arrive on a barrier of either CTA of the pair.  The default (CTA-scope)
// release: the arrive only has to follow the thread's completed tcgen05.ld of
// the accumulator (ordered by tcgen05.fence::before_thread_sync), not its
// global stores, which a cluster-scope release would wait for.
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t cluster_addr) {
    asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}

// Wait on a local barrier that threads of the peer CTA arrive on.
__device__ __forceinline__ bool mbar_try_wait_cluster(uint64_t *bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}

__device__ __forceinline__ bool mbar_wait_cluster(uint64_t *bar, uint32_t parity) {
    if (mbar_try_wait_cluster(bar, parity)) return true;
    const uint64_t t0 = globaltimer_ns();
    for (uint32_t spin = 1;; ++spin) {
        if (mbar_try_wait_cluster(bar, parity)) return true;
        if ((spin & 255u) == 0 && globaltimer_ns() - t0 > kWaitLimitNs) return false;
    }
}

__device__ __forceinline__ bool mbar_wait_cluster_timed(uint64_t *bar, uint32_t parity, unsigned long long *acc) {
    if (!acc) return mbar_wait_cluster(bar, parity);
    const long long t0 = clock64();
    const bool ok = mbar_wait_cluster(bar, parity);
    *acc += (unsigned long long)(clock64() - t0);
    return ok;
}

// TMA load into this CTA's shared memory whose completion is counted on the
// barrier at `bar_cluster_addr` (the leader CTA's).
__device__ __forceinline__ void tma_load_2d_pair(void *dst, const CUtensorMap *tm, int x, int y,
                                                 uint32_t bar_cluster_addr) {
    asm volatile(
        "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, "
        "%3}], [%4];" ::"r"(smem_u32(dst)),
        "l"(reinterpret_cast<uint64_t>(tm)), "r"(x), "r"(y), "r"(bar_cluster_addr)
        : "memory");
}

__device__ __forceinline__ void tmem_alloc_pair(uint32_t *holder, uint32_t ncols) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(holder)),
                 "r"(ncols)
                 : "memory");
}

__device__ __forceinline__ void tmem_relinquish_pair() {
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}

__device__ __forceinline__ void tmem_dealloc_pair(uint32_t taddr, uint32_t ncols) {
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}

__device__ __forceinline__ void mma_f16_pair(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                              uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
        "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}

__device__ __forceinline__ void mma_f8_pair(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                             uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f8f6f4 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
        "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}

template <bool F8>
__device__ __forceinline__ void mma_op(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                       uint32_t accumulate) {
    if constexpr (F8)
        mma_f8(d_tmem, adesc, bdesc, idesc, accumulate);
    else
        mma_f16(d_tmem, adesc, bdesc, idesc, accumulate);
}

template <bool F8>
__device__ __forceinline__ void mma_op_pair(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                            uint32_t accumulate) {
    if constexpr (F8)
        mma_f8_pair(d_tmem, adesc, bdesc, idesc, accumulate);
    else
        mma_f16_pair(d_tmem, adesc, bdesc, idesc, accumulate);
}

// Arrive on the barrier at this offset in both CTAs of the pair once the
// issuing thread's earlier MMAs are complete.
__device__ __forceinline__ void mma_commit_pair(uint64_t *bar) {
    asm volatile(
        "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(
            smem_u32(bar)),
        "h"((unsigned short)3)
        : "memory");
}

__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t (&r)[32]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
        "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
          "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
          "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]),
          "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]),
          "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr));
}

// max of three floats in one instruction (PTX max.f32 with three inputs,
// sm_100 and later): NaN inputs are ignored as by fmaxf.
__device__ __forceinline__ float max3f(float a, float b, float c) {
    float d;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}

__device__ __forceinline__ void tmem_wait_ld() {
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

// Shared-memory matrix descriptor: K-major operand in the 128-byte swizzle
// layout written by TMA (8-row atoms of 128 B, atoms 1024 B apart).
__device__ __forceinline__ uint64_t sw128_desc(uint32_t saddr) {
    uint64_t desc = 0;
    desc |= (uint64_t)((saddr & 0x3FFFFu) >> 4);  // start address
    desc |= (uint64_t)1 << 16;                    // leading byte offset (unused for SW128 K-major)
    desc |= (uint64_t)(1024 >> 4) << 32;          // stride byte offset: 8 rows x 128 B
    desc |= (uint64_t)1 << 46;                    // descriptor version
    desc |= (uint64_t)2 << 61;                    // 128-byte swizzle
    return desc;
}

// Instruction descriptor of kind::f16: FP16 x FP16 (or BF16 x BF16) -> F32,
// both K-major.  The operand-type code 0 is E4M3 under kind::f8f6f4, so the
// FP16 descriptor also serves the FP8 MMA.
__host__ __device__ constexpr uint32_t make_idesc(int M, int N, bool bf16 = false) {
    return (1u << 4) | (bf16 ? ((1u << 7) | (1u << 10)) : 0u) | ((uint32_t)(N >> 3) << 17) |
           ((uint32_t)(M >> 4) << 24);
}

// Rounding of the float32 centering x' = fl(x - m): at most 2^-24 |x - m|
// per component, so 2^-23 (sx + sc) covers both operands.
constexpr float kCenterEps = 1.1920929e-07f;  // 2^-23

// Smallest accumulator a' that can still belong to a possible argmin, given
// the best accumulator so far: with H = (sqrt(vb + E) + R)^2 g_hi the upper
// end of the best distance, lo(v') <= H needs v' <= V = (sqrt(H / g_lo) + R)^2
// + E (worst-case R, E), and v' = (||x_hat||^2 - 2 a') / s^2.  The root of
// H / g_lo is (sqrt(vb + E) + R) sqrt(g_hi / g_lo): g_ratio is that factor
// inflated by 2^-19 (more than the roundings of the literal form), and
// R_pad = R + 1e-18 covers the root of hi_bound's 1e-37 term.  Rounded
// towards admitting more throughout; one root, no division.
__device__ __forceinline__ float window_threshold(float best, float xn2, float inv_s2, float s2, float E,
                                                  float R, float R_pad, float g_ratio) {
    const float vb = fmaf(-2.0f, best, xn2) * inv_s2;
    const float a = __fadd_ru(__fsqrt_ru(fmaxf(__fadd_ru(vb, E), 0.0f)), R);
    const float q = __fadd_ru(__fmul_ru(g_ratio, a), R_pad);
    const float V = __fadd_ru(__fmul_ru(q, q), E);
    const float t = __fmul_rd(__fsub_rd(xn2, __fmul_ru(V, s2)), 0.5f);
    return __fsub_rd(t, __fmul_ru(fabsf(t), 1e-6f)) - 1e-30f;
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                                  const cuuint64_t *, const cuuint32_t *, const cuuint32_t *,
                                  CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion,
                                  CUtensorMapFloatOOBfill);

EncodeTiledFn get_encode() {
    static EncodeTiledFn fn = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void *p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) ==
                cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<EncodeTiledFn>(p);
    });
    return fn;
}

bool device_is_sm10x() {
    static int cc[kDeviceSlots] = {};  // compute capability major + 1 (0: not read yet)
    const int dev = current_device();
    if (dev >= 0 && dev < kDeviceSlots && cc[dev]) return cc[dev] == 11;
    int major = 0;
    cudaDeviceGetAttribute(&major, cudaDevAttrComputeCapabilityMajor, dev);
    if (dev >= 0 && dev < kDeviceSlots) cc[dev] = major + 1;
    return major == 10;
}

}  // namespace

}  // namespace km
