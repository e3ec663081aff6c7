// assign_small.cu -- nearest-center assignment of narrow frames (d <= 31):
// tcgen05 distances from split operands pick eight centers per frame, and
// their exact float32 distances give the label, in one kernel.
//
// Reference: ClusterModel(centers, 'euclidean').transform(X),
// pyemma/coordinates/clustering/interface.py:157-167 (and the assignment step
// inside KMeans.fit, kmeans.py:253).
//
// At small d the tensor pipe is idle whatever the operands are, so it can
// afford precision: with x' = x - m and c' = c - m scaled by a power of two
// as in assign_tc.cu, every value is split into two FP16 parts, x = xh + xl
// and c = ch + cl (to about 2^-23 of the value), and feature f takes four
// columns, (xh, xl, xh, xl) against (ch, ch, cl, cl), whose products are all
// exact.  Three more columns carry -||c||^2 / 2 in three FP16 parts.  The
// accumulator a_j = x.c_j - ||c_j||^2 / 2 is then within a few 2^-21 of the
// row norms, so the centers that could be the argmin of the exact float32
// distances (window_threshold of assign_tc.cu's bound with these operands)
// are nearly always one, where plain FP16 operands leave several.
//
// That allows an epilogue without branches or lists.  Per frame (a thread)
// and eight accumulator columns: their maximum, and with it the best group's
// maximum and index and the best maximum outside that group; 9 instructions
// per 8 columns.  At the end, when the second value is below the acceptance
// threshold of the first, every possible argmin lies in the best group: the
// thread computes the eight exact distances (feature order, every operation
// rounded on its own) and takes the lowest index among the minima.
// Otherwise, and where a value is not finite, the frame is listed with its
// threshold.
//
// Listed frames (0.02-5% of continuous data at d >= 2, up to all of them on a
// lattice or with duplicate centers) are compared with all centers, by a warp
// each, or by a warp per eight where the list is long.  Large calls take long
// lists through the same kernel again, which now leaves a bit per group of
// eight centers that reaches the frame's threshold, and only those groups'
// exact distances follow; frames that are not finite, and frames beyond the
// room for the bits, are still compared with all centers.
//
// One persistent CTA per SM.  Warps 0-3 and 4-7 take the frame tiles (128
// frames, one per thread) in turn and write their split operand rows to
// shared memory in the 128-byte swizzle of the MMA descriptors: no 16-bit
// frame copy goes through HBM.  Two sets of eight epilogue warps (two per TMEM
// lane quarter, each for half of the columns) take every other frame tile,
// each set with two 128-column TMEM accumulators and a warp that issues its
// MMAs.  At the end of a tile one of the two warps of a quarter, in turn,
// takes the other's values and settles the frames.  Rows, accumulators and
// barriers of a set's tiles are never shared with the other set (tile u
// belongs to set u mod 2, converter half u mod 2 and row slot u mod NS with NS
// even), so every barrier sees its phases in order however far the sets
// drift apart.  The centers are loaded once (TMA) and stay in shared memory.
// Center sets that do not fit are taken in several launches that carry the
// three values per frame in the workspace.
//
// What bounds it: a scan of 32 columns takes 64 cycles of a quarter's ALU
// pipe (maxima, compares and selects issue at half rate), 256 per 128 x 128
// tile, and the kernel takes about 460: an accumulator's way from its release
// to the next full one (300-450 cycles until the MMA warp sees the release,
// 900-1,500 from the first MMA to the waiting warps) is longer than the scans
// of the 512 columns that TMEM holds.  Measured per 1,000,000 x 10 frames, k =
// 1024, in us: 169 in this form; 210 with one epilogue warp per quarter and
// set; 191 with one 256-column accumulator per set; 231 with four sets of one
// 128-column accumulator behind one MMA warp; groups of 16 columns (26
// instead of 36 instructions per chunk) 173.  The tensor-core form with
// stored FP16 rows, candidate lists and re-checks: 498 + 39.
#include <algorithm>
#include <cmath>
#include <cstdlib>

#include <cuda_fp16.h>

#include "km_common.cuh"
#include "km_internal.h"
#include "tc_ptx.cuh"

namespace km {

namespace {

constexpr int kSmMaxD = 31;
constexpr int kSmConvWarps = 8;
constexpr int kSmN = 128;                   // columns per MMA tile
constexpr int kSmPanel = 128 * 128;         // bytes of 128 rows x 64 FP16 columns
constexpr int kSmSmem = 232448;
// Lists from which eight frames share a warp: the 4,864 warps then have about
// eight each (10,000 frames beside the segment sums of 4.3M x 10, k = 1000: 8 us
// per iteration more in eights).
constexpr int kSmFew = 32768;
// The second pass.  It is launched from n k (3 d + 2) = 2e10 on, where the 4 us
// of an empty launch are at most 1.5% of the call (1M x 10, k = 1000 270 us),
// and goes over lists whose comparison with all centers takes longer than it
// does (list k (3 d + 2) = 1e9, about 50 us).  us per assignment with every
// center twice, a warp per listed frame / eight / a second pass (and by the exact
// kernel or the general pass): 1M x 2, k = 500 698 / 470 / 284 (370); 1M x 10, k
// = 1000 3613 / 1436 / 599 (3908); 1M x 16, k = 2000 14,055 / 4231 / 2319 (4626).
// Frames on a lattice of spacing 0.5: 1M x 16, k = 2000 2229 -> 1118 (1909).
constexpr double kSmTwiceWork = 2e10, kSmTwiceList = 1e9;
constexpr size_t kSmBitsMax = size_t(256) << 20;
int sm_twice_few(int d, int k) { return std::max(kSmFew, (int)(kSmTwiceList / ((double)k * (3 * d + 2)))); }

// 64-column panels per operand row: 4 columns per feature and 4 for the norm.
__host__ __device__ constexpr int sm_panels(int d) { return 4 * (d + 1) > 64 ? 2 : 1; }
__host__ __device__ constexpr int sm_ksteps(int d) { return (d + 4) / 4; }  // ceil(4 (d + 1) / 16)
__host__ __device__ constexpr int sm_slots(int panels) { return panels == 1 ? 4 : 2; }  // frame tiles in flight
constexpr int kSmSets = 2;   // epilogue sets
constexpr int kSmBufs = 2;   // accumulators per set
constexpr int kSmThreads = (kSmConvWarps + 9 * kSmSets) * 32;

int sm_kpad(int k) { return (k + kSmN - 1) / kSmN * kSmN; }

struct SmParams {
    const float *X;
    int64_t n;
    int d, k;
    int ct0, n_ct;       // center tiles of this launch
    int ksteps;
    int first, last;     // first / last launch over the centers
    float e_coef, g_ratio, norm_inflate;
    const float *shift;
    const uint32_t *scal;
    const float *cg;     // centers by groups of eight: [group][feature][8]
    float *state;        // (m1, m2, group) per frame between launches
    int32_t *labels;
    int32_t *label_counts;
    int32_t *full_frames;  // listed frames; the second pass goes over them
    float *full_thr;       // the thresholds of the first `cap` of them (NaN: none)
    int64_t cap;
    int few;               // no second pass over lists of this many
    uint8_t *bits;         // the second pass: bit q of byte t of a frame: group 8 t + q reaches its threshold
    int bit_row;           // bytes per frame
    int32_t *counters;
    uint32_t *err;
};

// A read-only load that stays where it is written (the compiler may move plain
// ones down to their use, and the wait for memory with them).
__device__ __forceinline__ float ldg_pinned(const float *p) {
    float v;
    asm volatile("ld.global.nc.f32 %0, [%1];" : "=f"(v) : "l"(p));
    return v;
}

// tcgen05.wait::ld that the loaded registers pass through, so that no use of
// them can be scheduled before it.
__device__ __forceinline__ void tmem_wait_ld32(uint32_t (&r)[32]) {
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]),
                   "+r"(r[8]), "+r"(r[9]), "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]),
                   "+r"(r[15]), "+r"(r[16]), "+r"(r[17]), "+r"(r[18]), "+r"(r[19]), "+r"(r[20]), "+r"(r[21]),
                   "+r"(r[22]), "+r"(r[23]), "+r"(r[24]), "+r"(r[25]), "+r"(r[26]), "+r"(r[27]), "+r"(r[28]),
                   "+r"(r[29]), "+r"(r[30]), "+r"(r[31])
                 :
                 : "memory");
}

struct Best2 {
    float m1, m2;  // largest group maximum; largest outside that group
    int group;
};

// 32 accumulator columns from column j0 on; MASK: columns >= k count as -inf.
template <bool MASK>
__device__ __forceinline__ void sm_scan(const uint32_t (&r)[32], int j0, int k, Best2 &b) {
    float v[32];
#pragma unroll
    for (int c = 0; c < 32; ++c) {
        v[c] = __uint_as_float(r[c]);
        if (MASK && j0 + c >= k) v[c] = __int_as_float(0xff800000);
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const float *w = v + 8 * q;
        const float g = max3f(max3f(w[0], w[1], w[2]), max3f(w[3], w[4], w[5]), fmaxf(w[6], w[7]));
        b.m2 = fmaxf(b.m2, fminf(b.m1, g));
        if (g > b.m1) b.group = (j0 >> 3) + q;
        b.m1 = fmaxf(b.m1, g);
    }
}

// Bit q: group q of the 32 columns reaches thr (a NaN threshold: none does).
template <bool MASK>
__device__ __forceinline__ uint32_t sm_reach(const uint32_t (&r)[32], int j0, int k, float thr) {
    uint32_t m = 0u;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        float w[8];
#pragma unroll
        for (int c = 0; c < 8; ++c) {
            w[c] = __uint_as_float(r[8 * q + c]);
            if (MASK && j0 + 8 * q + c >= k) w[c] = __int_as_float(0xff800000);
        }
        const float g = max3f(max3f(w[0], w[1], w[2]), max3f(w[3], w[4], w[5]), fmaxf(w[6], w[7]));
        if (g >= thr) m |= 1u << q;
    }
    return m;
}

__device__ __forceinline__ uint32_t half_bits(__half a, __half b) {
    const __half2 h = __halves2half2(a, b);
    uint32_t w;
    memcpy(&w, &h, 4);
    return w;
}

// DP: features padded to 4, 8, 12, 16 or 32 (registers).  TWICE: the second
// pass, over the first `cap` listed frames.
template <int DP, bool TWICE>
__global__ void __launch_bounds__(kSmThreads, 1)
    small_assign_kernel(const __grid_constant__ CUtensorMap tmB, const SmParams p) {
    constexpr int PANELS = DP > 16 ? 2 : 1;  // DP = 16 covers d <= 15
    constexpr int NS = sm_slots(PANELS);
    constexpr int SETS = kSmSets;
    constexpr int BUFS = kSmBufs;
    // the MMA warps first: the scheduler prefers older warps, and theirs is
    // the shortest and most waited-for work
    constexpr int kConvWarp = SETS, kEpiWarp = SETS + kSmConvWarps;
    extern __shared__ uint8_t sm_raw[];
    uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(sm_raw) + 1023) & ~uintptr_t(1023));
    uint8_t *sA = smem;
    uint8_t *sB = sA + NS * PANELS * kSmPanel;
    float4 *fpar = reinterpret_cast<float4 *>(sB + p.n_ct * PANELS * kSmPanel);  // [slot][128]
    float *shift = reinterpret_cast<float *>(fpar + NS * 128);                   // [32]
    float *xch = shift + 32;  // [set][tile parity][m1, m2, group][128]: a tile's values from half to half
    uint64_t *bars = reinterpret_cast<uint64_t *>(xch + SETS * 2 * 3 * 128);
    uint64_t *a_full = bars;            // NS
    uint64_t *a_empty = a_full + NS;    // NS
    uint64_t *acc_full = a_empty + NS;  // [set][buffer]
    uint64_t *acc_empty = acc_full + 4;
    uint64_t *drain = acc_empty + 4;
    uint64_t *x_full = drain + 1;       // [set][tile parity][quarter]
    uint64_t *b_full = x_full + SETS * 8;  // n_ct
    uint32_t *tmem_holder = reinterpret_cast<uint32_t *>(b_full + 16);
    volatile uint32_t *abort_flag = tmem_holder + 1;

    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    int64_t rows = p.n;
    if (TWICE) {
        rows = p.counters[1];
        // (a center that FP16 cannot encode, a NaN, leaves no thresholds)
        if (rows <= p.few || !(__uint_as_float(p.scal[kSmallHcMax]) < __int_as_float(0x7f800000))) return;
        rows = min(rows, p.cap);
    }
    const int64_t n_tiles = (rows + 127) / 128;
    if (TWICE && blockIdx.x >= n_tiles) return;
    // This CTA's tiles are blockIdx.x + u gridDim.x, u < nt.
    const int nt = (int)((n_tiles - blockIdx.x + gridDim.x - 1) / gridDim.x);

    if (threadIdx.x < 32) shift[threadIdx.x] = (int)threadIdx.x < p.d ? p.shift[threadIdx.x] : 0.0f;
    if (threadIdx.x == 0) {
        for (int s = 0; s < NS; ++s) {
            mbar_init(&a_full[s], 4);
            mbar_init(&a_empty[s], 1 + 8);  // the MMAs, the set's epilogue warps (fpar)
        }
        for (int b = 0; b < 4; ++b) {
            mbar_init(&acc_full[b], 1);
            mbar_init(&acc_empty[b], 8);
        }
        for (int b = 0; b < SETS * 8; ++b) mbar_init(&x_full[b], 1);
        mbar_init(drain, SETS);
        for (int t = 0; t < p.n_ct; ++t) mbar_init(&b_full[t], 1);
        *abort_flag = 0;
        fence_mbar_init();
    }
    if (warp == 0) {
        tmem_alloc(tmem_holder, 512);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_holder;
    bool ok = true;

    if (warp >= kConvWarp && warp < kEpiWarp) {
        // ---------------- operand rows ----------------
        const int half = (warp - kConvWarp) >> 2;  // tiles half, half + 2, ...
        const int r = (threadIdx.x - kConvWarp * 32) & 127;
        const float sc = __uint_as_float(p.scal[kScale]);
        const float inv_sc = 1.0f / sc;  // exact: a power of two
        const float sc_max = __uint_as_float(p.scal[kSmallCmax]);
        const float hc_max = __uint_as_float(p.scal[kSmallHcMax]);
        const uint32_t one2 = half_bits(__float2half_rn(1.0f), __float2half_rn(1.0f));
        const uint32_t one1 = half_bits(__float2half_rn(1.0f), __float2half_rn(0.0f));
        float x[DP];
        auto load = [&](int u) {
            int64_t i = ((int64_t)blockIdx.x + (int64_t)u * gridDim.x) * 128 + r;
            if (u >= nt || i >= rows) i = 0;
            if (TWICE) i = p.full_frames[i];
            const float *src = p.X + i * p.d;
#pragma unroll
            for (int f = 0; f < DP; ++f)
                if (f < p.d) x[f] = ldg_pinned(src + f);
        };
        load(half);
        for (int u = half; u < nt; u += 2) {
            const int slot = u % NS;
            const bool valid = ((int64_t)blockIdx.x + (int64_t)u * gridDim.x) * 128 + r < rows;
            // ||x||^2 of the split values by a Kahan sum (the distance bound
            // allows 8 u for it); the two norms of bounds by plain sums
            // inflated by norm_inflate.
            uint32_t w[DP];
            float hs = 0.0f, hc = 0.0f, s2 = 0.0f, e2 = 0.0f;
#pragma unroll
            for (int f = 0; f < DP; ++f) {
                w[f] = 0u;
                if (f < p.d) {
                    const float a = valid ? __fsub_rn(x[f], shift[f]) : 0.0f;
                    const float as = a * sc;
                    const __half h = __float2half_rn(as);
                    const float hf = __half2float(h);
                    const __half l = __float2half_rn(__fsub_rn(as, hf));
                    const float xt = __fadd_rn(hf, __half2float(l));  // exact
                    const float e = __fsub_rn(xt, as);
                    const float y = __fsub_rn(__fmul_rn(xt, xt), hc);
                    const float t = __fadd_rn(hs, y);
                    hc = __fsub_rn(__fsub_rn(t, hs), y);
                    hs = t;
                    s2 = __fmaf_rn(a, a, s2);
                    e2 = __fmaf_rn(e, e, e2);
                    w[f] = half_bits(h, l);
                }
            }
            load(u + 2);  // in flight while the rows are written
            const float sx = __fsqrt_ru(__fmul_ru(s2, p.norm_inflate));
            const float hx = __fmul_ru(__fadd_ru(__fsqrt_ru(__fmul_ru(e2, p.norm_inflate)), 1e-30f), inv_sc);
            const float smax = sx + sc_max;
            const float Rmax = __fadd_ru(__fadd_ru(hx, hc_max), __fmul_ru(kCenterEps, smax));
            const float Emax = __fmul_ru(p.e_coef, __fmul_ru(smax, smax));
            ok = mbar_wait(&a_empty[slot], ((u / NS) & 1) ^ 1u);
            ok = __all_sync(0xffffffffu, ok) && !__any_sync(0xffffffffu, *abort_flag != 0);
            if (!ok) break;
            fpar[slot * 128 + r] = make_float4(hs, Rmax, Emax, 0.0f);
            uint8_t *row = sA + slot * PANELS * kSmPanel + (r >> 3) * 1024 + (r & 7) * 128;
#pragma unroll
            for (int c = 0; c < DP / 2 + 2; ++c) {  // 16-byte chunks: two features each
                if (c >= 2 * p.ksteps) break;       // columns no K step reads
                uint4 v;
                v.x = v.y = v.z = v.w = 0u;
                if (2 * c < DP) v.x = v.y = w[2 * c < DP ? 2 * c : 0];
                if (2 * c + 1 < DP) v.z = v.w = w[2 * c + 1 < DP ? 2 * c + 1 : 0];
                if (2 * c == p.d) {
                    v.x = one2;
                    v.y = one1;
                }
                if (2 * c + 1 == p.d) {
                    v.z = one2;
                    v.w = one1;
                }
                *reinterpret_cast<uint4 *>(row + (c >> 3) * kSmPanel + (((c & 7) ^ (r & 7)) << 4)) = v;
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(&a_full[slot]);
        }
        if (!ok) {
            atomicOr(p.err, (uint32_t)kDevTimeoutTma);
            *abort_flag = 1;
        }
    } else if (warp < kConvWarp) {
        // ---------------- centers and MMAs ----------------
        const int g = warp;  // the set
        const uint32_t idesc = make_idesc(128, kSmN);
        const uint64_t a0 = sw128_desc(smem_u32(sA));
        const uint64_t b0 = sw128_desc(smem_u32(sB));
        constexpr uint64_t kPanelStep = kSmPanel >> 4;
        if (g == 0 && elect_one()) {
            for (int t = 0; t < p.n_ct; ++t) {
                mbar_arrive_expect_tx(&b_full[t], PANELS * kSmPanel);
#pragma unroll
                for (int q = 0; q < PANELS; ++q)
                    tma_load_2d(sB + (t * PANELS + q) * kSmPanel, &tmB, 64 * q, (p.ct0 + t) * kSmN, &b_full[t]);
            }
        }
        __syncwarp();
        // (ok stays the same in every lane: the waits are agreed by vote)
        uint32_t accq = 0;  // accumulators filled
        for (int u = g; u < nt && ok; u += SETS) {
            ok = __all_sync(0xffffffffu, mbar_wait(&a_full[u % NS], (u / NS) & 1));
            const uint64_t ad = a0 + (uint64_t)((u % NS) * PANELS) * kPanelStep;
            for (int t = 0; t < p.n_ct && ok; ++t) {
                if (u == g) ok = __all_sync(0xffffffffu, mbar_wait(&b_full[t], 0));
                const uint32_t buf = accq % BUFS;
                if (ok)
                    ok = __all_sync(0xffffffffu, mbar_wait(&acc_empty[BUFS * g + buf], ((accq / BUFS) & 1u) ^ 1u));
                if (!ok) break;
                tc_fence_after();
                if (elect_one()) {
                    const uint32_t d_tmem = tmem_base + (BUFS * g + buf) * kSmN;
                    const uint64_t bd = b0 + (uint64_t)(t * PANELS) * kPanelStep;
#pragma unroll
                    for (int s = 0; s < 4 * PANELS; ++s)
                        if (s < p.ksteps)
                            mma_f16(d_tmem, ad + (s >> 2) * kPanelStep + 2 * (s & 3),
                                    bd + (s >> 2) * kPanelStep + 2 * (s & 3), idesc, s != 0);
                    mma_commit(&acc_full[BUFS * g + buf]);
                    if (t == p.n_ct - 1) mma_commit(&a_empty[u % NS]);
                }
                __syncwarp();
                ++accq;
            }
            ok = ok && !__any_sync(0xffffffffu, *abort_flag != 0);
        }
        if (!ok && lane == 0) {
            atomicOr(p.err, (uint32_t)kDevTimeoutMma);
            *abort_flag = 1;
        }
        // Every copy has landed and every MMA is complete before the CTA's
        // shared memory and TMEM go.
        for (int t = 0; t < p.n_ct; ++t) mbar_wait(&b_full[t], 0);
        if (elect_one()) mma_commit(drain);
        __syncwarp();
        mbar_wait(drain, 0);
        __syncwarp();
    } else {
        // ---------------- epilogue ----------------
        const int g = (warp - kEpiWarp) >> 3;
        const int half = ((warp - kEpiWarp) >> 2) & 1;  // columns 64 half .. + 64 of every tile
        const int row = (warp & 3) * 32 + lane;
        const uint32_t lane_off = (uint32_t)((warp & 3) * 32) << 16;
        const float inv_s2 = __uint_as_float(p.scal[kInvScale2]);
        const float s2 = 1.0f / inv_s2;  // exact: a power of two
        const float kNegInf = __int_as_float(0xff800000);
        const float kInf = __int_as_float(0x7f800000);
        uint32_t accq = 0;
        for (int u = g; u < nt && ok; u += SETS) {
            const int slot = u % NS;
            const int64_t i = ((int64_t)blockIdx.x + (int64_t)u * gridDim.x) * 128 + row;
            ok = __all_sync(0xffffffffu, mbar_wait(&a_full[slot], (u / NS) & 1));
            if (!ok) break;
            const float4 fp = fpar[slot * 128 + row];
            __syncwarp();
            if (lane == 0) mbar_arrive(&a_empty[slot]);
            if constexpr (TWICE) {
                const float thr = i < rows ? p.full_thr[i] : kInf;
                for (int t = 0; t < p.n_ct; ++t) {
                    const uint32_t buf = accq % BUFS;
                    ok = __all_sync(0xffffffffu, mbar_wait(&acc_full[BUFS * g + buf], (accq / BUFS) & 1u));
                    if (!ok) break;
                    tc_fence_after();
                    const uint32_t base = tmem_base + lane_off + (BUFS * g + buf) * kSmN + 64 * half;
                    const int j0 = (p.ct0 + t) * kSmN + 64 * half;
                    uint32_t r[32];
                    tmem_ld32(base, r);
                    tmem_wait_ld32(r);
                    uint32_t m = sm_reach<true>(r, j0, p.k, thr);
                    tmem_ld32(base + 32, r);
                    tmem_wait_ld32(r);
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&acc_empty[BUFS * g + buf]);
                    m |= sm_reach<true>(r, j0 + 32, p.k, thr) << 4;
                    if (i < rows) p.bits[i * p.bit_row + 2 * (p.ct0 + t) + half] = (uint8_t)m;
                    ++accq;
                }
                if (__any_sync(0xffffffffu, *abort_flag != 0)) ok = false;
                continue;
            }
            Best2 b{kNegInf, kNegInf, 0};
            if (!p.first && half == 0 && i < p.n) {
                b.m1 = p.state[3 * i];
                b.m2 = p.state[3 * i + 1];
                b.group = __float_as_int(p.state[3 * i + 2]);
            }
            for (int t = 0; t < p.n_ct; ++t) {
                const uint32_t buf = accq % BUFS;
                ok = __all_sync(0xffffffffu, mbar_wait(&acc_full[BUFS * g + buf], (accq / BUFS) & 1u));
                if (!ok) break;
                tc_fence_after();
                const uint32_t base = tmem_base + lane_off + (BUFS * g + buf) * kSmN;
                const int j0 = (p.ct0 + t) * kSmN;
                const bool whole = j0 + kSmN <= p.k;
                uint32_t r[32];
                tmem_ld32(base + 64 * half, r);
                tmem_wait_ld32(r);
                if (whole)
                    sm_scan<false>(r, j0 + 64 * half, p.k, b);
                else
                    sm_scan<true>(r, j0 + 64 * half, p.k, b);
                tmem_ld32(base + 64 * half + 32, r);
                tmem_wait_ld32(r);
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(&acc_empty[BUFS * g + buf]);
                if (whole)
                    sm_scan<false>(r, j0 + 64 * half + 32, p.k, b);
                else
                    sm_scan<true>(r, j0 + 64 * half + 32, p.k, b);
                ++accq;
            }
            if (!ok) break;
            // One half hands its values over, the other settles the frames;
            // they take turns, so a buffer is rewritten only after its reader
            // has handed over the tile in between.
            const int par = (u / SETS) & 1;
            float *xc = xch + ((g * 2 + par) * 3) * 128 + row;
            uint64_t *xb = &x_full[(g * 2 + par) * 4 + (warp & 3)];
            if (half != par) {
                xc[0] = b.m1;
                xc[128] = b.m2;
                xc[256] = __int_as_float(b.group);
                __syncwarp();
                if (lane == 0) mbar_arrive(xb);
                continue;
            }
            ok = __all_sync(0xffffffffu, mbar_wait(xb, (u / (2 * SETS)) & 1));
            if (!ok) break;
            const float o1 = xc[0], o2 = xc[128];
            if (o1 > b.m1) b.group = __float_as_int(xc[256]);
            b.m2 = fmaxf(fmaxf(b.m2, o2), fminf(b.m1, o1));
            b.m1 = fmaxf(b.m1, o1);
            if (!p.last) {
                if (i < p.n) {
                    p.state[3 * i] = b.m1;
                    p.state[3 * i + 1] = b.m2;
                    p.state[3 * i + 2] = __int_as_float(b.group);
                }
                continue;
            }
            bool need_full = false;
            float thr = 0.0f;  // of a listed frame
            if (i < p.n) {
                // The exact distances of the best group's centers.
                float acc[8];
#pragma unroll
                for (int q = 0; q < 8; ++q) acc[q] = 0.0f;
                const float *cg = p.cg + (int64_t)b.group * p.d * 8;
#pragma unroll
                for (int f = 0; f < DP; ++f) {
                    if (f < p.d) {
                        const float xf = __ldg(p.X + i * p.d + f);
                        float c[8];
                        ldg_f32x8(cg + 8 * f, c);
#pragma unroll
                        for (int q = 0; q < 8; ++q) acc[q] = __fadd_rn(acc[q], sq_term(xf, c[q]));
                    }
                }
                float best = kInf;
                int label = 0;
#pragma unroll
                for (int q = 0; q < 8; ++q)
                    if (acc[q] < best) {  // the centers beyond k lie at infinity
                        best = acc[q];
                        label = b.group * 8 + q;
                    }
                thr = window_threshold(b.m1, fp.x, inv_s2, s2, fp.z, fp.y, __fadd_ru(fp.y, 1e-18f), p.g_ratio);
                const bool finite = b.m1 > kNegInf && b.m1 < kInf && fp.y < kInf && fp.z < kInf && fp.x < kInf &&
                                    best < kInf;
                need_full = !finite || !(b.m2 < thr);
                if (!finite) thr = __int_as_float(0x7fc00000);
                p.labels[i] = label;  // provisional when the frame is re-checked
                if (p.label_counts) atomicAdd(&p.label_counts[label], 1);
            }
            const unsigned m_full = __ballot_sync(0xffffffffu, need_full);
            if (m_full) {
                const int leader = __ffs(m_full) - 1;
                int at = 0;
                if (lane == leader) at = atomicAdd(&p.counters[1], __popc(m_full));
                at = __shfl_sync(0xffffffffu, at, leader) + __popc(m_full & ((1u << lane) - 1u));
                if (need_full) {
                    p.full_frames[at] = (int32_t)i;
                    if (at < p.cap) p.full_thr[at] = thr;
                }
            }
            if (__any_sync(0xffffffffu, *abort_flag != 0)) ok = false;
        }
        if (!ok && lane == 0) {
            atomicOr(p.err, (uint32_t)kDevTimeoutEpi);
            *abort_flag = 1;
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0) {
        tc_fence_after();
        tmem_dealloc(tmem_base, 512);
    }
}

// The exact distances of the listed frames: every distance in feature order
// with every operation rounded on its own, the lexicographic (distance, index)
// minimum, label 0 when no distance is finite.  A changed label is written, or
// listed (flips non-null).
//   * A frame of a long list with bits: a thread, over its groups' eight
//     centers at a time (ascending, so the first minimum has the lowest index).
//   * Others are compared with all centers by a warp whose lanes own centers
//     (the grouped copy gives each eight of them 32 consecutive bytes per
//     feature): one at a time, or in a long list up to eight together, so that
//     each center value read serves eight distances.
// 1M x 2, k = 500: frames with bits, a warp each 523 us the call, a thread each
// 284; a NaN center (no bits), a warp per frame 907, per eight 420.
constexpr int kFullWarps = 8;
template <int DP>
__global__ void __launch_bounds__(kFullWarps * 32, DP > 16 ? 2 : 4) small_full_kernel(
    const float *__restrict__ X, int d, int k, const float *__restrict__ cg, const int32_t *__restrict__ frames,
    const int32_t *__restrict__ n_dev, int64_t n_max, const float *__restrict__ thr, const uint16_t *__restrict__ bits,
    int bit_row, int64_t cap, int few, int32_t *__restrict__ labels, unsigned long long *flipped,
    int32_t *__restrict__ flips, int32_t *__restrict__ n_flips, int64_t max_flips) {
    __shared__ __align__(16) float xs_s[kFullWarps][kSmMaxD * 8];  // [feature][frame]
    __shared__ int32_t id_s[kFullWarps][32];                       // frames of a unit without bits
    int64_t n = *n_dev;
    if (n > n_max) n = n_max;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const bool lng = n > kSmFew;
    if (n <= few) cap = 0;  // no second pass, no bits
    const int unit = !lng ? 1 : cap > 0 ? 32 : 8;
    const int64_t nw = (int64_t)gridDim.x * kFullWarps;
    const float kInf = __int_as_float(0x7f800000);
    auto settle = [&](int64_t i, int label) {
        const int before = labels[i];
        if (before == label) return;
        if (flipped) atomicAdd(flipped, 1ull);
        if (flips) {
            const int slot = atomicAdd(n_flips, 1);
            if (slot < max_flips) {
                flips[3 * (int64_t)slot] = (int32_t)i;
                flips[3 * (int64_t)slot + 1] = before;
                flips[3 * (int64_t)slot + 2] = label;
            }
        } else {
            labels[i] = label;
        }
    };
    auto load = [&](int64_t i, float (&x)[DP]) {
#pragma unroll
        for (int f = 0; f < DP; ++f) x[f] = f < d ? __ldg(X + i * d + f) : 0.0f;
    };
    const float *c_lane = cg + (int64_t)(lane >> 3) * d * 8 + (lane & 7);  // the first 32 centers
    auto one = [&](int64_t i) {
        float x[DP], bd = kInf;
        load(i, x);
        int bj = 0;
        const float *c = c_lane;
#pragma unroll 2
        for (int j0 = 0; j0 < k; j0 += 32, c += 32 * d) {
            float acc = 0.0f;
#pragma unroll
            for (int f = 0; f < DP; ++f)
                if (f < d) acc = __fadd_rn(acc, sq_term(x[f], __ldg(c + 8 * f)));
            if (acc < bd) {  // the centers beyond k lie at infinity
                bd = acc;
                bj = j0 + lane;
            }
        }
        warp_argmin(bd, bj);
        if (lane == 0) settle(i, bj);
    };
    float *xs = xs_s[warp];
    auto eight = [&](const int32_t *ids, int m) {  // m frames, two to eight
        for (int t = lane; t < 8 * d; t += 32) {
            const int q = t / d, f = t - q * d;
            xs[f * 8 + q] = q < m ? __ldg(X + (int64_t)ids[q] * d + f) : 0.0f;
        }
        __syncwarp();
        float bd[8];
        int bj[8];
#pragma unroll
        for (int q = 0; q < 8; ++q) bd[q] = kInf, bj[q] = 0;
        const float *c = c_lane;
#pragma unroll 2
        for (int j0 = 0; j0 < k; j0 += 32, c += 32 * d) {
            float acc[8];
#pragma unroll
            for (int q = 0; q < 8; ++q) acc[q] = 0.0f;
#pragma unroll
            for (int f = 0; f < DP; ++f) {
                if (f >= d) break;
                const float cf = __ldg(c + 8 * f);
                const float4 a = *reinterpret_cast<const float4 *>(xs + 8 * f);
                const float4 b = *reinterpret_cast<const float4 *>(xs + 8 * f + 4);
                const float xq[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
#pragma unroll
                for (int q = 0; q < 8; ++q) acc[q] = __fadd_rn(acc[q], sq_term(xq[q], cf));
            }
#pragma unroll
            for (int q = 0; q < 8; ++q)
                if (acc[q] < bd[q]) {
                    bd[q] = acc[q];
                    bj[q] = j0 + lane;
                }
        }
        int label = 0;
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            warp_argmin(bd[q], bj[q]);
            if (lane == q) label = bj[q];
        }
        if (lane < m) settle(ids[lane], label);
        __syncwarp();  // xs is rewritten by the next eight
    };
    for (int64_t e0 = ((int64_t)blockIdx.x * kFullWarps + warp) * unit; e0 < n; e0 += nw * unit) {
        if (!lng) {
            one(frames[e0]);
            continue;
        }
        const int64_t e = e0 + lane;
        bool todo = lane < unit && e < n;
        const int64_t i = todo ? frames[e] : 0;
        if (todo && e < cap && thr[e] == thr[e]) {
            float x[DP], bd = kInf;
            load(i, x);
            int bj = 0;
            for (int t = 0; t < bit_row; ++t) {
                for (uint32_t v = bits[e * bit_row + t]; v; v &= v - 1u) {
                    todo = false;
                    const int g = 16 * t + __ffs(v) - 1;
                    const float *c = cg + (int64_t)g * d * 8;
                    float acc[8];
#pragma unroll
                    for (int q = 0; q < 8; ++q) acc[q] = 0.0f;
#pragma unroll
                    for (int f = 0; f < DP; ++f) {
                        if (f < d) {
                            float w[8];
                            ldg_f32x8(c + 8 * f, w);
#pragma unroll
                            for (int q = 0; q < 8; ++q) acc[q] = __fadd_rn(acc[q], sq_term(x[f], w[q]));
                        }
                    }
#pragma unroll
                    for (int q = 0; q < 8; ++q)
                        if (acc[q] < bd) {
                            bd = acc[q];
                            bj = 8 * g + q;
                        }
                }
            }
            if (!todo) settle(i, bj);  // (the best center reaches its threshold; else all are compared)
        }
        const unsigned rest = __ballot_sync(0xffffffffu, todo);
        const int cnt = __popc(rest);
        int32_t *ids = id_s[warp];
        if (todo) ids[__popc(rest & ((1u << lane) - 1u))] = (int32_t)i;
        __syncwarp();
        for (int q = 0; q < cnt; q += 8) {
            if (cnt - q > 1)
                eight(ids + q, min(8, cnt - q));
            else
                one(ids[q]);
        }
        __syncwarp();  // ids are rewritten
    }
}

// The centers' operand rows and their grouped float copy: a warp per center,
// lane f for feature f (four columns), lane d for the norm.  kSmallCmax and kSmallHcMax
// get the largest bounds of ||c'|| and of the split's rounding error; a norm
// that FP16 cannot encode poisons them (every frame is then re-checked).
// Rows and groups beyond k: zero operands, centers at infinity.
__global__ void small_prep_centers_kernel(const float *__restrict__ C, int k, int kpad, int d, int panels,
                                          const float *__restrict__ shift, uint32_t *__restrict__ scal,
                                          __half *__restrict__ ch, float *__restrict__ cg, float norm_inflate) {
    const int lane = threadIdx.x & 31;
    const int nw = (int)((gridDim.x * blockDim.x) >> 5);
    const float sc = __uint_as_float(scal[kScale]);
    const float inv_sc = 1.0f / sc;
    for (int j = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5); j < kpad; j += nw) {
        const bool real = j < k;
        float a = 0.0f, xt = 0.0f, e = 0.0f;
        uint2 w = make_uint2(0u, 0u);
        if (lane < d) {
            const float c = real ? C[(int64_t)j * d + lane] : __int_as_float(0x7f800000);
            cg[((int64_t)(j >> 3) * d + lane) * 8 + (j & 7)] = c;
            if (real) {
                a = __fsub_rn(c, shift[lane]);
                const float as = a * sc;
                const __half h = __float2half_rn(as);
                const float hf = __half2float(h);
                const __half l = __float2half_rn(__fsub_rn(as, hf));
                xt = __fadd_rn(hf, __half2float(l));  // exact
                e = __fsub_rn(xt, as);
                w.x = half_bits(h, h);
                w.y = half_bits(l, l);
            }
        }
        double h2 = (double)xt * (double)xt, s2 = (double)a * (double)a, e2 = (double)e * (double)e;
        for (int off = 16; off > 0; off >>= 1) {
            h2 += __shfl_xor_sync(0xffffffffu, h2, off);
            s2 += __shfl_xor_sync(0xffffffffu, s2, off);
            e2 += __shfl_xor_sync(0xffffffffu, e2, off);
        }
        if (lane == d && real) {
            const double val = -0.5 * h2;
            const __half n1 = __float2half_rn((float)val);
            const double r1 = val - (double)__half2float(n1);
            const __half n2 = __float2half_rn((float)r1);
            const __half n3 = __float2half_rn((float)(r1 - (double)__half2float(n2)));
            w.x = half_bits(n1, n2);
            w.y = half_bits(n3, __float2half_rn(0.0f));
            const float nrm = __fsqrt_ru(__fmul_ru((float)s2, norm_inflate));
            const float hc = __fmul_ru(__fadd_ru(__fsqrt_ru(__fmul_ru((float)e2, norm_inflate)), 1e-30f), inv_sc);
            const bool fine = fabs(val) < 65504.0 && nrm == nrm && hc == hc;
            atomicMax(&scal[kSmallCmax], fine ? __float_as_uint(nrm) : 0x7f800000u);
            atomicMax(&scal[kSmallHcMax], fine ? __float_as_uint(hc) : 0x7f800000u);
        }
        if (lane < 16 * panels) reinterpret_cast<uint2 *>(ch)[(int64_t)j * 16 * panels + lane] = w;
    }
}

int sm_env() {
    const char *e = std::getenv("KM_TC_SMALL");
    return !e ? -1 : e[0] == '0' ? 0 : 1;
}

size_t sm_fixed_smem(int panels) {
    const int ns = sm_slots(panels);
    return 1024 + (size_t)ns * panels * kSmPanel + (size_t)ns * 128 * 16 + 32 * 4 + kSmSets * 2 * 3 * 128 * 4 +
           (2 * ns + 9 + 8 * kSmSets + 16) * 8 + 16;
}

// Center tiles that one launch keeps in shared memory.
int sm_tiles_fit(int panels) {
    return (int)std::min<size_t>(16, (kSmSmem - sm_fixed_smem(panels)) / ((size_t)panels * kSmPanel));
}

}  // namespace

bool small_shape_ok(int d, int k) {
    (void)k;
    return d >= 1 && d <= kSmMaxD;
}

bool small_allowed() { return sm_env() != 0; }
bool small_forced() { return sm_env() == 1; }

size_t small_centers_elems(int d, int k) { return (size_t)sm_kpad(k) * 64 * sm_panels(d); }
size_t small_groups_floats(int d, int k) { return (size_t)sm_kpad(k) * d; }

int small_prepare_centers(const float *C, int d, int k, TcBuffers &b, cudaStream_t s) {
    KM_CUDA(cudaMemsetAsync(b.scal + kSmallCmax, 0, 2 * sizeof(uint32_t), s));
    const int kpad = sm_kpad(k);
    const float inflate = 1.0f + (float)(d + 8) * 5.9604645e-8f + 1e-6f;
    small_prep_centers_kernel<<<(unsigned)std::min((kpad + 7) / 8, num_sms() * 8), 256, 0, s>>>(
        C, k, kpad, d, sm_panels(d), b.shift, b.scal, static_cast<__half *>(b.sch), b.scg, inflate);
    KM_CUDA(cudaGetLastError());
    return KM_OK;
}

namespace {

int sm_bit_row(int k) { return 2 * (sm_kpad(k) / kSmN); }

// Launches over the centers.
int sm_passes(int d, int k) {
    const int tiles = sm_kpad(k) / kSmN, fit = sm_tiles_fit(sm_panels(d));
    return (tiles + fit - 1) / fit;
}

// Frames that a second pass takes at most (0: none is made).
int64_t sm_twice_cap(int64_t n, int d, int k) {
    if (n <= sm_twice_few(d, k) || (double)n * k * (3 * d + 2) < kSmTwiceWork) return 0;
    return std::min<int64_t>(n, (int64_t)(kSmBitsMax / (size_t)(sm_bit_row(k) + 4)));
}

size_t carve_lists(void *ws, int64_t n, int d, int k, TcBuffers &b) {
    Carver c(ws);
    const size_t nn = n > 0 ? n : 1;
    b.counters = c.take<int32_t>(kTcStatusWords);
    b.flipped = reinterpret_cast<unsigned long long *>(b.counters + 4);
    b.err = reinterpret_cast<uint32_t *>(b.counters + 6);
    b.full_frames = c.take<int32_t>(nn);
    b.pair_lo = sm_passes(d, k) > 1 ? c.take<float>(3 * nn) : nullptr;
    b.wide_cap = sm_twice_cap(n, d, k);
    b.wide_thr = b.wide_cap > 0 ? c.take<float>(b.wide_cap) : nullptr;
    b.wide_bits = b.wide_cap > 0 ? c.take<uint32_t>(((size_t)b.wide_cap * sm_bit_row(k) + 3) / 4) : nullptr;
    return c.bytes();
}

}  // namespace

size_t small_lists_ws_size(int64_t n, int d, int k) {
    TcBuffers b;
    return carve_lists(nullptr, n, d, k, b);
}

void small_carve_lists(void *ws, int64_t n, int d, int k, TcBuffers &b) { carve_lists(ws, n, d, k, b); }

namespace {

template <int DP, bool TWICE>
int launch_small_dp(const CUtensorMap &tmB, const SmParams &p, unsigned grid, size_t smem, cudaStream_t s) {
    static bool attr_done[kDeviceSlots] = {};
    const int dev = current_device();
    if (dev < 0 || dev >= kDeviceSlots || !attr_done[dev]) {
        KM_CUDA(cudaFuncSetAttribute(small_assign_kernel<DP, TWICE>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     kSmSmem));
        if (dev >= 0 && dev < kDeviceSlots) attr_done[dev] = true;
    }
    small_assign_kernel<DP, TWICE><<<grid, kSmThreads, smem, s>>>(tmB, p);
    KM_CUDA(cudaGetLastError());
    return KM_OK;
}

// A pass over all center tiles, `per` at a time.
template <bool TWICE>
int launch_small(const CUtensorMap &tmB, SmParams p, int tiles, int per, unsigned grid, cudaStream_t s) {
    const int panels = sm_panels(p.d);
    for (int t = 0; t < tiles; t += per) {
        p.ct0 = t;
        p.n_ct = std::min(per, tiles - t);
        p.first = t == 0;
        p.last = t + p.n_ct == tiles;
        // at least 120 KB: one CTA per SM (it takes all of TMEM)
        const size_t smem = std::max<size_t>(120 * 1024, sm_fixed_smem(panels) + (size_t)p.n_ct * panels * kSmPanel);
        if (p.d <= 4)
            KM_TRY((launch_small_dp<4, TWICE>(tmB, p, grid, smem, s)));
        else if (p.d <= 8)
            KM_TRY((launch_small_dp<8, TWICE>(tmB, p, grid, smem, s)));
        else if (p.d <= 12)
            KM_TRY((launch_small_dp<12, TWICE>(tmB, p, grid, smem, s)));
        else if (p.d <= 15)
            KM_TRY((launch_small_dp<16, TWICE>(tmB, p, grid, smem, s)));
        else
            KM_TRY((launch_small_dp<32, TWICE>(tmB, p, grid, smem, s)));
    }
    return KM_OK;
}

template <int DP>
void launch_small_full(const float *X, int64_t n, int d, int k, const TcBuffers &b, int64_t cap, int32_t *labels,
                       const FlipList *fl, unsigned grid, cudaStream_t s) {
    small_full_kernel<DP><<<grid, kFullWarps * 32, 0, s>>>(
        X, d, k, b.scg, b.full_frames, b.counters + 1, n, b.wide_thr, reinterpret_cast<const uint16_t *>(b.wide_bits),
        sm_bit_row(k) / 2, cap, sm_twice_few(d, k), labels, b.flipped, fl ? fl->rows : nullptr, fl ? fl->count : nullptr, fl ? fl->cap : 0);
}

}  // namespace

int small_assign(const float *X, int64_t n, int d, int k, int32_t *labels, TcBuffers &b, cudaStream_t s,
                 ProfEvents *prof, cudaStream_t side, cudaEvent_t fork, const FlipList *fl,
                 int32_t *label_counts) {
    if (n == 0) return KM_OK;
    const int panels = sm_panels(d);
    const int kpad = sm_kpad(k);
    CUtensorMap tmB;
    EncodeTiledFn enc = get_encode();
    if (!enc || !device_is_sm10x()) {
        set_error("no tensor-core kernel for d=%d k=%d on this device", d, k);
        return KM_ERR_UNSUPPORTED;
    }
    cuuint64_t dims[2] = {(cuuint64_t)(64 * panels), (cuuint64_t)kpad};
    cuuint64_t strides[1] = {(cuuint64_t)(128 * panels)};
    cuuint32_t box[2] = {64, kSmN};
    cuuint32_t estr[2] = {1, 1};
    const CUresult cr = enc(&tmB, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, b.sch, dims, strides, box, estr,
                            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                            CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (cr != CUDA_SUCCESS) {
        set_error("cuTensorMapEncodeTiled failed (%d) for %d x %d", (int)cr, kpad, 64 * panels);
        return KM_ERR_CUDA;
    }
    KM_TRY(tc_clear_status(b, s));

    const double u = 5.9604644775390625e-08;  // 2^-24
    SmParams p;
    p.X = X;
    p.n = n;
    p.d = d;
    p.k = k;
    p.ksteps = sm_ksteps(d);
    // Accumulation as in assign_tc.cu (2^-21 per 16-term step), the split
    // operands' norms, the rounding of ||x||^2, of the norm's three parts
    // and of the epilogue (10 u).
    p.e_coef = (float)(((p.ksteps + 1) * std::ldexp(1.0, -21) * 1.006 + 10.0 * u) * 1.01);
    const double gm = (d + 2) * u / (1.0 - (d + 2) * u) * 1.01;
    const float g_lo = (float)((1.0 - gm) * (1.0 - 4.0 * u)), g_hi = (float)((1.0 + gm) * (1.0 + 4.0 * u));
    p.g_ratio = std::nextafter((float)(std::sqrt((double)g_hi / (double)g_lo) * (1.0 + std::ldexp(1.0, -19))), INFINITY);
    p.norm_inflate = 1.0f + (float)(d + 8) * 5.9604645e-8f + 1e-6f;
    p.shift = b.shift;
    p.scal = b.scal;
    p.cg = b.scg;
    p.state = b.pair_lo;  // three floats per frame
    p.labels = labels;
    p.label_counts = label_counts;
    p.full_frames = b.full_frames;
    p.full_thr = b.wide_thr;
    // (beside the caller's next work a list of up to a sixteenth of the frames
    // costs nothing, and a second pass before it does: 4.3M x 10, k = 1000, with
    // 1% listed 1.10 -> 1.12 ms per Lloyd iteration)
    p.cap = side ? 0 : b.wide_cap;
    p.bits = reinterpret_cast<uint8_t *>(b.wide_bits);
    p.bit_row = sm_bit_row(k);
    p.few = sm_twice_few(d, k);
    p.counters = b.counters;
    p.err = b.err;

    const int tiles = kpad / kSmN;
    const int passes = sm_passes(d, k);
    const int per = (tiles + passes - 1) / passes;
    const int64_t n_tiles = (n + 127) / 128;
    const unsigned grid = (unsigned)std::min<int64_t>(num_sms(), n_tiles);
    if (prof) prof->begin(kProfTc, s);
    KM_TRY(launch_small<false>(tmB, p, tiles, per, grid, s));
    if (p.cap > 0) KM_TRY(launch_small<true>(tmB, p, tiles, per, grid, s));
    if (prof) prof->end(kProfTc, s);
    cudaStream_t r = side ? side : s;
    if (side) {
        KM_CUDA(cudaEventRecord(fork, s));
        KM_CUDA(cudaStreamWaitEvent(side, fork, 0));
    }
    if (prof) prof->begin(kProfFull, r);
    const unsigned fgrid = (unsigned)std::min<int64_t>((n + 7) / 8, (int64_t)num_sms() * 4);
    if (d <= 4)
        launch_small_full<4>(X, n, d, k, b, p.cap, labels, fl, fgrid, r);
    else if (d <= 8)
        launch_small_full<8>(X, n, d, k, b, p.cap, labels, fl, fgrid, r);
    else if (d <= 16)
        launch_small_full<16>(X, n, d, k, b, p.cap, labels, fl, fgrid, r);
    else
        launch_small_full<32>(X, n, d, k, b, p.cap, labels, fl, fgrid, r);
    KM_CUDA(cudaGetLastError());
    if (prof) prof->end(kProfFull, r);
    return KM_OK;
}

}  // namespace km
