// kmpp.cu -- kernel (d): kmeans++ D^2 sampling.
//
// Reference: KMeans(init_strategy='kmeans++', fixed_seed=seed).fit, called at
// pyemma/coordinates/clustering/kmeans.py:211-212,253 (seed rules at
// kmeans.py:146-164).  The first center is a uniformly drawn frame; every
// later center is drawn with probability proportional to D^2(x), the squared
// distance of x to the nearest center chosen so far.
//
// Determinism: D^2 is the exact float32 distance of the assignment kernel.
// Weights are quantised once per run to integers w_i = floor(D^2_i * 2^e)
// with e fixed after the first round so that the sum of all weights stays
// below 2^62; every sum and prefix sum is then exact, so the draw does not
// depend on the reduction order.  Round r draws a 64-bit number u from
// Philox4x32-10 (counter (r, 0, tag, 0), key (seed, tag)), takes
// t = floor(u * W / 2^64) for the weight total W and picks the first frame
// whose inclusive prefix weight exceeds t.
//
// Euclidean rounds run in cooperative launches of up to kRoundBatch rounds
// (kmpp_rounds_kernel): every warp keeps the same frames in every round,
// lowers their minima by the newest center and adds the change of their
// integer weights to the tile sums; after a grid barrier every CTA makes the
// same draw from the same sums, so the new center needs no second exchange.
//
// Pruning (large n d): each frame keeps, besides D^2 = mind, the index a of a
// center whose exact distance is mind.  Each round starts with
//   cc_j = ||c_new - c_j||^2 for every earlier center j (float32), a warp per
//   center over the whole grid, and a second barrier.
// By the triangle inequality ||x - c_new|| >= ||c_new - c_a|| - ||x - c_a||,
// so when cc_a >= 4 mind (times a factor covering the float32 rounding of
// mind, of the new distance and of cc) the exact new distance cannot fall
// below mind and the frame's row is not read.  The running minima, and so the
// draws, are the same as without pruning, bit for bit.  A skipped frame costs
// 8 bytes (mind, a) instead of 4d + 4.
//
// Under the minRMSD metric a round is one launch per center: a pass over the
// frames, after which the CTA that finishes last (a fenced atomic count, no
// waiting) draws the round's frame and copies it into the centers.
#include <algorithm>
#include <climits>
#include <cmath>
#include <cstdlib>
#include <type_traits>

#include "km_common.cuh"
#include "km_internal.h"
#include "km_rmsd.cuh"

namespace km {

namespace {

constexpr int kTile = 2048;  // frames per weight tile (minRMSD)
constexpr int kTileThreads = 256;
constexpr int kRoundThreads = 1024;
constexpr int kRoundBatch = 64;   // rounds per launch
constexpr int kWide = 32;         // features from which a warp forms the distances together

// Tiles of the Euclidean rounds: 128 to 16,384 frames, about 2,048 tiles in
// between (the draw scans the tiles, then one tile: two or three values per
// thread each up to 4 million frames).
int tile_shift(int64_t n) {
    int sh = 7;
    while (sh < 14 && (n >> sh) > 2048) ++sh;
    return sh;
}

int64_t tile_slots(int64_t n) {
    const int sh = tile_shift(n);
    return std::max<int64_t>((n + (int64_t(1) << sh) - 1) >> sh, 1);
}

struct KmppWs {
    float *mind;
    int32_t *near;  // a center whose exact distance is mind (pruned rounds), or mind of the other parity
    float *cc;      // bounds of ||c_new - c_j||^2 for the current round
    unsigned long long *tile_sum;  // three sets (Euclidean) of tile_slots, or one of n / kTile
    uint32_t *maxbits;
    int *qexp;      // e of the weights floor(D^2 2^e); INT_MIN: every weight is 0
    unsigned int *done;  // CTAs of the current round that have finished; barrier count
    uint32_t *err;
};

KmppWs carve(void *ws, int64_t n, int k, size_t *bytes) {
    Carver c(ws);
    KmppWs w;
    const int64_t tiles = std::max<int64_t>(3 * tile_slots(n), (n + kTile - 1) / kTile);
    w.mind = c.take<float>(n > 0 ? n : 1);
    w.near = c.take<int32_t>(n > 0 ? n : 1);
    w.cc = c.take<float>(k > 0 ? k : 1);
    w.tile_sum = c.take<unsigned long long>(tiles);
    w.maxbits = c.take<uint32_t>(1);
    w.qexp = c.take<int>(1);
    w.done = c.take<unsigned int>(1);
    w.err = c.take<uint32_t>(1);
    if (bytes) *bytes = c.bytes();
    return w;
}

// floor(w 2^e) for a finite w > 0, else 0: the integer weight of a squared
// distance, from the float's bits (no FP64 arithmetic; equal to converting
// the exact double product w * 2^e).  e is chosen so that every weight fits.
__device__ __forceinline__ unsigned long long quant_weight(float w, int e) {
    const uint32_t b = __float_as_uint(w);
    if (e == INT_MIN || b == 0u || b >= 0x7f800000u) return 0ull;  // also every negative value
    const int be = (int)(b >> 23);
    const unsigned long long m = be ? (unsigned long long)((b & 0x7FFFFFu) | 0x800000u) : (unsigned long long)b;
    const int sh = (be ? be : 1) - 150 + e;
    if (sh >= 0) return m << sh;
    return sh <= -32 ? 0ull : (m >> (-sh));
}

__device__ __forceinline__ unsigned long long block_sum_u64(unsigned long long v,
                                                            unsigned long long *red) {
    for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (lane == 0) red[warp] = v;
    __syncthreads();
    unsigned long long s = 0;
    if (threadIdx.x == 0)
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) s += red[w];
    return s;  // valid in thread 0
}

// D^2 of frame i to the center drawn in round r under the minRMSD metric.
__device__ __forceinline__ float kmpp_rmsd_d2(int64_t i, int d, const KmppMetric &m, int r) {
    const int64_t p = m.idx[r];
    return __double2float_rn(rmsd_msd_rows(m.Xc + i * d, m.Xc + p * d, m.G[i], m.G[p], d / 3));
}

// minRMSD, round 1: mind = D^2 to center 0; max of the finite values.
__global__ void __launch_bounds__(kTileThreads) kmpp_first_kernel(int64_t n, int d, float *__restrict__ mind,
                                                                  uint32_t *__restrict__ maxbits, KmppMetric m) {
    float mx = 0.0f;
    const int64_t t0 = (int64_t)blockIdx.x * kTile;
    for (int u = 0; u < kTile / kTileThreads; ++u) {
        const int64_t i = t0 + u * kTileThreads + threadIdx.x;
        if (i < n) {
            const float dd = kmpp_rmsd_d2(i, d, m, 0);
            mind[i] = dd;
            if (dd < __int_as_float(0x7f800000) && dd > mx) mx = dd;
        }
    }
    for (int off = 16; off > 0; off >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, off));
    if ((threadIdx.x & 31) == 0 && mx > 0.0f) atomicMax(maxbits, __float_as_uint(mx));
}

// e = 62 - ceil(log2 n) - E(max) with 2^(E-1) <= max < 2^E (weights
// floor(D^2 2^e)); INT_MIN when no distance is finite and positive.
__device__ __forceinline__ int weight_exponent(uint32_t b, int64_t n) {
    const float m = __uint_as_float(b);
    if (!(m > 0.0f) || m == __int_as_float(0x7f800000)) return INT_MIN;
    int L = 0;
    while ((int64_t(1) << L) < n) ++L;
    const int be = (int)((b >> 23) & 0xFFu);
    int E;
    if (be) {
        E = be - 126;
    } else {
        const int p = 31 - __clz(b & 0x7FFFFFu);
        E = p - 148;
    }
    return 62 - L - E;
}

__global__ void kmpp_scale_kernel(const uint32_t *__restrict__ maxbits, int64_t n, int *__restrict__ qexp) {
    *qexp = weight_exponent(*maxbits, n);
}

// Exclusive prefix sum of v over the CTA (THREADS threads, warp shuffles
// and one pass over the warp totals); *total gets the sum.
template <int THREADS>
__device__ __forceinline__ unsigned long long cta_exclusive_scan_u64(unsigned long long v,
                                                                     unsigned long long *warp_tot,
                                                                     unsigned long long *total) {
    constexpr int kWarps = THREADS / 32;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    unsigned long long x = v;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
        const unsigned long long y = __shfl_up_sync(0xffffffffu, x, off);
        if (lane >= off) x += y;
    }
    __syncthreads();  // warp_tot of an earlier scan has been read
    if (lane == 31) warp_tot[warp] = x;
    __syncthreads();
    if (warp == 0) {
        unsigned long long w = lane < kWarps ? warp_tot[lane] : 0ull;
#pragma unroll
        for (int off = 1; off < kWarps; off <<= 1) {
            const unsigned long long y = __shfl_up_sync(0xffffffffu, w, off);
            if (lane >= off) w += y;
        }
        if (lane < kWarps) warp_tot[lane] = w;
    }
    __syncthreads();
    *total = warp_tot[kWarps - 1];
    return (warp > 0 ? warp_tot[warp - 1] : 0ull) + x - v;
}

// The draw of round r by a whole CTA (the tile sums and the minima of other
// CTAs are read past L1): t = floor(u W / 2^64) for the weight total W over
// the tiles of 2^shift frames, the first frame whose inclusive prefix weight
// exceeds t (a uniform frame when W = 0).  The frame, in every thread.
template <int THREADS>
__device__ __forceinline__ int64_t kmpp_draw_round(int64_t ntiles, int shift, int64_t n,
                                                   const float *__restrict__ mind, int qexp,
                                                   const unsigned long long *__restrict__ tile_sum, int r,
                                                   uint32_t seed) {
    __shared__ unsigned long long red[THREADS / 32];
    __shared__ long long tile_hit, pick;
    __shared__ unsigned long long target;
    __syncthreads();  // the last draw's values have been read
    if (threadIdx.x == 0) {
        tile_hit = -1;
        pick = -1;
    }
    __syncthreads();
    const uint64_t u = kmpp_draw(seed, (uint32_t)r);
    const int64_t per = (ntiles + THREADS - 1) / THREADS;
    const int64_t lo = min((int64_t)threadIdx.x * per, ntiles), hi = min(lo + per, ntiles);
    unsigned long long ts = 0;
    for (int64_t b = lo; b < hi; ++b) ts += __ldcg(tile_sum + b);
    unsigned long long total;
    const unsigned long long excl = cta_exclusive_scan_u64<THREADS>(ts, red, &total);
    if (total > 0) {
        const unsigned long long t = __umul64hi(u, total);
        if (excl <= t && t < excl + ts) {
            unsigned long long run = excl;
            for (int64_t b = lo; b < hi; ++b) {
                const unsigned long long w = __ldcg(tile_sum + b);
                if (t < run + w) {
                    tile_hit = b;
                    target = t - run;
                    break;
                }
                run += w;
            }
        }
    }
    __syncthreads();
    if (tile_hit >= 0) {
        // Inside the tile: consecutive frames per thread.
        const int tper = max(1, (1 << shift) / THREADS);
        const int64_t first = (int64_t)tile_hit << shift, end = min(n, first + (int64_t(1) << shift));
        const int64_t f0 = min(first + (int64_t)threadIdx.x * tper, end), f1 = min(f0 + tper, end);
        unsigned long long ws = 0;
        for (int64_t f = f0; f < f1; ++f) ws += quant_weight(__ldcg(mind + f), qexp);
        unsigned long long tile_total;
        unsigned long long run = cta_exclusive_scan_u64<THREADS>(ws, red, &tile_total);
        const unsigned long long tt = target;
        if (run <= tt && tt < run + ws) {
            for (int64_t f = f0; f < f1; ++f) {
                const unsigned long long w = quant_weight(__ldcg(mind + f), qexp);
                if (tt < run + w) {
                    pick = f;
                    break;
                }
                run += w;
            }
        }
    }
    __syncthreads();
    return pick >= 0 ? (int64_t)pick : (int64_t)__umul64hi(u, (unsigned long long)n);
}

// True in every thread of the CTA that counts itself last among gridDim.x
// (after a fence of this thread's writes); the others' writes are visible
// to it past L1.
__device__ __forceinline__ bool kmpp_last_cta(unsigned int *__restrict__ done) {
    __shared__ bool last;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) last = atomicAdd(done, 1u) == gridDim.x - 1;
    __syncthreads();
    if (last) __threadfence();
    return last;
}

// minRMSD, round r >= 1, one CTA per tile of kTile frames, one thread per
// frame (at a time).  With r_center >= 0 the running minimum first takes the
// distance to center r_center (rounds >= 2; round 1 uses the minimum of
// kmpp_first_kernel as it is).  Then the tile's weight sum is stored and the
// CTA that finishes last draws.
__global__ void __launch_bounds__(kTileThreads) kmpp_round_kernel(
    const DenseRows src, int64_t n, int d, float *__restrict__ C0, int64_t *__restrict__ idx_out,
    float *__restrict__ mind, const int *__restrict__ qexp_p, unsigned long long *__restrict__ tile_sum,
    unsigned int *__restrict__ done, KmppMetric m, int r_center, int r, uint32_t seed) {
    __shared__ unsigned long long red[kTileThreads / 32];
    const int qexp = *qexp_p;
    const int64_t t0 = (int64_t)blockIdx.x * kTile;
    unsigned long long s = 0;
    for (int u = 0; u < kTile / kTileThreads; ++u) {
        const int64_t i = t0 + u * kTileThreads + threadIdx.x;
        if (i < n) {
            float mi = mind[i];
            if (r_center >= 0) {
                const float dd = kmpp_rmsd_d2(i, d, m, r_center);
                if (dd < mi) {
                    mi = dd;
                    mind[i] = mi;
                }
            }
            s += quant_weight(mi, qexp);
        }
    }
    s = block_sum_u64(s, red);
    if (threadIdx.x == 0) tile_sum[blockIdx.x] = s;
    if (!kmpp_last_cta(done)) return;
    const int64_t p = kmpp_draw_round<kTileThreads>(gridDim.x, 11, n, mind, qexp, tile_sum, r, seed);
    for (int f = threadIdx.x; f < d; f += kTileThreads) C0[(int64_t)r * d + f] = src.get(p, f);
    if (threadIdx.x == 0) {
        if (idx_out) idx_out[r] = p;
        *done = 0u;  // for the next round's launch
    }
}
static_assert(kTile == 1 << 11, "the draw's tiles");

// Round 0 under the minRMSD metric: a uniformly drawn frame, copied into C0[0].
__global__ void __launch_bounds__(kTileThreads) kmpp_uniform_kernel(const DenseRows src, int64_t n, int d,
                                                                    float *__restrict__ C0,
                                                                    int64_t *__restrict__ idx_out, uint32_t seed) {
    const int64_t p = (int64_t)__umul64hi(kmpp_draw(seed, 0u), (unsigned long long)n);
    for (int f = threadIdx.x; f < d; f += blockDim.x) C0[f] = src.get(p, f);
    if (idx_out && threadIdx.x == 0) idx_out[0] = p;
}

// ---- Euclidean rounds ----------------------------------------------------------

// A warp's scratch for the distances of wide rows.  With more (5 KB squares,
// lists of 160 frames and their minima) the shared memory of 32 warps left the
// L1 cache so little that rows in flight were evicted: 500,000 x 528, every
// row, 290 us instead of 194.
struct WarpScratch {
    float sq[128 * 9];  // [feature][frame], row stride frames + 1 (odd: no bank conflicts either way)
    int32_t id[96];     // the frames that the bound left, compacted
};

// Exact distances of the m <= J rows ids[0..m) to c, row j's in lane j.  Each
// run of 32 * (32 / J) features of J rows is loaded at once (32 coalesced
// loads in flight, beside the sums of the run before), squared and stored transposed; lane j then adds row j's
// squares in feature order, so each distance is the same sequence of float32
// operations as sqdist_exact, bit for bit.
template <int J, class Src>
__device__ __forceinline__ float warp_rows_sqdist(const Src &src, const int32_t *ids, int m, const float *c, int d,
                                                  float *sq) {
    constexpr int kRuns = 32 / J;
    const int lane = threadIdx.x & 31, j0 = lane & (J - 1);
    float v[32];
    auto load = [&](int f0) {
#pragma unroll
        for (int j = 0; j < J; ++j)
#pragma unroll
            for (int q = 0; q < kRuns; ++q) {
                const int f = f0 + q * 32 + lane;
                v[j * kRuns + q] = (j < m && f < d) ? src.get(ids[j], f) : 0.0f;
            }
    };
    load(0);
    float acc = 0.0f;
    for (int f0 = 0; f0 < d; f0 += 32 * kRuns) {
#pragma unroll
        for (int q = 0; q < kRuns; ++q) {
            const int f = f0 + q * 32 + lane;
            const float cf = f < d ? c[f] : 0.0f;
#pragma unroll
            for (int j = 0; j < J; ++j) sq[(q * 32 + lane) * (J + 1) + j] = sq_term(v[j * kRuns + q], cf);
        }
        __syncwarp();
        if (f0 + 32 * kRuns < d) load(f0 + 32 * kRuns);  // on its way during the sums
        const int run = min(32 * kRuns, d - f0);
        if (run == 32 * kRuns) {
#pragma unroll 8
            for (int f = 0; f < 32 * kRuns; ++f) acc = __fadd_rn(acc, sq[f * (J + 1) + j0]);
        } else {
#pragma unroll 8
            for (int f = 0; f < run; ++f) acc = __fadd_rn(acc, sq[f * (J + 1) + j0]);
        }
        __syncwarp();  // sq is overwritten by the next run of features
    }
    return acc;
}

template <class Src>
__device__ __forceinline__ float warp_rows_sqdist(const Src &src, const int32_t *ids, int m, const float *c, int d,
                                                  float *sq) {
    if (m > 16) return warp_rows_sqdist<32>(src, ids, m, c, d, sq);
    if (m > 8) return warp_rows_sqdist<16>(src, ids, m, c, d, sq);
    return warp_rows_sqdist<8>(src, ids, m, c, d, sq);
}

// Row i, zero beyond its d <= DP features.
template <int DP, class Src>
__device__ __forceinline__ void load_row(const Src &src, int64_t i, int d, float (&v)[DP]) {
    if constexpr (std::is_same<Src, DenseRows>::value && DP >= 4) {
        if ((d & 3) == 0 && (reinterpret_cast<uintptr_t>(src.X) & 15) == 0) {
            const float4 *x = reinterpret_cast<const float4 *>(src.X + i * d);
#pragma unroll
            for (int f = 0; f < DP; f += 4) {
                const float4 t = f < d ? __ldg(x + (f >> 2)) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                v[f] = t.x, v[f + 1] = t.y, v[f + 2] = t.z, v[f + 3] = t.w;
            }
            return;
        }
    }
#pragma unroll
    for (int f = 0; f < DP; ++f) v[f] = f < d ? src.get(i, f) : 0.0f;
}

// The operations of sqdist_exact on a loaded row; c is zero beyond d, where
// the added squares are zero.
template <int DP>
__device__ __forceinline__ float row_sqdist(const float (&v)[DP], const float *c) {
    float acc = 0.0f;
#pragma unroll
    for (int f = 0; f < DP; ++f) acc = __fadd_rn(acc, sq_term(v[f], c[f]));
    return acc;
}

__device__ __forceinline__ unsigned long long warp_sum_u64(unsigned long long v) {
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
    return v;
}

struct RoundParams {
    int64_t n, ntiles;
    int d, shift;
    int r0, r1;  // the rounds of this launch
    float *C0;
    int64_t *idx;
    KmppWs w;
    float prune;  // prune_factor(d)
    uint32_t seed;
    int cc_s;  // bounds that fit in shared memory
};

// Rounds r0..r1-1: round r lowers the minima by center r - 1 and draws center
// r (round 0 draws uniformly).  DP = 0: wide rows, whose distances a warp forms
// together; else rows of d <= DP features, a thread per frame.  PRUNE: see the
// head of this file; without it every round rewrites the minima into the
// buffer of the other parity and the tile sums from zero, so a CTA that is
// still drawing round r is not disturbed by one that works on round r + 1,
// and one barrier per round is enough.
//
// A warp's frames lie in runs of 8 (wide) or 32 spread evenly over the
// frames: the frames of a trajectory near the newest center are neighbours,
// and their rows are the work of a round.
//
// What bounds it: early rounds read nearly every row (HBM), later rounds are
// a chain of barrier, scans and row latency (about 6 us unpruned, 9 us
// pruned).  us per round, launches per round -> here: 100,000 x 2 10 -> 7;
// 500,000 x 10 15 -> 11; 100,000 x 67 21 -> 14; 20,000 x 528 33 -> 17;
// 500,000 x 528, k = 300 56 -> 44, its first 50 rounds 120 -> 120.
template <class Src, int DP, bool PRUNE>
__global__ void __launch_bounds__(kRoundThreads, 1) kmpp_rounds_kernel(const Src src, const RoundParams p) {
    extern __shared__ float4 kmpp_sm[];
    constexpr bool WIDE = DP == 0;
    constexpr int kRun = WIDE ? 8 : 32;                        // consecutive frames of a warp
    constexpr int kSlots = WIDE ? 2 : 4;                        // loads of 32 minima in flight,
    constexpr int kAll = WIDE || DP > 8 ? 1 : DP == 8 ? 2 : 4;  // and of 32 narrow rows
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    WarpScratch *scr = reinterpret_cast<WarpScratch *>(kmpp_sm) + warp;
    float *c_s = reinterpret_cast<float *>(reinterpret_cast<WarpScratch *>(kmpp_sm) + (WIDE ? kRoundThreads / 32 : 0));
    const int64_t n = p.n;
    const int d = p.d;
    const int64_t W = (int64_t)gridDim.x * (kRoundThreads / 32);
    const int64_t gw = (int64_t)warp * gridDim.x + blockIdx.x;  // neighbours in different CTAs
    const int64_t runs = (n + kRun - 1) / kRun;
    float *cc_s = c_s + (WIDE ? d : DP);
    unsigned int bars = 0;
    bool ok = *p.w.err == 0u;
    int qexp = INT_MIN;
    // frame of this lane in slot s (32 frames from 32 / kRun runs); >= n: none
    auto frame = [&](int64_t g0, int s) -> int64_t {
        const int64_t run = g0 + (int64_t)(s * (32 / kRun) + lane / kRun) * W;
        return run < runs ? run * kRun + lane % kRun : n;
    };
    auto barrier = [&]() { return grid_barrier(p.w.done, ++bars * gridDim.x, p.w.err); };
    if (!WIDE && threadIdx.x < DP) c_s[threadIdx.x] = 0.0f;  // stays zero beyond d
    __syncthreads();
    int r = p.r0;
    if (r > 0 && ok) {
        const float *row = p.C0 + (int64_t)(r - 1) * d;
        for (int f = threadIdx.x; f < d; f += kRoundThreads) c_s[f] = __ldcg(row + f);
        __syncthreads();
        if (r > 1) qexp = weight_exponent(__ldcg(p.w.maxbits), n);
    }
    for (; ok && r < p.r1; ++r) {
        int64_t pick;
        if (r == 0) {
            pick = (int64_t)__umul64hi(kmpp_draw(p.seed, 0u), (unsigned long long)n);
        } else {
            const float *m_in = PRUNE || ((r - 1) & 1) == 0 ? p.w.mind : reinterpret_cast<float *>(p.w.near);
            float *m_out = PRUNE || (r & 1) == 0 ? p.w.mind : reinterpret_cast<float *>(p.w.near);
            unsigned long long *tiles = p.w.tile_sum + (PRUNE ? 0 : (r % 3) * p.ntiles);
            if constexpr (PRUNE) {
                if (r > 1) {  // cc
                    for (int64_t j = gw; j < r - 1; j += W) {
                        const float *b = p.C0 + j * d;
                        float acc = 0.0f;
                        for (int f = lane; f < d; f += 32) {
                            const float t = __fsub_rn(c_s[f], __ldcg(b + f));
                            acc = __fmaf_rn(t, t, acc);
                        }
#pragma unroll
                        for (int off = 16; off > 0; off >>= 1)
                            acc = __fadd_rn(acc, __shfl_xor_sync(0xffffffffu, acc, off));
                        if (lane == 0) p.w.cc[j] = acc;
                    }
                    ok = barrier();
                    if (!ok) break;
                    // Read past L1 by every frame they would queue up at the
                    // few L2 lines that hold them (2M x 32, k = 300: 61 us a
                    // round, 46 from shared memory).
                    for (int j = threadIdx.x; j < min(r - 1, p.cc_s); j += kRoundThreads) cc_s[j] = __ldcg(p.w.cc + j);
                    __syncthreads();
                }
            }
            // Every frame's distance, 32 frames at a time (round 1, and every unpruned round).
            if (!PRUNE || r == 1) {
                float mx = 0.0f;
                for (int64_t g0 = gw; g0 < runs; g0 += W * (32 / kRun) * kAll) {
                    float dd[kAll], mi[kAll];
                    int64_t i[kAll];
#pragma unroll
                    for (int s = 0; s < kAll; ++s) {
                        i[s] = frame(g0, s);
                        mi[s] = r > 1 && i[s] < n ? __ldcg(m_in + i[s]) : 0.0f;
                    }
                    if constexpr (WIDE) {
                        scr->id[lane] = i[0] < n ? (int32_t)i[0] : 0;
                        const int m = __popc(__ballot_sync(0xffffffffu, i[0] < n));  // the first m lanes
                        __syncwarp();
                        dd[0] = warp_rows_sqdist(src, scr->id, m, c_s, d, scr->sq);
                    } else {
                        float v[kAll][DP];
#pragma unroll
                        for (int s = 0; s < kAll; ++s)
                            if (i[s] < n) load_row<DP>(src, i[s], d, v[s]);
#pragma unroll
                        for (int s = 0; s < kAll; ++s) dd[s] = i[s] < n ? row_sqdist<DP>(v[s], c_s) : 0.0f;
                    }
#pragma unroll
                    for (int s = 0; s < kAll; ++s) {
                        unsigned long long w = 0ull;
                        if (i[s] < n) {
                            if (r == 1) {
                                if (dd[s] < __int_as_float(0x7f800000) && dd[s] > mx) mx = dd[s];
                                if constexpr (PRUNE) p.w.near[i[s]] = 0;
                            } else {
                                dd[s] = dd[s] < mi[s] ? dd[s] : mi[s];
                                w = quant_weight(dd[s], qexp);
                            }
                            m_out[i[s]] = dd[s];
                        }
                        if (r > 1) {  // a run lies in one tile
#pragma unroll
                            for (int off = kRun / 2; off > 0; off >>= 1) w += __shfl_xor_sync(0xffffffffu, w, off);
                            if (lane % kRun == 0 && w) atomicAdd(tiles + (i[s] >> p.shift), w);
                        }
                    }
                }
                if (r == 1) {
                    for (int off = 16; off > 0; off >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, off));
                    if (lane == 0 && mx > 0.0f) atomicMax(p.w.maxbits, __float_as_uint(mx));
                    ok = barrier();
                    if (!ok) break;
                    qexp = weight_exponent(__ldcg(p.w.maxbits), n);
                    for (int64_t g0 = gw; g0 < runs; g0 += W * (32 / kRun)) {
                        const int64_t i = frame(g0, 0);
                        unsigned long long w = i < n ? quant_weight(__ldcg(m_out + i), qexp) : 0ull;
#pragma unroll
                        for (int off = kRun / 2; off > 0; off >>= 1) w += __shfl_xor_sync(0xffffffffu, w, off);
                        if (lane % kRun == 0 && w) atomicAdd(tiles + (i >> p.shift), w);
                    }
                }
            } else {
                const int rc = r - 1;
                // A smaller distance dd of frame i replaces its minimum mi and
                // a, and moves its integer weight in its tile's sum (modular
                // 64-bit deltas, exact).
                auto lower = [&](bool in, int64_t i, float mi, float dd) {
                    const bool less = in && dd < mi;
                    unsigned long long delta = 0ull;
                    if (less) {
                        p.w.mind[i] = dd;
                        p.w.near[i] = rc;
                        delta = quant_weight(dd, qexp) - quant_weight(mi, qexp);
                    }
                    const unsigned any = __ballot_sync(0xffffffffu, delta != 0ull);
                    if (!any) return;
                    const int t = (int)(i >> p.shift), first = __shfl_sync(0xffffffffu, t, __ffs(any) - 1);
                    if (__all_sync(0xffffffffu, delta == 0ull || t == first)) {
                        delta = warp_sum_u64(delta);
                        if (lane == 0 && delta) atomicAdd(tiles + first, delta);
                    } else if (delta) {
                        atomicAdd(tiles + t, delta);
                    }
                };
                int cnt = 0;  // wide: listed frames
                for (int64_t g0 = gw; g0 < runs; g0 += W * (32 / kRun) * kSlots) {
                    float mi[kSlots];
                    int32_t a[kSlots];
#pragma unroll
                    for (int s = 0; s < kSlots; ++s) {
                        const int64_t i = frame(g0, s);
                        mi[s] = i < n ? __ldcg(p.w.mind + i) : 0.0f;
                        a[s] = i < n ? __ldcg(p.w.near + i) : 0;
                    }
                    bool keep[kSlots];
#pragma unroll
                    for (int s = 0; s < kSlots; ++s) {  // the skip needs a finite minimum; a NaN bound never skips
                        const float cc = a[s] < p.cc_s ? cc_s[a[s]] : __ldcg(p.w.cc + a[s]);
                        keep[s] = frame(g0, s) < n &&
                                  !(mi[s] <= 3.4028234663852886e38f && cc >= __fmul_ru(mi[s], p.prune));
                    }
                    if constexpr (WIDE) {
                        // Full groups of 32 rows; the rest waits for the next
                        // frames' or the end.
#pragma unroll
                        for (int s = 0; s < kSlots; ++s) {
                            const unsigned b = __ballot_sync(0xffffffffu, keep[s]);
                            if (keep[s]) {
                                const int q = cnt + __popc(b & ((1u << lane) - 1u));
                                scr->id[q] = (int32_t)frame(g0, s);
                            }
                            cnt += __popc(b);
                        }
                        __syncwarp();
                        const bool last = g0 + W * (32 / kRun) * kSlots >= runs;
                        int b0 = 0;
                        for (; cnt - b0 >= 32 || (last && b0 < cnt); b0 += 32) {
                            const int m = min(32, cnt - b0);
                            const int32_t id = lane < m ? scr->id[b0 + lane] : 0;
                            const float old = __ldcg(p.w.mind + id);
                            lower(lane < m, id, old, warp_rows_sqdist(src, scr->id + b0, m, c_s, d, scr->sq));
                        }
                        cnt -= min(b0, cnt);
                        const int32_t id = lane < cnt ? scr->id[b0 + lane] : 0;
                        __syncwarp();
                        scr->id[lane] = id;
                        __syncwarp();
                    } else {
#pragma unroll
                        for (int s0 = 0; s0 < kSlots; s0 += kAll) {
                            float v[kAll][DP];
#pragma unroll
                            for (int s = 0; s < kAll; ++s)
                                if (keep[s0 + s]) load_row<DP>(src, frame(g0, s0 + s), d, v[s]);
#pragma unroll
                            for (int s = 0; s < kAll; ++s) {
                                const bool in = keep[s0 + s];
                                if (!__any_sync(0xffffffffu, in)) continue;
                                lower(in, frame(g0, s0 + s), mi[s0 + s], in ? row_sqdist<DP>(v[s], c_s) : 0.0f);
                            }
                        }
                    }
                }
            }
            if (!PRUNE && blockIdx.x == 0) {  // the next round's tile sums
                unsigned long long *z = p.w.tile_sum + ((r + 1) % 3) * p.ntiles;
                for (int64_t t = threadIdx.x; t < p.ntiles; t += kRoundThreads) z[t] = 0ull;
            }
            ok = barrier();
            if (!ok) break;
            pick = kmpp_draw_round<kRoundThreads>(p.ntiles, p.shift, n, m_out, qexp, tiles, r, p.seed);
        }
        // Center r: in every CTA's shared memory, and in C0.
        for (int f = threadIdx.x; f < d; f += kRoundThreads) {
            const float x = src.get(pick, f);
            c_s[f] = x;
            if (blockIdx.x == 0) p.C0[(int64_t)r * d + f] = x;
        }
        if (blockIdx.x == 0 && threadIdx.x == 0 && p.idx) p.idx[r] = pick;
        __syncthreads();
    }
    if (!ok && blockIdx.x == 0) {  // a wait ran out: no centers from here on
        for (; r < p.r1; ++r) {
            for (int f = threadIdx.x; f < d; f += kRoundThreads) p.C0[(int64_t)r * d + f] = __int_as_float(0x7fc00000);
            if (threadIdx.x == 0 && p.idx) p.idx[r] = -1;
        }
    }
}

template <class Src, int DP, bool PRUNE>
int launch_rounds_dp(const Src &src, RoundParams &p, int k, cudaStream_t s) {
    constexpr size_t kMax = 226 * 1024;
    const size_t fixed = (DP == 0 ? sizeof(WarpScratch) * (kRoundThreads / 32) : 0) +
                         sizeof(float) * (DP == 0 ? p.d : DP);
    p.cc_s = PRUNE ? (int)std::min<size_t>(k, (kMax - fixed) / sizeof(float)) : 0;
    const size_t smem = fixed + sizeof(float) * p.cc_s;
    static bool set[kDeviceSlots] = {};
    const int dev = current_device();
    if (!(dev >= 0 && dev < kDeviceSlots && set[dev])) {
        KM_CUDA(cudaFuncSetAttribute(kmpp_rounds_kernel<Src, DP, PRUNE>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)kMax));
        if (dev >= 0 && dev < kDeviceSlots) set[dev] = true;
    }
    KM_CUDA(cudaMemsetAsync(p.w.done, 0, sizeof(unsigned int), s));
    // one CTA per SM, all resident at once (they wait for each other)
    constexpr int kRun = DP == 0 ? 8 : 32;
    const unsigned grid = (unsigned)std::min<int64_t>(num_sms(), (p.n + kRun - 1) / kRun);
    void *args[] = {(void *)&src, (void *)&p};
    KM_CUDA(cudaLaunchCooperativeKernel((const void *)kmpp_rounds_kernel<Src, DP, PRUNE>, dim3(grid),
                                        dim3(kRoundThreads), args, smem, s));
    return KM_OK;
}

template <class Src, bool PRUNE>
int launch_rounds(const Src &src, RoundParams &p, int k, cudaStream_t s) {
    if (p.d >= kWide) return launch_rounds_dp<Src, 0, PRUNE>(src, p, k, s);
    if constexpr (std::is_same<Src, DenseRows>::value) {
        if (p.d <= 2) return launch_rounds_dp<Src, 2, PRUNE>(src, p, k, s);
        if (p.d <= 4) return launch_rounds_dp<Src, 4, PRUNE>(src, p, k, s);
        if (p.d <= 8) return launch_rounds_dp<Src, 8, PRUNE>(src, p, k, s);
        if (p.d <= 16) return launch_rounds_dp<Src, 16, PRUNE>(src, p, k, s);
    }
    return launch_rounds_dp<Src, 32, PRUNE>(src, p, k, s);
}

}  // namespace

size_t kmpp_ws_size(int64_t n, int d, int k) {
    (void)d;
    size_t b = 0;
    carve(nullptr, n, k, &b);
    return b;
}

// The prune factor F for d features: a frame is skipped when
// cc_a >= F mind.  With u = 2^-24, the oracle's sequential float32 distance D
// of a frame to a center lies within (1 -+ u)^(d+3) of the exact squared
// distance (d subtractions, d squares, d additions, each rounded once), and
// the cc kernel's value within (1 +- u)^2 (1 +- g_m) of it, g_m = m u / (1 -
// m u) for its m = ceil(d/32) + 5 roundings per sum.  The exact new distance
// is at least (sqrt(CC) - sqrt(D*))^2 once sqrt(CC) >= sqrt(D*), which gives
// F = 4 (1 + u)^2 (1 + g_m) / (1 - u)^(d+3), enlarged by 2^-20 and rounded up
// to float.
float prune_factor(int d) {
    const double u = std::ldexp(1.0, -24);
    const double mrnd = (double)((d + 31) / 32 + 5);
    const double gm = mrnd * u / (1.0 - mrnd * u);
    const double f = 4.0 * (1.0 + u) * (1.0 + u) * (1.0 + gm) / std::pow(1.0 - u, (double)(d + 3)) *
                     (1.0 + std::ldexp(1.0, -20));
    float ff = (float)f;
    if ((double)ff < f) ff = std::nextafter(ff, 8.0f);
    return ff;
}

namespace {

template <class Src>
int run_kmpp_src(const Src &src, int64_t n, int d, int k, uint32_t seed, float *C0, int64_t *idx,
                 void (*cb)(void *), void *cb_user, void *ws, cudaStream_t s) {
    RoundParams p;
    p.w = carve(ws, n, k, nullptr);
    p.n = n;
    p.ntiles = tile_slots(n);
    p.d = d;
    p.shift = tile_shift(n);
    p.C0 = C0;
    p.idx = idx;
    p.prune = prune_factor(d);
    p.seed = seed;
    KM_CUDA(cudaMemsetAsync(p.w.tile_sum, 0, 3 * p.ntiles * sizeof(unsigned long long), s));
    KM_CUDA(cudaMemsetAsync(p.w.maxbits, 0, sizeof(uint32_t), s));
    // (the planted bits of the test hook: the launches then draw nothing)
    KM_CUDA(cudaMemsetAsync(p.w.err, (int)(take_fake_device_error() & 0xffu), sizeof(uint32_t), s));
    // A pruned round pays a second barrier and the bounds, and saves rows of
    // d words less two.  us per round (unpruned, pruned), k = 300:
    //   d = 2:    n = 500,000 8.6, 10.5;  2M 16.2, 15.1;  10M 67, 39
    //   d = 10:   n = 100,000 6.6, 9.1;   500,000 11.4, 11.1;  2M 25, 17
    //   d = 67:   n = 20,000 9.0, 11.2;   100,000 15.0, 14.2;  500,000 46, 25
    //   d = 528:  n = 1,000 12, 15;       20,000 19, 17.5;     100,000 53, 21
    // KM_KMPP_PRUNE=0 or 1 in the environment forces the choice (both give
    // the same draws).
    bool prune = n * (int64_t)(d + 4) >= (int64_t(1) << 23);
    if (const char *e = std::getenv("KM_KMPP_PRUNE")) prune = e[0] == '1';
    const int batch = cb ? 1 : kRoundBatch;
    for (int r = 0; r < k; r += batch) {
        p.r0 = r;
        p.r1 = std::min(k, r + batch);
        KM_TRY(prune ? (launch_rounds<Src, true>(src, p, k, s)) : (launch_rounds<Src, false>(src, p, k, s)));
        if (cb) cb(cb_user);
    }
    return KM_OK;
}

int run_kmpp_rmsd(const DenseRows &src, int64_t n, int d, int k, uint32_t seed, float *C0, int64_t *idx,
                  void (*cb)(void *), void *cb_user, void *ws, cudaStream_t s, const KmppMetric &m) {
    KmppWs w = carve(ws, n, k, nullptr);
    const unsigned ntiles = (unsigned)((n + kTile - 1) / kTile);
    kmpp_uniform_kernel<<<1, kTileThreads, 0, s>>>(src, n, d, C0, idx, seed);
    KM_CUDA(cudaGetLastError());
    if (cb) cb(cb_user);
    if (k == 1) return KM_OK;
    KM_CUDA(cudaMemsetAsync(w.maxbits, 0, sizeof(uint32_t), s));
    KM_CUDA(cudaMemsetAsync(w.done, 0, sizeof(unsigned int), s));
    kmpp_first_kernel<<<ntiles, kTileThreads, 0, s>>>(n, d, w.mind, w.maxbits, m);
    KM_CUDA(cudaGetLastError());
    kmpp_scale_kernel<<<1, 1, 0, s>>>(w.maxbits, n, w.qexp);
    KM_CUDA(cudaGetLastError());
    for (int r = 1; r < k; ++r) {
        kmpp_round_kernel<<<ntiles, kTileThreads, 0, s>>>(src, n, d, C0, idx, w.mind, w.qexp, w.tile_sum, w.done, m,
                                                          r >= 2 ? r - 1 : -1, r, seed);
        KM_CUDA(cudaGetLastError());
        if (cb) cb(cb_user);
    }
    return KM_OK;
}

}  // namespace

int run_kmpp(const float *X, int64_t n, int d, int k, uint32_t seed, float *C0, int64_t *idx,
             void (*cb)(void *), void *cb_user, void *ws, cudaStream_t s, const KmppMetric *metric,
             const PairSrc *ps) {
    const KmppMetric m = metric ? *metric : KmppMetric{nullptr, nullptr, nullptr};
    if (n <= 0) {
        set_error("kmeans++ needs at least one frame");
        return KM_ERR_BAD_SHAPE;
    }
    if (ps) {
        if (m.Xc) {
            set_error("kmeans++ under the minRMSD metric takes dense frames");
            return KM_ERR_UNSUPPORTED;
        }
        const PairRows pr{ps->xyz, reinterpret_cast<const int2 *>(ps->pairs), ps->n_atoms, d};
        return run_kmpp_src(pr, n, d, k, seed, C0, idx, cb, cb_user, ws, s);
    }
    if (m.Xc) return run_kmpp_rmsd(DenseRows{X, d}, n, d, k, seed, C0, idx, cb, cb_user, ws, s, m);
    return run_kmpp_src(DenseRows{X, d}, n, d, k, seed, C0, idx, cb, cb_user, ws, s);
}

}  // namespace km
