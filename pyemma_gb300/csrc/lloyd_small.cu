// lloyd_small.cu -- Lloyd iterations of few, narrow centers in one launch.
//
// Reference: KMeans.fit from given centers, pyemma/coordinates/clustering/
// kmeans.py:253-258, with the stopping rule of kmeans.py:432-436.
//
// With d <= 16 and centers and sums that fit in shared memory, an iteration is
// a few microseconds of work, and separate launches for the assignment, the
// sums, the new centers and the stopping rule cost more than that (40 us per
// iteration on 100,000 x 2 frames, k = 50, inside a graph loop).  Here one
// cooperative launch runs up to the requested number of iterations.  In each,
// every CTA
//   1. assigns its frames, a thread each, exactly (feature order, every
//      operation rounded on its own, lowest index among the minima) to the
//      centers in its shared memory, and sums the float32 deviations from
//      them per center.  Float64 atomics in shared memory are retry loops, and
//      32 lanes that meet on one center serialise them; so the 512 frames are
//      sorted by label in shared memory (native integer counts) and four
//      lanes per center and feature (one, where the centers outnumber a
//      quarter of the frames) walk its members with compensated float32 sums
//      (in float64 where those leave the range of float32).
//      A warp whose frames all have one label (consecutive frames often do)
//      adds them by shuffles and stays out of the sort;
//   2. adds its sums to the iteration's global sums and meets the other CTAs
//      at a barrier (one atomic count; the wait is bounded);
//   3. forms all new centers, the inertia and the stopping decision from the
//      global sums, each CTA for itself: the same inputs in the same order
//      give the same values in every CTA, so nothing has to be handed out.
// The global sums rotate through three buffers: the one of iteration i + 1 is
// cleared before the barrier of iteration i, when every CTA has come through
// that of iteration i - 1 and so is done with its use in iteration i - 2.
//
// What bounds it: at small n the chain of one iteration (first distance to
// barrier to new centers), 12-20 us; at large n the FP32 pipe of the
// distances.  us per iteration, the graph loop of separate kernels -> here:
// 100,000 x 2, k = 50 40 -> 19; 50,000 x 4, k = 100 77 -> 20; 1M x 8, k = 50
// 444 -> 139; 4M x 16, k = 100 2533 -> 1249.  Sums by float64 shared-memory
// atomics on runs of frames took 85 us at 1M x 2, k = 50 (58 here) and 55 us
// at 50,000 x 2, k = 10 (13 here).
#include <algorithm>

#include "km_common.cuh"
#include "km_internal.h"

namespace km {

namespace {

constexpr int kFuThreads = 512;
constexpr size_t kFuSumsMax = 48 * 1024;   // centers and sums (the limit of the shapes taken)
constexpr size_t kFuMaxSmem = 88 * 1024;   // with the deviations of 512 frames: two CTAs per SM

int fu_dp(int d) { return d <= 1 ? 1 : d <= 2 ? 2 : d <= 4 ? 4 : d <= 8 ? 8 : 16; }

// Row stride of the deviations (d features and the squared length), odd.
__host__ __device__ inline int fu_stride(int d) { return (d + 1) | 1; }

// Centers, sums and counts of k centers.
size_t fu_sums_bytes(int d, int k) {
    return (size_t)k * d * 8 + (size_t)k * 8 + (size_t)k * fu_dp(d) * 4 + (size_t)k * 4;
}

size_t fu_smem(int d, int k) {
    // + members of a chunk and their offsets, the deviations, the sorted order
    return fu_sums_bytes(d, k) + (size_t)(2 * k + 1) * 4 + (size_t)kFuThreads * fu_stride(d) * 4 + kFuThreads * 2;
}

// Doubles of one buffer of global sums: S (k x d), Q (k), and the counts.
__host__ __device__ inline size_t fu_buf_doubles(int d, int k) { return (size_t)k * d + k + (k + 1) / 2; }

// Sums of finite terms may leave the range of float32 (squares of 1e18 and
// more); they are then made in float64.  Terms that are not finite leave a NaN.
__device__ __forceinline__ bool fu_finite(double v) { return fabs(v) <= 1.7976931348623157e308; }

// Sum over the CTA in a fixed order (warp shuffles, then warp 0), in every thread.
__device__ __forceinline__ double fu_block_sum(double v, double *red) {
    for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
    __syncthreads();  // red of an earlier sum has been read
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
    __syncthreads();
    double s = 0.0;
    for (int w = 0; w < kFuThreads / 32; ++w) s += red[w];
    return s;
}

// Exclusive prefix sums of m[0..k) into off[0..k], by the whole CTA.
__device__ __forceinline__ void fu_scan(const int32_t *m, int k, int32_t *off) {
    __shared__ int32_t tot[kFuThreads / 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int32_t base = 0;
    for (int j0 = 0; j0 < k; j0 += kFuThreads) {
        const int j = j0 + threadIdx.x;
        const int32_t v = j < k ? m[j] : 0;
        int32_t x = v;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int32_t y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += y;
        }
        if (lane == 31) tot[warp] = x;
        __syncthreads();
        int32_t before = 0, all = 0;
        for (int w = 0; w < kFuThreads / 32; ++w) {
            if (w < warp) before += tot[w];
            all += tot[w];
        }
        if (j < k) off[j] = base + before + x - v;
        base += all;
        __syncthreads();
    }
}

template <int DP>
__global__ void __launch_bounds__(kFuThreads, 2) small_lloyd_kernel(
    const float *__restrict__ X, int64_t n, int d, int k, float *C, int32_t *__restrict__ labels, double *bufs,
    unsigned int *bar, LoopState *st, double *__restrict__ inertias) {
    extern __shared__ double fu_sm[];
    double *S_s = fu_sm;                                    // [k][d]
    double *Q_s = S_s + (size_t)k * d;                      // [k]
    float *C_s = reinterpret_cast<float *>(Q_s + k);        // [k][DP], zero beyond d
    int32_t *c_s = reinterpret_cast<int32_t *>(C_s + (size_t)k * DP);
    int32_t *mem = c_s + k;                                 // members of the chunk per center
    int32_t *off = mem + k;                                 // their first place in order
    float *dev = reinterpret_cast<float *>(off + k + 1);    // [frame][stride]: deviations, squared length
    const int stride = fu_stride(d);
    uint16_t *order = reinterpret_cast<uint16_t *>(dev + kFuThreads * stride);
    __shared__ double red[kFuThreads / 32];
    const int tid = threadIdx.x, lane = tid & 31;
    const size_t bd = fu_buf_doubles(d, k);
    const int max_it = st->max_it;
    const double tol = st->tol;
    double prev = st->prev;
    for (int e = tid; e < k * DP; e += kFuThreads) {
        const int j = e / DP, f = e - j * DP;
        C_s[e] = f < d ? C[(int64_t)j * d + f] : 0.0f;
    }
    bool ok = true;
    int it = 0, conv = 0;
    for (; it < max_it && !conv; ++it) {
        double *S = bufs + (size_t)(it % 3) * bd;
        double *Q = S + (size_t)k * d;
        int32_t *cnt_g = reinterpret_cast<int32_t *>(Q + k);
        __syncthreads();  // the last iteration's sums have been added, its centers are complete
        for (int e = tid; e < k * d + k; e += kFuThreads) S_s[e] = 0.0;
        for (int e = tid; e < k; e += kFuThreads) {
            c_s[e] = 0;
            mem[e] = 0;
        }
        __syncthreads();
        for (int64_t c0 = (int64_t)blockIdx.x * kFuThreads; c0 < n; c0 += (int64_t)gridDim.x * kFuThreads) {
            const int64_t i = c0 + tid;
            int lab = -1;
            float *row = dev + tid * stride;
            float x[DP];
            float q = 0.0f;
            if (i < n) {
#pragma unroll
                for (int f = 0; f < DP; ++f) x[f] = f < d ? __ldg(X + i * d + f) : 0.0f;
                // features beyond d add a zero square, which leaves the sum as it is
                float best = __int_as_float(0x7f800000);
                lab = 0;
#pragma unroll 4
                for (int j = 0; j < k; ++j) {
                    const float *c = C_s + j * DP;
                    float a = 0.0f;
#pragma unroll
                    for (int f = 0; f < DP; ++f) a = __fadd_rn(a, sq_term(x[f], c[f]));
                    if (a < best) {
                        best = a;
                        lab = j;
                    }
                }
                labels[i] = lab;
#pragma unroll
                for (int f = 0; f < DP; ++f) {
                    x[f] = f < d ? __fsub_rn(x[f], C_s[lab * DP + f]) : 0.0f;
                    q = __fmaf_rn(x[f], x[f], q);
                }
            }
            const int lab0 = __shfl_sync(0xffffffffu, lab, 0);
            const bool one = __all_sync(0xffffffffu, lab == lab0);
            int rank = 0;
            if (one) {
                if (lab0 >= 0) {
                    // the warp's sums as float pairs (TwoSum of the leading
                    // parts, errors carried)
                    auto add = [&](float v, double *to) {
                        float s = v, c = 0.0f;
#pragma unroll
                        for (int o = 16; o > 0; o >>= 1) {
                            const float s2 = __shfl_xor_sync(0xffffffffu, s, o);
                            const float c2 = __shfl_xor_sync(0xffffffffu, c, o);
                            const float t = __fadd_rn(s, s2);
                            const float bp = __fsub_rn(t, s);
                            const float e = __fadd_rn(__fsub_rn(s, __fsub_rn(t, bp)), __fsub_rn(s2, bp));
                            s = t;
                            c = __fadd_rn(__fadd_rn(c, c2), e);
                        }
                        double w = (double)s + (double)c;
                        if (__any_sync(0xffffffffu, !fu_finite(w))) {
                            double a = (double)v;
#pragma unroll 1
                            for (int o = 16; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
                            if (fu_finite(a)) w = a;
                        }
                        if (lane == 0) atomicAdd(to, w);
                    };
#pragma unroll
                    for (int f = 0; f < DP; ++f)
                        if (f < d) add(x[f], &S_s[lab0 * d + f]);
                    add(q, &Q_s[lab0]);
                    if (lane == 0) atomicAdd(&c_s[lab0], 32);
                }
            } else if (lab >= 0) {
#pragma unroll
                for (int f = 0; f < DP; ++f)
                    if (f < d) row[f] = x[f];
                row[d] = q;
                rank = atomicAdd(&mem[lab], 1);
            }
            const bool sorted = !one && lab >= 0;
            if (!__syncthreads_or(sorted)) continue;  // every warp had one label
            fu_scan(mem, k, off);
            if (sorted) order[off[lab] + rank] = (uint16_t)tid;
            __syncthreads();
            // four lanes (or one) per (center, feature); feature d is the squared length
            const int pairs = k * (d + 1);
            const int ls = 4 * k <= kFuThreads ? 2 : 0, lanes = 1 << ls;
            for (int p0 = 0; p0 < pairs << ls; p0 += kFuThreads) {
                const int p = (p0 + tid) >> ls, h = tid & (lanes - 1);
                const int j = p < pairs ? p / (d + 1) : 0, f = p < pairs ? p - j * (d + 1) : 0;
                const int m = p < pairs ? mem[j] : 0;
                CSum sum;
                for (int e = h; e < m; e += lanes) sum.add(dev[order[off[j] + e] * stride + f]);
                double v = sum.value();
                if (!fu_finite(v)) {
                    double a = 0.0;
                    for (int e = h; e < m; e += lanes) a += (double)dev[order[off[j] + e] * stride + f];
                    if (fu_finite(a)) v = a;
                }
                if (lanes == 4) {
                    v += __shfl_xor_sync(0xffffffffu, v, 1);
                    v += __shfl_xor_sync(0xffffffffu, v, 2);
                }
                if (h == 0 && m > 0) {
                    if (f < d)
                        S_s[j * d + f] += v;
                    else
                        Q_s[j] += v;
                }
            }
            __syncthreads();
            for (int e = tid; e < k; e += kFuThreads) {
                c_s[e] += mem[e];
                mem[e] = 0;
            }
            __syncthreads();
        }
        __syncthreads();
        for (int e = tid; e < k * d; e += kFuThreads)
            if (S_s[e] != 0.0) atomicAdd(&S[e], S_s[e]);
        for (int e = tid; e < k; e += kFuThreads) {
            if (c_s[e]) {
                atomicAdd(&Q[e], Q_s[e]);
                atomicAdd(&cnt_g[e], c_s[e]);
            }
        }
        if (blockIdx.x == 0) {  // the next iteration's buffer
            double *z = bufs + (size_t)((it + 1) % 3) * bd;
            for (size_t e = tid; e < bd; e += kFuThreads) z[e] = 0.0;
        }
        ok = grid_barrier(bar, (unsigned int)(it + 1) * gridDim.x, &st->err);
        if (!ok) break;
        // New centers, a thread per center:
        //   mu_j = c_j + S_j / n_j, inertia_j = Q_j - 2 delta_j.S_j + n_j ||delta_j||^2
        double cost = 0.0;
        for (int j = tid; j < k; j += kFuThreads) {
            const int cnt = __ldcg(cnt_g + j);
            if (cnt == 0) continue;
            const double dc = (double)cnt;
            const double inv = 1.0 / dc;
            double cross = 0.0, sq = 0.0;
#pragma unroll
            for (int f = 0; f < DP; ++f) {
                if (f < d) {
                    const double s = __ldcg(S + (size_t)j * d + f);
                    const double c = (double)C_s[j * DP + f];
                    const float mu = (float)(c + s * inv);
                    const double dl = (double)mu - c;
                    cross += dl * s;
                    sq += dl * dl;
                    C_s[j * DP + f] = mu;
                }
            }
            cost += __ldcg(Q + j) - 2.0 * cross + dc * sq;
        }
        cost = fu_block_sum(cost, red);
        const double rel = cost != 0.0 ? fabs(cost - prev) / cost : 0.0;
        prev = cost;
        conv = rel <= tol ? 1 : 0;
        if (blockIdx.x == 0 && tid == 0) inertias[it] = cost;
    }
    __syncthreads();
    if (blockIdx.x == 0) {
        for (int e = tid; e < k * DP; e += kFuThreads) {
            const int j = e / DP, f = e - j * DP;
            if (f < d) C[(int64_t)j * d + f] = C_s[e];
        }
        if (tid == 0) {
            st->prev = prev;
            st->it = it;
            st->converged = conv;
        }
    }
}

template <int DP>
int launch_dp(const float *X, int64_t n, int d, int k, float *C, int32_t *labels, double *bufs, unsigned int *bar,
              LoopState *st, double *inertias, cudaStream_t s) {
    const size_t smem = fu_smem(d, k);
    static int per_sm_dev[kDeviceSlots] = {};  // CTAs per SM at the largest shared memory
    const int dev = current_device();
    int per_sm = dev >= 0 && dev < kDeviceSlots ? per_sm_dev[dev] : 0;
    if (per_sm <= 0) {
        KM_CUDA(cudaFuncSetAttribute(small_lloyd_kernel<DP>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)kFuMaxSmem));
        int v = 0;
        KM_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&v, small_lloyd_kernel<DP>, kFuThreads, kFuMaxSmem));
        per_sm = v > 0 ? v : 1;
        if (dev >= 0 && dev < kDeviceSlots) per_sm_dev[dev] = per_sm;
    }
    // all CTAs resident at once (they wait for each other): at most two per SM
    const int64_t slots = (int64_t)num_sms() * std::min(per_sm, 2);
    const unsigned grid = (unsigned)std::min<int64_t>(slots, (n + kFuThreads - 1) / kFuThreads);
    void *args[] = {(void *)&X,    (void *)&n,   (void *)&d,  (void *)&k, (void *)&C, (void *)&labels,
                    (void *)&bufs, (void *)&bar, (void *)&st, (void *)&inertias};
    KM_CUDA(cudaLaunchCooperativeKernel((const void *)small_lloyd_kernel<DP>, dim3(grid), dim3(kFuThreads), args,
                                        smem, s));
    return KM_OK;
}

}  // namespace

bool small_lloyd_shape_ok(int d, int k) { return d <= 16 && fu_sums_bytes(d, k) <= kFuSumsMax; }

// Every CTA clears, adds out and re-forms all k centers, whatever its share of
// the frames; with k near n the separate kernels, which spread that over the
// chip, are faster (us per iteration, separate -> here):
//   d = 1, k = 2000:  n = 3,000 38 -> 69, 40,000 65 -> 67, 150,000 162 -> 111
//   d = 4, k = 800:   n = 3,000 42 -> 54, 10,000 48 -> 57, 40,000 86 -> 60
//   d = 16, k = 240:  n = 300 43 -> 52, 1,000 52 -> 56, 3,000 77 -> 58
//   d = 16, k = 100:  n = 300 41 -> 38
bool small_lloyd_ok(int64_t n, int d, int k) {
    return small_lloyd_shape_ok(d, k) && 32.0 * (double)n >= (double)k * k;
}

// Microseconds per iteration of either form, less what they share, fitted to
// d = 2..16, k = 20..1000 and n = 20,000..4,000,000: here n k distances of DP
// features and k (d + 1) sums per CTA; there launches, the packed update and a
// pass over the frames.  Measured (here, narrow):
//   d = 2:   n = 500,000 k = 200 76, 117 and k = 500 161, 119
//   d = 6:   n = 500,000 k = 200 170, 229 and k = 500 366, 240;
//            n = 4,000,000 k = 50 395, 595 and k = 200 1008, 628
//   d = 16:  n = 2,000,000 k = 50 447, 933 and k = 200 1046, 930
bool small_lloyd_beats_narrow(int64_t n, int d, int k) {
    const double here = (double)n * k * (1.7 + 1.2 * fu_dp(d)) * 1e-7 + 0.012 * k * (d + 1);
    return here < 20.0 * (d + 1) + 8e-5 * (double)n;
}

size_t small_lloyd_ws_size(int d, int k) { return 256 + 3 * fu_buf_doubles(d, k) * sizeof(double); }

int launch_small_lloyd(const float *X, int64_t n, int d, int k, float *C, int32_t *labels, void *ws, LoopState *st,
                       double *inertias, cudaStream_t s) {
    // the barrier count in the first word, the rotating sums behind it
    KM_CUDA(cudaMemsetAsync(ws, 0, small_lloyd_ws_size(d, k), s));
    unsigned int *bar = static_cast<unsigned int *>(ws);
    double *bufs = reinterpret_cast<double *>(static_cast<char *>(ws) + 256);
    switch (fu_dp(d)) {
        case 1: return launch_dp<1>(X, n, d, k, C, labels, bufs, bar, st, inertias, s);
        case 2: return launch_dp<2>(X, n, d, k, C, labels, bufs, bar, st, inertias, s);
        case 4: return launch_dp<4>(X, n, d, k, C, labels, bufs, bar, st, inertias, s);
        case 8: return launch_dp<8>(X, n, d, k, C, labels, bufs, bar, st, inertias, s);
        default: return launch_dp<16>(X, n, d, k, C, labels, bufs, bar, st, inertias, s);
    }
}

}  // namespace km
