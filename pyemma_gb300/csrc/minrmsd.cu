// minrmsd.cu -- k-means under the minRMSD metric: assignment, the metric of
// row pairs, kmeans++ and Lloyd iterations (km_*_minrmsd).
//
// Reference: the minRMSD metric plug-in, pyemma/coordinates/clustering/src/
// clustering_module.cpp:9-36, registered into deeptime's clustering and
// reached through cluster_kmeans(metric='minRMSD') / assign_to_centers(
// metric='minRMSD') (pyemma/coordinates/api.py, clustering/kmeans.py:114-115).
// Frames are atom-major rows of d = 3 n_atoms floats.  The squared metric is
// the mean square deviation after optimal superposition (km_rmsd.cuh); the
// label is the lowest index with the smallest msd.  The center update of a
// Lloyd iteration is the mean of the members, as for the Euclidean metric;
// the inertia is the sum of the members' msd to their new centers.
//
// Layout: frames and centers are centered once into float copies with their
// traces G (double).  The centered centers are also stored transposed
// (feature-major, k padded to 32) so that the lanes of a warp, one center
// each, read them coalesced.
//
// Assignment: the double QCP solve is the expensive part of a pair (about 180
// float64 operations, and this part runs two of them per SM and clock), and
// almost every center is far from being the nearest.  So a warp takes several
// frames, every lane the nine float correlation sums of its center with each
// of them, and a float32 bracket of the largest root (qcp_bracket) gives a
// lower and an upper bound of every msd.  Only the centers whose lower bound
// does not exceed the frame's smallest upper bound are solved in double, with
// the same sums and operations as before, so labels and distances are the
// same bit for bit.
#include <algorithm>

#include "km_common.cuh"
#include "km_internal.h"
#include "km_rmsd.cuh"

namespace km {

namespace {

constexpr int kRmsdWarps = 8;  // warps per CTA

// Every row of an (n, d) array centered into Xc, traces into G: a warp per
// row.  For rows that rmsd_center_tile_kernel does not take.
__global__ void __launch_bounds__(kRmsdWarps * 32) rmsd_center_kernel(const float *__restrict__ X, int64_t n, int d,
                                                                      float *__restrict__ Xc, double *__restrict__ G) {
    const int lane = threadIdx.x & 31;
    const int64_t nw = (int64_t)gridDim.x * kRmsdWarps;
    for (int64_t r = (int64_t)blockIdx.x * kRmsdWarps + (threadIdx.x >> 5); r < n; r += nw) {
        const double g = rmsd_center_row_warp(X + r * d, d / 3, Xc + r * d);
        if (lane == 0) G[r] = g;
    }
}

// The same with one thread per row: a warp stages its 32 rows in shared
// memory (coalesced; odd row stride).  The results are those of
// rmsd_center_row_warp bit for bit, with as little float64 work as that
// allows (two float64 lanes per SM and clock here, conversions at the same
// rate):
//   * the sum over an axis: every float64 partial sum is exact while the
//     values span at most 53 - ceil(log2 n_atoms) bits, and then any exact
//     summation gives the same value: each value is cut into three slices
//     whose float32 sums are exact;
//   * a = (float)(x - mean): x - mean to 2^-47 in float pairs; its float
//     rounding is final unless the value lies that close to the middle of two
//     floats, where the float64 form decides;
//   * G: the square of a float is exact in float64, so a fused multiply-add
//     rounds as product and sum; the tree over the 32 partial sums is walked
//     in bit-reversed order with a five-entry stack.
// Rows outside these conditions take the float64 form.  1,000,000 rows of 58
// atoms: 1.5 ms (FP64 pipe 40% busy); 5.9 ms with a warp per row, which
// repeats the divisions and the tree in every lane.
constexpr int kCenterSlicedAtoms = 128;  // a slice's sum of this many values is exact
constexpr int kCenterMaxAtoms = 150;
constexpr int kCenterWarps = 2;          // per CTA: 115 KB of rows at most

int center_stride(int d) { return d | 1; }
size_t center_smem(int d) { return (size_t)kCenterWarps * 32 * center_stride(d) * sizeof(float); }

// The tree of rmsd_center_row_warp (offsets 16, 8, 4, 2, 1) over the 32
// partial sums leaf(l): leaves in bit-reversed order, equal subtrees added as
// soon as both are complete.
template <class Leaf>
__device__ __forceinline__ double rmsd_tree32(const Leaf &leaf) {
    double st[6];  // in local memory: a loop of its own, or every level's addition is made and selected
    double v = 0.0;
#pragma unroll 1
    for (int q = 0; q < 32; ++q) {
        v = leaf((int)(__brev((unsigned)q) >> 27));
        int b = 0;
#pragma unroll 1
        for (; (q >> b) & 1; ++b) v = __dadd_rn(st[b], v);
        st[b] = v;
    }
    return v;
}

// The exact sum of n_atoms values x[0], x[3], ... as a double; false when the
// values span too many bits for the slices (or are not finite).
__device__ __forceinline__ bool rmsd_sliced_sum(const float *x, int n_atoms, double &sum) {
    unsigned hi = 0u, lo = 0xffffffffu;  // bits of the largest, of the smallest non-zero magnitude less one
    for (int i = 0; i < n_atoms; ++i) {
        const unsigned b = __float_as_uint(x[3 * i]) & 0x7fffffffu;
        hi = max(hi, b);
        lo = min(lo, b - 1u);
    }
    sum = 0.0;
    if (hi == 0u) return true;
    const int e = (int)(hi >> 23), el = (int)((lo + 1u) >> 23);
    // |x| < 2^(E + 1), E = e - 127; every x a multiple of 2^(E - 46)
    if (e > 200 || el < 60 || e - el > 23) return false;
    const float m1 = __uint_as_float((unsigned)(e + 8) << 23 | 0x400000u);  // 1.5 2^(E + 8): slice of 2^(E - 15)
    const float m2 = __uint_as_float((unsigned)(e - 9) << 23 | 0x400000u);  // 1.5 2^(E - 9): slice of 2^(E - 32)
    float s1 = 0.0f, s2 = 0.0f, s3 = 0.0f;
    for (int i = 0; i < n_atoms; ++i) {
        const float v = x[3 * i];
        const float h1 = __fsub_rn(__fadd_rn(v, m1), m1);
        const float r1 = __fsub_rn(v, h1);
        const float h2 = __fsub_rn(__fadd_rn(r1, m2), m2);
        const float r2 = __fsub_rn(r1, h2);
        s1 = __fadd_rn(s1, h1);
        s2 = __fadd_rn(s2, h2);
        s3 = __fadd_rn(s3, r2);
    }
    sum = __dadd_rn(__dadd_rn((double)s1, (double)s2), (double)s3);
    return true;
}

// The float64 forms, out of line: inlined, the compiler computes them for
// every value and selects.
__device__ __noinline__ float rmsd_center_value_d(float x, double mean) {
    return __double2float_rn(__dsub_rn((double)x, mean));
}
__device__ __noinline__ double rmsd_widen_d(float v) { return (double)v; }

// (float)(x - mean) as double subtraction and conversion give it; mh + ml is
// mean to 2^-49.
__device__ __forceinline__ float rmsd_center_value(float x, double mean, float mh, float ml) {
    // x - mh = s + e exactly, t = e - ml, s + t = v + r exactly
    const float s = __fsub_rn(x, mh);
    const float bb = __fsub_rn(s, x);
    const float e = __fsub_rn(__fsub_rn(x, __fsub_rn(s, bb)), __fadd_rn(mh, bb));
    const float t = __fsub_rn(e, ml);
    const float v = __fadd_rn(s, t);
    const float tv = __fsub_rn(v, s);
    const float r = __fadd_rn(__fsub_rn(s, __fsub_rn(v, tv)), __fsub_rn(t, tv));
    const unsigned b = __float_as_uint(v);
    const float half = __uint_as_float((b & 0x7f800000u) - (24u << 23));  // half a unit in the last place
    const float tol = 1.42e-14f * (fabsf(s) + fabsf(mh));                 // 2^-46
    const bool sure = (b & 0x7f800000u) > (60u << 23) && (b & 0x7fffffu) != 0u && half - fabsf(r) > tol;
    if (!sure) return rmsd_center_value_d(x, mean);
    return v;
}

// (double)v without the conversion unit.
__device__ __forceinline__ double rmsd_widen(float v) {
    const unsigned b = __float_as_uint(v), a = b & 0x7fffffffu;
    if (a - 0x800000u >= 0x7f000000u) return rmsd_widen_d(v);  // zero, subnormal, infinite, NaN
    return __hiloint2double((int)((b & 0x80000000u) | ((a >> 3) + 0x38000000u)), (int)(b << 29));
}

__global__ void __launch_bounds__(kCenterWarps * 32) rmsd_center_tile_kernel(const float *__restrict__ X, int64_t n, int d,
                                                              int stride, float *__restrict__ Xc,
                                                              double *__restrict__ G) {
    extern __shared__ float center_rows_s[];
    const int lane = threadIdx.x & 31;
    float *rows = center_rows_s + (size_t)(threadIdx.x >> 5) * 32 * stride;
    const int n_atoms = d / 3;
    const int64_t tiles = (n + 31) / 32;
    for (int64_t tile = (int64_t)blockIdx.x * kCenterWarps + (threadIdx.x >> 5); tile < tiles;
         tile += (int64_t)gridDim.x * kCenterWarps) {
        const int64_t r0 = tile * 32;
        const int m = (int)(n - r0 < 32 ? n - r0 : 32);
        // the tile's rows are consecutive floats; eight loads in flight per lane
        const float *src = X + r0 * d;
        const int total = m * d;
        int f = lane % d, r = lane / d;
        for (int e0 = lane; e0 < total; e0 += 256) {
            float v[8];
#pragma unroll
            for (int q = 0; q < 8; ++q) v[q] = e0 + 32 * q < total ? __ldg(src + e0 + 32 * q) : 0.0f;
#pragma unroll
            for (int q = 0; q < 8; ++q) {
                if (e0 + 32 * q < total) rows[r * stride + f] = v[q];
                f += 32;
                while (f >= d) {
                    f -= d;
                    ++r;
                }
            }
        }
        __syncwarp();
        if (lane < m) {
            float *x = rows + lane * stride;
            double mean[3];
            float mh[3], ml[3];
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                double sum;
                if (n_atoms > kCenterSlicedAtoms || !rmsd_sliced_sum(x + c, n_atoms, sum))
                    sum = rmsd_tree32([&](int l) {
                        double acc = 0.0;
                        for (int i = l; i < n_atoms; i += 32) acc = __dadd_rn(acc, (double)x[3 * i + c]);
                        return acc;
                    });
                mean[c] = __ddiv_rn(sum, (double)n_atoms);
                mh[c] = __double2float_rn(mean[c]);
                ml[c] = __double2float_rn(__dsub_rn(mean[c], (double)mh[c]));
            }
            G[r0 + lane] = rmsd_tree32([&](int l) {
                double acc = 0.0;
                for (int i = l; i < n_atoms; i += 32) {
#pragma unroll
                    for (int c = 0; c < 3; ++c) {
                        const float v = rmsd_center_value(x[3 * i + c], mean[c], mh[c], ml[c]);
                        x[3 * i + c] = v;
                        const double w = rmsd_widen(v);
                        acc = __fma_rn(w, w, acc);
                    }
                }
                return acc;
            });
        }
        __syncwarp();
        f = lane % d;
        r = lane / d;
        for (int e = lane; e < total; e += 32) {
            Xc[r0 * d + e] = rows[r * stride + f];
            f += 32;
            while (f >= d) {
                f -= d;
                ++r;
            }
        }
        __syncwarp();
    }
}

// The centers by groups of 32 lanes: Ct[(g * n_atoms + i) * 96 + 32 c + l] =
// coordinate c of atom i of center 32 g + l; zero for the padding centers.
__global__ void rmsd_transpose_kernel(const float *__restrict__ Cc, int k, int kp, int d, float *__restrict__ Ct) {
    const int64_t total = (int64_t)kp * d;
    for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < total; e += (int64_t)gridDim.x * blockDim.x) {
        const int f = (int)((e >> 5) % d);  // feature 3 i + c
        const int j = (int)((e >> 5) / d) * 32 + (int)(e & 31);
        Ct[e] = j < k ? Cc[(int64_t)j * d + f] : 0.0f;
    }
}

// (msd, index) of the better of two candidates: a number beats NaN or no
// candidate (index < 0), then the smaller msd, then the lower index.
__device__ __forceinline__ bool rmsd_better(double m, int j, double bm, int bj) {
    if (j < 0 || m != m) return false;
    if (bj < 0) return true;
    return m < bm || (m == bm && j < bj);
}

// The nearest center of one frame with every pair solved in double, by one
// warp (lanes own centers); (msd, index) in every lane.
__device__ __noinline__ void rmsd_full_frame(const float *__restrict__ a, double ga, int n_atoms,
                                             const float *__restrict__ Ct, const double *__restrict__ H, int k,
                                             int lane, double &bm, int &bj) {
    bm = 0.0;
    bj = -1;
    for (int j0 = 0; j0 < k; j0 += 32) {
        const int j = j0 + lane;  // j < kp: the padding centers are zero rows
        float S[9];
#pragma unroll
        for (int e = 0; e < 9; ++e) S[e] = 0.0f;
        const float *b = Ct + (int64_t)j0 * 3 * n_atoms + lane;
        for (int i = 0; i < n_atoms; ++i, b += 96) {
            const float a0 = a[3 * i], a1 = a[3 * i + 1], a2 = a[3 * i + 2];
            const float b0 = b[0], b1 = b[32], b2 = b[64];
            S[0] = __fmaf_rn(a0, b0, S[0]);
            S[1] = __fmaf_rn(a0, b1, S[1]);
            S[2] = __fmaf_rn(a0, b2, S[2]);
            S[3] = __fmaf_rn(a1, b0, S[3]);
            S[4] = __fmaf_rn(a1, b1, S[4]);
            S[5] = __fmaf_rn(a1, b2, S[5]);
            S[6] = __fmaf_rn(a2, b0, S[6]);
            S[7] = __fmaf_rn(a2, b1, S[7]);
            S[8] = __fmaf_rn(a2, b2, S[8]);
        }
        if (j < k) {
            const double m = qcp_msd(S, ga, H[j], n_atoms);
            if (rmsd_better(m, j, bm, bj)) {
                bm = m;
                bj = j;
            }
        }
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
        const double om = __shfl_xor_sync(0xffffffffu, bm, off);
        const int oj = __shfl_xor_sync(0xffffffffu, bj, off);
        if (rmsd_better(om, oj, bm, bj)) {
            bm = om;
            bj = oj;
        }
    }
}

__device__ __forceinline__ void rmsd_store(int64_t r, double bm, int bj, int32_t *__restrict__ labels,
                                           float *__restrict__ rmsd) {
    labels[r] = bj < 0 ? 0 : bj;
    if (rmsd) rmsd[r] = bj < 0 ? __int_as_float(0x7fc00000) : __double2float_rn(sqrt(bm));
}

// One warp per frame, every pair solved in double.  Always for one or two
// atoms, whose correlation matrices have rank at most one: the largest root is
// then a double root, and qcp_bracket never holds.
__global__ void __launch_bounds__(kRmsdWarps * 32) rmsd_assign_full_kernel(
    const float *__restrict__ Xc, const double *__restrict__ G, int64_t n, int d, const float *__restrict__ Ct,
    const double *__restrict__ H, int k, int32_t *__restrict__ labels, float *__restrict__ rmsd) {
    const int lane = threadIdx.x & 31;
    const int64_t nw = (int64_t)gridDim.x * kRmsdWarps;
    for (int64_t r = (int64_t)blockIdx.x * kRmsdWarps + (threadIdx.x >> 5); r < n; r += nw) {
        double bm;
        int bj;
        rmsd_full_frame(Xc + r * d, G[r], d / 3, Ct, H, k, lane, bm, bj);
        if (lane == 0) rmsd_store(r, bm, bj, labels, rmsd);
    }
}

// A bracket of E = Ga + Gb - 2 lambda (n_atoms times the msd before it is
// clipped at 0) from the correlation sums S in float32: lb <= E_qcp <= ub for
// the lambda that qcp_msd finds.  tot: Ga + Gb rounded to float (within 3 u).
//
// With s = ||S||_F and T = S / s the quartic of the key matrix is
//   P(x) = x^4 - 2 x^2 - 8 det(T) x + (2 ||T T^t||_F^2 - 1),
// lambda = s x for its largest root x <= sqrt(3).  (Its constant term is the
// product of the key matrix's eigenvalues.)  u = 2^-24.  ||T||^2 = 1 within
// 20 u; the float values of the coefficients are off by at most 40 u, 64 u
// and 75 u, and P at 0 < x <= 1.75 by at most 120 + 110 + 75 + 45 = 350 u:
// kQcpErr allows 512 u.  All roots are real, so
//   P(x) > 0, P'(x) > 0, P''(x) > 0 (x > 0.6)  =>  x is above every root;
//   P(x) < 0                                   =>  x is below the largest.
// Both tests are made on the float value with the margin kQcpErr.  The
// roundings of s, T and of E itself are below kQcpSlack tot = 64 u tot.
//
// qcp_msd's double Newton ends at the largest root (within 1e-9 of s) when
// that root is well separated: P' there is 8 (a + b)(a + c)(b + c) for the
// singular values a >= b >= |c| of T, c with the sign of det(T).  well says
// that it is 1e-5 at least, from
//   a^2 (b + c)^2 >= ||cof T||^2 - det^2 / a^2 - 2 a |det|   (det < 0)
// with ||T T^t||_F^2 <= a^2 <= ||T T^t||_F and ||cof T||^2 = (1 - ||T
// T^t||_F^2) / 2 (for det >= 0 the first term alone bounds b + c).  Measured
// on random-walk chains: 99% of the pairs.
// Where a test fails (an ill-conditioned root, sums outside the range in
// which qcp_msd's float reciprocal is normal, a value that is not finite) the
// bound is 0 or infinity and the pair is solved in double.
struct QcpQuartic {
    float s, C1, C0;
    bool well;  // the double solve ends at the largest root
    __device__ __forceinline__ void eval(float x, float &P, float &D) const {
        const float l2 = x * x;
        const float a2 = l2 - 2.0f;
        P = fmaf(a2, l2, fmaf(C1, x, C0));
        D = fmaf(2.0f * x, l2 + a2, C1);
    }
};

constexpr float kQcpErr = 512.0f * 5.9604645e-8f;
constexpr float kQcpSlack = 64.0f * 5.9604645e-8f;

__device__ __forceinline__ QcpQuartic qcp_quartic(const float (&S)[9], float tot) {
    float ss = 0.0f;
#pragma unroll
    for (int e = 0; e < 9; ++e) ss = fmaf(S[e], S[e], ss);
    const float rs = rsqrtf(ss);
    float T[9];
#pragma unroll
    for (int e = 0; e < 9; ++e) T[e] = S[e] * rs;
    const float m0 = fmaf(T[4], T[8], -T[5] * T[7]);
    const float m1 = fmaf(T[3], T[8], -T[5] * T[6]);
    const float m2 = fmaf(T[3], T[7], -T[4] * T[6]);
    const float b00 = fmaf(T[0], T[0], fmaf(T[1], T[1], T[2] * T[2]));
    const float b11 = fmaf(T[3], T[3], fmaf(T[4], T[4], T[5] * T[5]));
    const float b22 = fmaf(T[6], T[6], fmaf(T[7], T[7], T[8] * T[8]));
    const float b01 = fmaf(T[0], T[3], fmaf(T[1], T[4], T[2] * T[5]));
    const float b02 = fmaf(T[0], T[6], fmaf(T[1], T[7], T[2] * T[8]));
    const float b12 = fmaf(T[3], T[6], fmaf(T[4], T[7], T[5] * T[8]));
    const float diag = fmaf(b00, b00, fmaf(b11, b11, b22 * b22));
    const float offd = fmaf(b01, b01, fmaf(b02, b02, b12 * b12));
    QcpQuartic q;
    q.s = ss * rs;
    q.C1 = -8.0f * fmaf(T[0], m0, fmaf(T[2], m2, -T[1] * m1));
    q.C0 = fmaf(2.0f, fmaf(2.0f, offd, diag), -1.0f);
    const float nb = 0.5f * (q.C0 + 1.0f);
    const float det = fmaxf(0.125f * q.C1, 0.0f) + 2e-6f;  // of a negative determinant, its size
    const float sep = fmaf(0.25f, 1.0f - q.C0, -__fdividef(det * det, nb)) - 2.0f * det * sqrtf(sqrtf(nb));
    q.well = sep >= 2e-5f && ss >= 1e-22f && ss <= 1e30f && tot <= 1e37f;
    return q;
}

// True when E_qcp > best is certain: the point x at which E would be best
// (less the slack) is above every root (sqrt(3) always is).
__device__ __forceinline__ bool qcp_beyond(const QcpQuartic &q, float tot, float best) {
    const float x = fminf(__fdividef(0.5f * (tot - best - 2.0f * kQcpSlack * tot), q.s), 1.74f);
    float P, D;
    q.eval(x, P, D);
    return q.well && x > 0.6f && (x == 1.74f || (P > kQcpErr && D >= 1e-3f));
}

// The bracket at the point that eight Newton steps from above reach.
__device__ __forceinline__ void qcp_bracket(const QcpQuartic &q, float tot, float &lb, float &ub) {
    lb = 0.0f;
    ub = __int_as_float(0x7f800000);
    float x = fminf(1.7320509f, __fdividef(0.500001f * tot, q.s));
    float P, D;
#pragma unroll
    for (int it = 0; it < 8; ++it) {
        q.eval(x, P, D);
        x -= __fdividef(P, D);
    }
    q.eval(x, P, D);
    const float inv = __fdividef(1.0f, D);
    const float xu = x + fmaf(fmaxf(-P, 0.0f), 1.01f * inv, 2.5f * kQcpErr * inv);
    const float xl = x - fmaf(fmaxf(P, 0.0f), 1.01f * inv, 2.5f * kQcpErr * inv);
    q.eval(xu, P, D);
    if (q.well && xu > 0.6f && xu < 1.75f && P > kQcpErr && D >= 1e-3f)
        lb = fmaxf(fmaf(-2.0f * xu, q.s, tot) - kQcpSlack * tot, 0.0f);
    q.eval(xl, P, D);
    if (q.well && xl > 0.0f && xl < 1.75f && P < -kQcpErr)
        ub = fmaxf(fmaf(-2.0f * xl, q.s, tot) + kQcpSlack * tot, 0.0f);
}

// Two float32 fused multiply-adds in one instruction.
__device__ __forceinline__ void fma2(unsigned long long &d, unsigned long long a, unsigned long long b) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(a), "l"(b));
}
__device__ __forceinline__ unsigned long long pack2(float lo, float hi) {
    unsigned long long v;
    asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "f"(lo), "f"(hi));
    return v;
}
__device__ __forceinline__ void unpack2(unsigned long long v, float &lo, float &hi) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}

// The assignment: a warp takes F frames at a time and walks the centers in
// groups of 32, one per lane.  The frames' coordinates lie in shared memory
// atom by atom with the F frames side by side, so that one broadcast load
// serves two frames' packed multiply-adds; each center coordinate, read once
// from L1/L2, serves all F frames (9 F multiply-adds per 3 loads).
// Per frame a list of the centers whose lower bound does not exceed the
// smallest upper bound so far, with their correlation sums; at the end the
// lists of all F frames are solved in double, one entry per lane.  Pairs
// without a bracket (1%) fill the lists of large center sets: there a list more
// than half full is solved after a group of centers (k = 1000, 58 atoms: 64,000
// frames 5.2 -> 2.6 ms, 1,000 frames 1.38 -> 0.46).  A frame with many near-ties
// has all its pairs solved in double.
// Bound by the FP32 pipe: 9 n_atoms multiply-adds and about 140 operations of
// the bracket per pair, with three warps in four waiting (ncu, 200,000 frames:
// issue slots 40% busy, FP32 pipe 34%, FP64 pipe 33%).  1,000,000 frames of
// 58 atoms, k = 100: 5.9 ms; solving every pair in double took 68.6 ms.
// Four frames per warp, 24 warps per SM: 7.7 ms the whole call; eight frames reuse each
// center coordinate twice as often but leave 16 warps per SM (126 registers)
// and twice the code after the sums: 9.3 ms.
constexpr int kRmsdFrames = 4;
constexpr int kRmsdAtoms = 96;  // atoms staged at a time
constexpr int kRmsdList = 8;    // candidates kept per frame
constexpr int kRmsdMany = 128;  // centers from which lists are solved on the way

template <int F>
struct RmsdWarpSmem {
    // [atom][axis][frame]; the row of 3 F floats is padded by 4 (fewer store conflicts)
    float a[kRmsdAtoms][3 * F + 4];
    float S[F][kRmsdList][9];
    float lb[F][kRmsdList];
    int32_t j[F][kRmsdList];
    double ga[F];
    double bm[F];     // the best of the entries solved so far
    int32_t bj[F];    // (-1: none)
    int32_t cnt[F];   // entries listed
    int32_t room[F];  // times that a full list may still be solved in between
    int32_t full[F];  // every pair is solved
};

// Solves the entries of frame f's list, one per lane, into its best so far, and
// empties the list.
template <int F>
__device__ __noinline__ void rmsd_solve_list(RmsdWarpSmem<F> &sm, int f, const double *__restrict__ H, int n_atoms) {
    const int lane = threadIdx.x & 31;
    const int cnt = sm.cnt[f];
    double m = 0.0;
    int j = -1;
    if (lane < cnt) {
        float S[9];
#pragma unroll
        for (int e = 0; e < 9; ++e) S[e] = sm.S[f][lane][e];
        j = sm.j[f][lane];
        m = qcp_msd(S, sm.ga[f], H[j], n_atoms);
    }
#pragma unroll
    for (int off = kRmsdList / 2; off > 0; off >>= 1) {
        const double om = __shfl_xor_sync(0xffffffffu, m, off);
        const int oj = __shfl_xor_sync(0xffffffffu, j, off);
        if (rmsd_better(om, oj, m, j)) {
            m = om;
            j = oj;
        }
    }
    __syncwarp();
    if (lane == 0) {
        if (rmsd_better(m, j, sm.bm[f], sm.bj[f])) {
            sm.bm[f] = m;
            sm.bj[f] = j;
        }
        sm.cnt[f] = 0;
        --sm.room[f];
    }
    __syncwarp();
}

// Brackets one frame's pairs with the warp's 32 centers, lists the ones that
// the smallest upper bound (returned) does not rule out.  Out of line: few
// groups of centers need it, and a copy per frame would not stay in the
// instruction cache.
template <int F>
__device__ __noinline__ float rmsd_candidates(RmsdWarpSmem<F> &sm, int f, const float (&S)[9], QcpQuartic qu,
                                              float tot, float best, int j, int k) {
    const int lane = threadIdx.x & 31;
    const float kInf = __int_as_float(0x7f800000);
    float lb, ub;
    qcp_bracket(qu, tot, lb, ub);
    if (j >= k) ub = kInf;
    // non-negative floats order as their bits
    best = fminf(best, __uint_as_float(__reduce_min_sync(0xffffffffu, __float_as_uint(ub))));
    const unsigned cand = __ballot_sync(0xffffffffu, j < k && lb <= best);
    if (cand == 0u) return best;
    // When the list would run over, first drop the entries that the bound
    // rules out by now.
    int cnt = sm.cnt[f];
    if (cnt + __popc(cand) > kRmsdList) {
        float l = kInf, Sl[9];
        int jl = -1;
        if (lane < cnt) {
            l = sm.lb[f][lane];
            jl = sm.j[f][lane];
#pragma unroll
            for (int e = 0; e < 9; ++e) Sl[e] = sm.S[f][lane][e];
        }
        const unsigned keep = __ballot_sync(0xffffffffu, lane < cnt && l <= best);
        __syncwarp();
        if ((keep >> lane) & 1u) {
            const int to = __popc(keep & ((1u << lane) - 1u));
            sm.lb[f][to] = l;
            sm.j[f][to] = jl;
#pragma unroll
            for (int e = 0; e < 9; ++e) sm.S[f][to][e] = Sl[e];
        }
        cnt = __popc(keep);
        __syncwarp();
    }
    if ((cand >> lane) & 1u) {
        const int to = cnt + __popc(cand & ((1u << lane) - 1u));
        if (to < kRmsdList) {
            sm.lb[f][to] = lb;
            sm.j[f][to] = j;
#pragma unroll
            for (int e = 0; e < 9; ++e) sm.S[f][to][e] = S[e];
        }
    }
    __syncwarp();
    if (lane == 0) {
        sm.cnt[f] = min(cnt + __popc(cand), kRmsdList);
        if (cnt + __popc(cand) > kRmsdList) sm.full[f] = 1;
    }
    __syncwarp();
    return best;
}

template <int F>
__global__ void __launch_bounds__(kRmsdWarps * 32, 3) rmsd_assign_kernel(
    const float *__restrict__ Xc, const double *__restrict__ G, int64_t n, int d, const float *__restrict__ Ct,
    const double *__restrict__ H, int k, int32_t *__restrict__ labels, float *__restrict__ rmsd) {
    static_assert(F % 4 == 0, "frames go in fours (16-byte shared loads)");
    extern __shared__ __align__(16) unsigned char rmsd_smem[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    RmsdWarpSmem<F> &sm = reinterpret_cast<RmsdWarpSmem<F> *>(rmsd_smem)[warp];
    const int n_atoms = d / 3;
    const int64_t tiles = (n + F - 1) / F;
    const float kInf = __int_as_float(0x7f800000);
    auto stage = [&](int64_t r0, int i0, int cnt) {
        __syncwarp();
        for (int i = lane; i < cnt; i += 32)
#pragma unroll
            for (int f = 0; f < F; ++f) {
                const bool in = r0 + f < n;
                const float *src = Xc + (in ? r0 + f : r0) * d + 3 * (i0 + i);
#pragma unroll
                for (int c = 0; c < 3; ++c) sm.a[i][c * F + f] = __ldg(src + c);
            }
        __syncwarp();
    };
    for (int64_t t = (int64_t)blockIdx.x * kRmsdWarps + warp; t < tiles; t += (int64_t)gridDim.x * kRmsdWarps) {
        const int64_t r0 = t * F;
        if (n_atoms <= kRmsdAtoms) stage(r0, 0, n_atoms);
        if (lane < F) {
            sm.ga[lane] = G[r0 + lane < n ? r0 + lane : r0];
            sm.bj[lane] = -1;
            sm.cnt[lane] = 0;
            sm.room[lane] = 1 + k / 64;  // half of what solving every pair takes
            sm.full[lane] = 0;
        }
        __syncwarp();
        float best[F];  // smallest upper bound so far
#pragma unroll
        for (int f = 0; f < F; ++f) best[f] = kInf;
        for (int j0 = 0; j0 < k; j0 += 32) {
            const int j = j0 + lane;  // j < kp: the padding centers are zero rows
            unsigned long long S2[F / 2][9];
#pragma unroll
            for (int q = 0; q < F / 2; ++q)
#pragma unroll
                for (int e = 0; e < 9; ++e) S2[q][e] = 0ull;
            for (int i0 = 0; i0 < n_atoms; i0 += kRmsdAtoms) {
                const int cnt = min(kRmsdAtoms, n_atoms - i0);
                if (n_atoms > kRmsdAtoms) stage(r0, i0, cnt);
                // the next atom's center coordinates are loaded one step ahead
                const float *b = Ct + ((int64_t)(j0 >> 5) * n_atoms + i0) * 96 + lane;
                float nb[3] = {__ldg(b), __ldg(b + 32), __ldg(b + 64)};
#pragma unroll 2
                for (int i = 0; i < cnt; ++i) {
                    unsigned long long bb[3];
#pragma unroll
                    for (int c = 0; c < 3; ++c) bb[c] = pack2(nb[c], nb[c]);
                    if (i + 1 < cnt) b += 96;
#pragma unroll
                    for (int c = 0; c < 3; ++c) nb[c] = __ldg(b + 32 * c);
#pragma unroll
                    for (int c = 0; c < 3; ++c)
#pragma unroll
                        for (int q = 0; q < F / 4; ++q) {
                            const ulonglong2 av = *reinterpret_cast<const ulonglong2 *>(&sm.a[i][c * F + 4 * q]);
#pragma unroll
                            for (int e = 0; e < 3; ++e) {
                                fma2(S2[2 * q][3 * c + e], av.x, bb[e]);
                                fma2(S2[2 * q + 1][3 * c + e], av.y, bb[e]);
                            }
                        }
                }
            }
            const float hj = j < k ? (float)H[j] : 0.0f;
#pragma unroll
            for (int q = 0; q < F / 2; ++q) {
                float Sp[2][9];
#pragma unroll
                for (int e = 0; e < 9; ++e) unpack2(S2[q][e], Sp[0][e], Sp[1][e]);
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int f = 2 * q + h;
                    const float tot = (float)sm.ga[f] + hj;
                    const QcpQuartic qu = qcp_quartic(Sp[h], tot);
                    // one evaluation of the quartic rules out most centers
                    // once the frame has a bound
                    if (__all_sync(0xffffffffu, j >= k || qcp_beyond(qu, tot, best[f]))) continue;
                    best[f] = rmsd_candidates<F>(sm, f, Sp[h], qu, tot, best[f], j, k);
                }
            }
            // here, where no sums are held, and not inside rmsd_candidates,
            // whose calls would then spill them (4% of 1M x 58, k = 100)
            if (k > kRmsdMany)
                for (int f = 0; f < F; ++f)
                    if (sm.cnt[f] > kRmsdList / 2 && sm.room[f] > 0 && !sm.full[f])
                        rmsd_solve_list<F>(sm, f, H, n_atoms);
        }
        // Lane f < F keeps frame f's best; lane e solves entry e of the
        // frames' lists laid end to end.
        float my_best = kInf;
#pragma unroll
        for (int f = 0; f < F; ++f)
            if (lane == f) my_best = best[f];
        const bool mine = lane < F && r0 + lane < n && !sm.full[lane < F ? lane : 0];
        const int my_cnt = mine ? sm.cnt[lane] : 0;
        int end = my_cnt;
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, end, off);
            if (lane >= off) end += y;
        }
        const int total = __shfl_sync(0xffffffffu, end, 31);
        double bm = lane < F ? sm.bm[lane] : 0.0;  // read where bj >= 0
        int bj = lane < F ? sm.bj[lane] : -1;
        for (int e0 = 0; e0 < total; e0 += 32) {
            const int e = e0 + lane;
            // the frame whose range holds e
            int f = 0;
#pragma unroll
            for (int q = 0; q < F; ++q) f += e >= __shfl_sync(0xffffffffu, end, q) ? 1 : 0;
            const int first = __shfl_sync(0xffffffffu, end - my_cnt, f < F ? f : 0);
            const float ubf = __shfl_sync(0xffffffffu, my_best, f < F ? f : 0);
            double m = 0.0;
            int j = -1;
            if (e < total) {
                const int slot = e - first;
                if (sm.lb[f][slot] <= ubf) {
                    j = sm.j[f][slot];
                    float S[9];
#pragma unroll
                    for (int q = 0; q < 9; ++q) S[q] = sm.S[f][slot][q];
                    m = qcp_msd(S, sm.ga[f], H[j], n_atoms);
                }
            }
            // every frame's lane collects its entries of this round
            for (int q = 0; q < 32; ++q) {
                const double om = __shfl_sync(0xffffffffu, m, q);
                const int oj = __shfl_sync(0xffffffffu, j, q);
                const int x = e0 + q;
                if (x >= total) break;
                if (x >= end - my_cnt && x < end && rmsd_better(om, oj, bm, bj)) {
                    bm = om;
                    bj = oj;
                }
            }
        }
        if (mine) rmsd_store(r0 + lane, bm, bj, labels, rmsd);
        for (int f = 0; f < F; ++f) {
            if (!sm.full[f] || r0 + f >= n) continue;
            double fm;
            int fj;
            rmsd_full_frame(Xc + (r0 + f) * d, sm.ga[f], n_atoms, Ct, H, k, lane, fm, fj);
            if (lane == 0) rmsd_store(r0 + f, fm, fj, labels, rmsd);
        }
        __syncwarp();
    }
}

// rmsd[i] = sqrt(msd(A[i], B[i])) of centered row pairs.
__global__ void rmsd_rows_kernel(const float *__restrict__ A, const double *__restrict__ GA,
                                 const float *__restrict__ B, const double *__restrict__ GB, int64_t n, int d,
                                 float *__restrict__ out) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        out[i] = __double2float_rn(sqrt(rmsd_msd_rows(A + i * d, B + i * d, GA[i], GB[i], d / 3)));
}

// cost += sum_i msd(frame i, center labels[i]).
__global__ void __launch_bounds__(256) rmsd_cost_kernel(const float *__restrict__ Xc, const double *__restrict__ G,
                                                        int64_t n, int d, const int32_t *__restrict__ labels,
                                                        const float *__restrict__ Cc, const double *__restrict__ H,
                                                        double *__restrict__ cost) {
    __shared__ double red[8];
    double s = 0.0;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const int j = labels[i];
        s += rmsd_msd_rows(Xc + i * d, Cc + (int64_t)j * d, G[i], H[j], d / 3);
    }
    for (int off = 16; off > 0; off >>= 1) s += __shfl_xor_sync(0xffffffffu, s, off);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = 0.0;
        for (int w = 0; w < 8; ++w) t += red[w];
        atomicAdd(cost, t);
    }
}

unsigned rmsd_grid(int64_t warps_needed) {
    int64_t g = (warps_needed + kRmsdWarps - 1) / kRmsdWarps;
    const int64_t cap = (int64_t)num_sms() * 8;
    if (g > cap) g = cap;
    return (unsigned)(g < 1 ? 1 : g);
}

int kp_of_k(int k) { return (k + 31) / 32 * 32; }

struct RmsdCenters {
    float *Cc;
    double *H;
    float *Ct;
};

RmsdCenters carve_centers(Carver &c, int d, int k) {
    RmsdCenters r;
    r.Cc = c.take<float>((size_t)k * d);
    r.H = c.take<double>((size_t)k);
    r.Ct = c.take<float>((size_t)kp_of_k(k) * d);
    return r;
}

int check_rmsd_shape(int64_t n, int d, int k) {
    KM_TRY(check_shape(n, d, k));
    if (d % 3 != 0) {
        set_error("the minRMSD metric needs atom-major rows of 3 n_atoms floats (d=%d is not divisible by 3)", d);
        return KM_ERR_BAD_SHAPE;
    }
    return KM_OK;
}

int center_rows(const float *X, int64_t n, int d, float *Xc, double *G, cudaStream_t s) {
    if (n == 0) return KM_OK;
    // A warp per row while the rows (centers, short calls) give every SM no
    // more than a few tiles: the thread-per-row form takes 0.18 ms for one
    // tile.  And for long rows, of which few fit beside each other (us for twice n
    // rows and their distances, thread per row, warp per row: n = 100,000, 58
    // atoms 422, 1291; 100 1101, 2696; 140 1874, 2152; 200 4419, 2808; 400
    // 15,661, 4877; n = 20,000, 100 atoms 331, 587; 140 603, 485).
    const int64_t tiles_from = (int64_t)num_sms() * (d <= 3 * kCenterSlicedAtoms ? 128 : 512);
    if (d <= 3 * kCenterMaxAtoms && n >= tiles_from) {
        static bool attr_done[kDeviceSlots] = {};
        const int dev = current_device();
        if (dev < 0 || dev >= kDeviceSlots || !attr_done[dev]) {
            KM_CUDA(cudaFuncSetAttribute(rmsd_center_tile_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)center_smem(3 * kCenterMaxAtoms)));
            if (dev >= 0 && dev < kDeviceSlots) attr_done[dev] = true;
        }
        int64_t g = ((n + 31) / 32 + kCenterWarps - 1) / kCenterWarps;
        const int64_t cap = (int64_t)num_sms() * 16;
        if (g > cap) g = cap;
        rmsd_center_tile_kernel<<<(unsigned)g, kCenterWarps * 32, center_smem(d), s>>>(X, n, d, center_stride(d), Xc,
                                                                                        G);
    } else {
        rmsd_center_kernel<<<rmsd_grid(n), kRmsdWarps * 32, 0, s>>>(X, n, d, Xc, G);
    }
    KM_CUDA(cudaGetLastError());
    return KM_OK;
}

int prepare_centers(const float *C, int d, int k, const RmsdCenters &rc, cudaStream_t s) {
    KM_TRY(center_rows(C, k, d, rc.Cc, rc.H, s));
    const int kp = kp_of_k(k);
    int64_t g = ((int64_t)kp * d + 255) / 256;
    const int64_t cap = (int64_t)num_sms() * 8;
    if (g > cap) g = cap;
    rmsd_transpose_kernel<<<(unsigned)(g < 1 ? 1 : g), 256, 0, s>>>(rc.Cc, k, kp, d, rc.Ct);
    KM_CUDA(cudaGetLastError());
    return KM_OK;
}

template <int F>
int launch_rmsd_assign_f(const float *Xc, const double *G, int64_t n, int d, const RmsdCenters &rc, int k,
                         int32_t *labels, float *rmsd, cudaStream_t s) {
    const size_t smem = sizeof(RmsdWarpSmem<F>) * kRmsdWarps;
    static bool attr_done[kDeviceSlots] = {};
    const int dev = current_device();
    if (dev < 0 || dev >= kDeviceSlots || !attr_done[dev]) {
        KM_CUDA(cudaFuncSetAttribute(rmsd_assign_kernel<F>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        if (dev >= 0 && dev < kDeviceSlots) attr_done[dev] = true;
    }
    int64_t g = ((n + F - 1) / F + kRmsdWarps - 1) / kRmsdWarps;
    const int64_t cap = (int64_t)num_sms() * 3;
    if (g > cap) g = cap;
    rmsd_assign_kernel<F><<<(unsigned)g, kRmsdWarps * 32, smem, s>>>(Xc, G, n, d, rc.Ct, rc.H, k, labels, rmsd);
    KM_CUDA(cudaGetLastError());
    return KM_OK;
}

// Every pair in double by a warp per frame: for one or two atoms (see the
// kernel), and for so few frames that each SM has no more than eight of these
// warps, where the four frames of a bracket warp would wait for each other: with
// one group of centers, with 6 to 24 atoms, whose many near-ties fill the lists,
// or with rows that are staged again for every group; up to sixteen warps per SM
// with long rows.  us, here and bracketed: k = 10, 1,000 frames of 58 atoms 67,
// 72, 2,000 95, 83; k = 100, 1,216 of 6 atoms 133, 168, of 8 134, 238; k = 500, 957
// of 20 391, 1013, 1,216 of 4 388, 185; k = 100, 1,000 frames of 97 atoms 175, 158,
// of 200 214, 232, 2,000 of 200 300, 247, of 400 400, 421, 4,000 of 400 694, 475.
bool rmsd_full_route(int64_t n, int d, int k) {
    const int64_t sms = num_sms();
    return d < 9 || (n <= 8 * sms && (k <= 32 || (d >= 18 && d <= 72) || d >= 3 * 192)) ||
           (n <= 16 * sms && d >= 3 * 384);
}

int launch_rmsd_assign(const float *Xc, const double *G, int64_t n, int d, const RmsdCenters &rc, int k,
                       int32_t *labels, float *rmsd, cudaStream_t s) {
    if (n == 0) return KM_OK;
    if (rmsd_full_route(n, d, k)) {
        rmsd_assign_full_kernel<<<rmsd_grid(n), kRmsdWarps * 32, 0, s>>>(Xc, G, n, d, rc.Ct, rc.H, k, labels,
                                                                        rmsd);
        KM_CUDA(cudaGetLastError());
        return KM_OK;
    }
    return launch_rmsd_assign_f<kRmsdFrames>(Xc, G, n, d, rc, k, labels, rmsd, s);
}

}  // namespace

}  // namespace km

using namespace km;

extern "C" {

size_t km_assign_minrmsd_workspace_size(int64_t n, int32_t d, int32_t k) {
    if (check_rmsd_shape(n, d, k) != KM_OK) return 0;
    Carver c(nullptr);
    c.take<float>((size_t)(n > 0 ? n : 1) * d);
    c.take<double>((size_t)(n > 0 ? n : 1));
    carve_centers(c, d, k);
    return c.bytes();
}

int km_assign_minrmsd(const float *X, int64_t n, int32_t d, const float *C, int32_t k, int32_t *labels, float *rmsd,
                      void *workspace, size_t workspace_bytes, void *stream) {
    KM_TRY(check_rmsd_shape(n, d, k));
    if ((n > 0 && (!X || !labels)) || !C) {
        set_error("km_assign_minrmsd needs non-NULL X, C and labels");
        return KM_ERR_BAD_SHAPE;
    }
    KM_TRY(check_ws(workspace, workspace_bytes, km_assign_minrmsd_workspace_size(n, d, k)));
    if (n == 0) return KM_OK;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    Carver c(workspace);
    float *Xc = c.take<float>((size_t)n * d);
    double *G = c.take<double>((size_t)n);
    RmsdCenters rc = carve_centers(c, d, k);
    KM_TRY(center_rows(X, n, d, Xc, G, s));
    KM_TRY(prepare_centers(C, d, k, rc, s));
    return launch_rmsd_assign(Xc, G, n, d, rc, k, labels, rmsd, s);
}

size_t km_minrmsd_rows_workspace_size(int64_t n, int32_t d) {
    if (check_rmsd_shape(n, d, 1) != KM_OK) return 0;
    Carver c(nullptr);
    for (int t = 0; t < 2; ++t) {
        c.take<float>((size_t)(n > 0 ? n : 1) * d);
        c.take<double>((size_t)(n > 0 ? n : 1));
    }
    return c.bytes();
}

int km_minrmsd_rows(const float *X, const float *Y, int64_t n, int32_t d, float *rmsd, void *workspace,
                    size_t workspace_bytes, void *stream) {
    KM_TRY(check_rmsd_shape(n, d, 1));
    if (n > 0 && (!X || !Y || !rmsd)) {
        set_error("km_minrmsd_rows needs non-NULL X, Y and rmsd");
        return KM_ERR_BAD_SHAPE;
    }
    KM_TRY(check_ws(workspace, workspace_bytes, km_minrmsd_rows_workspace_size(n, d)));
    if (n == 0) return KM_OK;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    Carver c(workspace);
    float *A = c.take<float>((size_t)n * d);
    double *GA = c.take<double>((size_t)n);
    float *B = c.take<float>((size_t)n * d);
    double *GB = c.take<double>((size_t)n);
    KM_TRY(center_rows(X, n, d, A, GA, s));
    KM_TRY(center_rows(Y, n, d, B, GB, s));
    int64_t g = (n + 255) / 256;
    const int64_t cap = (int64_t)num_sms() * 8;
    if (g > cap) g = cap;
    rmsd_rows_kernel<<<(unsigned)g, 256, 0, s>>>(A, GA, B, GB, n, d, rmsd);
    KM_CUDA(cudaGetLastError());
    return KM_OK;
}

size_t km_kmpp_minrmsd_workspace_size(int64_t n, int32_t d, int32_t k) {
    if (check_rmsd_shape(n, d, k) != KM_OK) return 0;
    Carver c(nullptr);
    c.take<float>((size_t)(n > 0 ? n : 1) * d);
    c.take<double>((size_t)(n > 0 ? n : 1));
    c.take<int64_t>((size_t)k);
    c.take<char>(kmpp_ws_size(n, d, k));
    return c.bytes();
}

int km_kmpp_minrmsd(const float *X, int64_t n, int32_t d, int32_t k, uint32_t seed, float *C0, int64_t *idx,
                    km_callback cb, void *cb_user, void *workspace, size_t workspace_bytes, void *stream) {
    KM_TRY(check_rmsd_shape(n, d, k));
    if (n < 1 || !X || !C0) {
        set_error("kmeans++ needs n >= 1 and non-NULL X, C0");
        return KM_ERR_BAD_SHAPE;
    }
    KM_TRY(check_ws(workspace, workspace_bytes, km_kmpp_minrmsd_workspace_size(n, d, k)));
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    Carver c(workspace);
    float *Xc = c.take<float>((size_t)n * d);
    double *G = c.take<double>((size_t)n);
    int64_t *idx_dev = c.take<int64_t>((size_t)k);
    void *ws_kmpp = c.take<char>(kmpp_ws_size(n, d, k));
    KM_TRY(center_rows(X, n, d, Xc, G, s));
    KmppMetric m{Xc, G, idx_dev};
    KM_TRY(run_kmpp(X, n, d, k, seed, C0, idx_dev, cb, cb_user, ws_kmpp, s, &m));
    if (idx) KM_CUDA(cudaMemcpyAsync(idx, idx_dev, sizeof(int64_t) * (size_t)k, cudaMemcpyDeviceToDevice, s));
    return KM_OK;
}

size_t km_lloyd_minrmsd_workspace_size(int64_t n, int32_t d, int32_t k) {
    if (check_rmsd_shape(n, d, k) != KM_OK) return 0;
    Carver c(nullptr);
    c.take<float>((size_t)(n > 0 ? n : 1) * d);
    c.take<double>((size_t)(n > 0 ? n : 1));
    carve_centers(c, d, k);
    c.take<float>((size_t)k * d);  // C_new
    c.take<double>(2);             // cost, the update's own cost
    c.take<uint32_t>(1);
    c.take<char>(update_ws_size(n, d, k));
    return c.bytes();
}

int km_lloyd_minrmsd(const float *X, int64_t n, int32_t d, int32_t k, float *C, int32_t max_iter, double tolerance,
                     int32_t *labels, double *inertias, int32_t *n_iter, int32_t *converged, km_callback cb,
                     void *cb_user, void *workspace, size_t workspace_bytes, void *stream) {
    KM_TRY(check_rmsd_shape(n, d, k));
    if (n < 1 || !X || !C || !labels || !n_iter || !converged || max_iter < 0) {
        set_error("km_lloyd_minrmsd needs n >= 1, max_iter >= 0 and non-NULL X, C, labels, n_iter, converged");
        return KM_ERR_BAD_SHAPE;
    }
    *n_iter = 0;
    *converged = 0;
    KM_TRY(check_ws(workspace, workspace_bytes, km_lloyd_minrmsd_workspace_size(n, d, k)));
    if (max_iter == 0) return KM_OK;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    Carver c(workspace);
    float *Xc = c.take<float>((size_t)n * d);
    double *G = c.take<double>((size_t)n);
    RmsdCenters rc = carve_centers(c, d, k);
    float *C_new = c.take<float>((size_t)k * d);
    double *cost = c.take<double>(2);
    uint32_t *err = c.take<uint32_t>(1);
    void *ws_update = c.take<char>(update_ws_size(n, d, k));
    KM_TRY(center_rows(X, n, d, Xc, G, s));
    KM_CUDA(cudaMemsetAsync(err, 0, sizeof(uint32_t), s));
    double prev = 0.0;
    for (int32_t it = 0; it < max_iter; ++it) {
        KM_TRY(prepare_centers(C, d, k, rc, s));
        KM_TRY(launch_rmsd_assign(Xc, G, n, d, rc, k, labels, nullptr, s));
        KM_TRY(launch_update(X, n, d, labels, k, C, C_new, nullptr, cost + 1, err, ws_update, s));
        // inertia under the metric, for the new centers
        KM_TRY(center_rows(C_new, k, d, rc.Cc, rc.H, s));
        KM_CUDA(cudaMemsetAsync(cost, 0, sizeof(double), s));
        int64_t g = (n + 255) / 256;
        const int64_t cap = (int64_t)num_sms() * 8;
        if (g > cap) g = cap;
        rmsd_cost_kernel<<<(unsigned)g, 256, 0, s>>>(Xc, G, n, d, labels, rc.Cc, rc.H, cost);
        KM_CUDA(cudaGetLastError());
        KM_CUDA(cudaMemcpyAsync(C, C_new, sizeof(float) * (size_t)k * d, cudaMemcpyDeviceToDevice, s));
        double h_cost = 0.0;
        uint32_t h_err = 0;
        KM_CUDA(cudaMemcpyAsync(&h_cost, cost, sizeof(double), cudaMemcpyDeviceToHost, s));
        KM_CUDA(cudaMemcpyAsync(&h_err, err, sizeof(uint32_t), cudaMemcpyDeviceToHost, s));
        KM_CUDA(cudaStreamSynchronize(s));
        KM_TRY(device_error_status(h_err));
        if (inertias) inertias[it] = h_cost;
        *n_iter = it + 1;
        const double rel = h_cost != 0.0 ? fabs(h_cost - prev) / h_cost : 0.0;
        prev = h_cost;
        if (cb) cb(cb_user);
        if (rel <= tolerance) {
            *converged = 1;
            break;
        }
    }
    return KM_OK;
}

}  // extern "C"
