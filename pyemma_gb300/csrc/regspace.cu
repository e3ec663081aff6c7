// regspace.cu -- regular space clustering, first pass (km_regspace).
//
// Reference: RegularSpaceClustering._estimate, pyemma/coordinates/clustering/
// regspace.py:140-152 (deeptime RegularSpace.partial_fit over the chunks in
// iteration order).  The first frame becomes a center; every later frame
// becomes one when its distance to every center found so far is at least
// dmin.  The distance is the square root (float32, correctly rounded) of the
// exact float32 squared distance in feature order, compared in double with
// dmin.
//
// The walk is sequential by definition; the GPU splits it by chunks of
// frames (1024, 2048, ... up to kRsChunk).  For a chunk, every SM tests the
// frames against the centers known before the chunk and leaves one bit per
// frame.  One CTA then lists the frames that passed, in order, and resolves
// them in windows of one frame per thread (or per warp): the window is tested
// against the centers added within the chunk, and then the first frame still
// standing becomes a center and every thread tests its own frame against it,
// until none stands.  So the serial steps number one per center, not one per
// frame that passed.  The center count stays on the device: the chunks are
// enqueued without waiting for each other's result.
//
// Bound by the latency of those steps (one CTA barrier and one distance
// each) and by the launches.  1,000,000 x 3 frames, dmin = 1: 0.68 ms on the
// device in 22 launches (filter 0.20, walk 0.48); the clustering with its final
// assignment takes 1.55 ms, 57 with one serial step per frame that passed.
#include <algorithm>
#include <cmath>
#include <cstring>

#include "km_common.cuh"
#include "km_internal.h"

namespace km {

namespace {

constexpr int64_t kRsFirst = 1024;     // frames of the first chunk; each chunk doubles it
constexpr int64_t kRsChunk = 262144;   // frames of a chunk at most
constexpr int64_t kRsChunkWide = 65536;  // the same for d > 32
constexpr int kRsCheck = 16;           // chunks between two looks at the stop flag
constexpr int kRsFilterThreads = 256;

// State words: centers so far, stopped (max_centers reached).
enum RsState { kRsCount = 0, kRsStop = 1 };

// The smallest float32 squared distance t with (double)sqrtf(t) >= dmin:
// sqrt is monotone, so dist >= dmin exactly when dist^2 >= t (and a NaN
// fails both).
float rs_threshold(double dmin) {
    uint32_t lo = 0u, hi = 0x7f800000u;  // hi: +inf, whose root is >= any dmin
    while (lo < hi) {
        const uint32_t mid = lo + (hi - lo) / 2;
        float t;
        std::memcpy(&t, &mid, sizeof(t));
        if ((double)std::sqrt(t) >= dmin)
            hi = mid;
        else
            lo = mid + 1;
    }
    float t;
    std::memcpy(&t, &lo, sizeof(t));
    return t;
}

// Frame row i into DP registers (zero beyond d).
template <int DP>
__device__ __forceinline__ void rs_load_row(const float *__restrict__ X, int64_t i, int d, float (&x)[DP]) {
#pragma unroll
    for (int f = 0; f < DP; ++f) x[f] = f < d ? __ldg(X + i * d + f) : 0.0f;
}

// sqdist_exact's arithmetic and order on a register row; the features beyond
// d add a zero square, which leaves the sum as it is.
template <int DP>
__device__ __forceinline__ float rs_sqdist(const float (&x)[DP], const float *c) {
    float acc = 0.0f;
#pragma unroll
    for (int f = 0; f < DP; ++f) acc = __fadd_rn(acc, sq_term(x[f], c[f]));
    return acc;
}

// d <= 32: one frame per thread (its row in registers) against all centers so
// far, staged through shared memory 256 at a time; a CTA leaves as soon as
// none of its frames stands.  bits: one bit per frame of the chunk [a, b).
template <int DP>
__global__ void __launch_bounds__(kRsFilterThreads) regspace_filter_kernel(
    const float *__restrict__ X, int64_t a, int64_t b, int d, const float *__restrict__ centers, float t2,
    const int32_t *__restrict__ state, uint32_t *__restrict__ bits) {
    constexpr int kTileC = 256;
    __shared__ __align__(16) float cs[kTileC * DP];
    if (state[kRsStop]) return;
    const int nc = state[kRsCount];
    for (int64_t base = a + (int64_t)blockIdx.x * kRsFilterThreads; base < b;
         base += (int64_t)gridDim.x * kRsFilterThreads) {
        const int64_t i = base + threadIdx.x;
        bool alive = i < b;
        float x[DP];
        rs_load_row<DP>(X, alive ? i : a, d, x);
        for (int c0 = 0; c0 < nc; c0 += kTileC) {
            if (!__syncthreads_or(alive)) break;  // also: the tile before has been read
            const int m = min(kTileC, nc - c0);
            for (int e = threadIdx.x; e < m * DP; e += kRsFilterThreads) {
                const int j = e / DP, f = e - j * DP;
                cs[e] = f < d ? __ldg(centers + (int64_t)(c0 + j) * d + f) : 0.0f;
            }
            __syncthreads();
            for (int j0 = 0; j0 < m; j0 += 16) {
                if (!__any_sync(0xffffffffu, alive)) break;
                const int j1 = min(j0 + 16, m);
#pragma unroll 4
                for (int j = j0; j < j1; ++j)
                    if (!(rs_sqdist<DP>(x, cs + j * DP) >= t2)) alive = false;
            }
        }
        const unsigned word = __ballot_sync(0xffffffffu, alive);
        if ((threadIdx.x & 31) == 0 && base + threadIdx.x < b) bits[(i - a) >> 5] = word;
        __syncthreads();  // the last tile has been read by every warp
    }
}

// d > 32: the bits from the smallest squared distances (launch_assign_fp32)
// to the nc centers so far.  A minimum passes over distances that are NaN,
// which stop a frame (not at least dmin).  Such a frame has no finite distance:
// it is not finite itself, or center 0 has a NaN and is the only one.  So the
// frames whose smallest distance is infinite meet every center again, a warp
// for each; finite data has none.
__global__ void __launch_bounds__(256) regspace_bits_kernel(const float *__restrict__ X, int64_t m, int d,
                                                            const float *__restrict__ centers, int nc,
                                                            const float *__restrict__ dist2, float t2,
                                                            uint32_t *__restrict__ bits) {
    const int lane = threadIdx.x & 31;
    const DenseRows rows{X, d};
    for (int64_t base = (int64_t)blockIdx.x * 256; base < m; base += (int64_t)gridDim.x * 256) {
        const int64_t i = base + threadIdx.x;
        const float v = i < m && nc > 0 ? dist2[i] : 0.0f;
        unsigned word = __ballot_sync(0xffffffffu, i < m && (nc == 0 || v >= t2));
        for (unsigned look = word & __ballot_sync(0xffffffffu, v == __int_as_float(0x7f800000)); look;
             look &= look - 1u) {
            const int q = __ffs(look) - 1;
            for (int j = 0; j < nc; ++j) {
                if (!(warp_sqdist_exact(rows, i - lane + q, centers + (int64_t)j * d, d, lane) >= t2)) {
                    word &= ~(1u << q);
                    break;
                }
            }
        }
        if (lane == 0 && i < m) bits[i >> 5] = word;
    }
}

// The set bits of the chunk's words in order: list[0..m) (frame offsets in
// the chunk); returns m in every thread.  One CTA of THREADS threads.
template <int THREADS>
__device__ __forceinline__ int rs_list(const uint32_t *__restrict__ bits, int64_t nbits, int32_t *__restrict__ list) {
    __shared__ int warp_tot[THREADS / 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int nw = (int)((nbits + 31) / 32);
    int run = 0;
    for (int w0 = 0; w0 < nw; w0 += THREADS) {
        const int w = w0 + threadIdx.x;
        uint32_t v = w < nw ? __ldcg(bits + w) : 0u;
        const int c = __popc(v);
        int x = c;
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, x, off);
            if (lane >= off) x += y;
        }
        if (lane == 31) warp_tot[warp] = x;
        __syncthreads();
        int before = 0, total = 0;
#pragma unroll
        for (int q = 0; q < THREADS / 32; ++q) {
            if (q < warp) before += warp_tot[q];
            total += warp_tot[q];
        }
        int at = run + before + x - c;
        while (v) {
            list[at++] = w * 32 + __ffs(v) - 1;
            v &= v - 1u;
        }
        run += total;
        __syncthreads();  // warp_tot is rewritten by the next round
    }
    return run;
}

// The lowest thread of the CTA with its flag set, or -1; the same in every
// thread.  slot alternates between 0 and 1 from call to call, so one barrier
// per call is enough (WARPS <= 32).
template <int WARPS>
__device__ __forceinline__ int rs_first(bool flag, uint32_t (*masks)[32], int slot) {
    const int lane = threadIdx.x & 31;
    const unsigned b = __ballot_sync(0xffffffffu, flag);
    if (lane == 0) masks[slot][threadIdx.x >> 5] = b;
    __syncthreads();
    const unsigned m = lane < WARPS ? masks[slot][lane] : 0u;
    const unsigned any = __ballot_sync(0xffffffffu, m != 0u);
    if (!any) return -1;
    const int w = __ffs(any) - 1;
    return w * 32 + __ffs(__shfl_sync(0xffffffffu, m, w)) - 1;
}

// d <= 32: windows of THREADS listed frames, one per thread, rows in
// registers and in shared memory (the next center's row is read from there);
// the first kNew centers added within the chunk are kept in shared memory,
// later ones are read back from the center array past L1.
constexpr int rs_threads(int dp) { return dp <= 16 ? 1024 : 512; }
constexpr int rs_kept(int dp) { return 16384 / dp; }
constexpr size_t rs_walk_smem(int dp) { return ((size_t)rs_threads(dp) + rs_kept(dp)) * dp * sizeof(float); }

template <int DP>
__global__ void __launch_bounds__(rs_threads(DP)) regspace_walk_kernel(
    const float *__restrict__ X, int64_t a, int64_t b, int d, const uint32_t *__restrict__ bits, float t2,
    int max_centers, float *__restrict__ centers, int32_t *__restrict__ list, int32_t *__restrict__ state) {
    constexpr int THREADS = rs_threads(DP);
    constexpr int kNew = rs_kept(DP);
    extern __shared__ __align__(16) float rs_smem[];
    float *rows = rs_smem;                 // [thread][DP]
    float *kept = rs_smem + THREADS * DP;  // [center - nc0][DP]
    __shared__ uint32_t masks[2][32];
    if (state[kRsStop]) return;
    const int tid = threadIdx.x;
    const int nc0 = state[kRsCount];
    int nc = nc0, stop = 0, slot = 0;
    const int m = rs_list<THREADS>(bits, b - a, list);
    __syncthreads();  // the list is complete
    for (int w0 = 0; w0 < m && !stop; w0 += THREADS) {
        bool alive = w0 + tid < m;
        float x[DP];
        rs_load_row<DP>(X, a + (alive ? list[w0 + tid] : 0), d, x);
#pragma unroll
        for (int f = 0; f < DP; ++f) rows[tid * DP + f] = x[f];
        // Against the centers added by earlier windows of this chunk.
        for (int j0 = nc0; j0 < nc; j0 += 16) {
            if (!__any_sync(0xffffffffu, alive)) break;
            const int j1 = min(j0 + 16, nc);
            if (j1 - nc0 <= kNew) {
#pragma unroll 4
                for (int j = j0; j < j1; ++j)
                    if (!(rs_sqdist<DP>(x, kept + (j - nc0) * DP) >= t2)) alive = false;
            } else {
                for (int j = j0; j < j1; ++j) {
                    float c[DP];
#pragma unroll
                    for (int f = 0; f < DP; ++f) c[f] = f < d ? __ldcg(centers + (int64_t)j * d + f) : 0.0f;
                    if (!(rs_sqdist<DP>(x, c) >= t2)) alive = false;
                }
            }
        }
        for (;;) {
            const int p = rs_first<THREADS / 32>(alive, masks, slot);
            slot ^= 1;
            if (p < 0) break;
            if (nc == max_centers) {
                stop = 1;
                break;
            }
            // Frame p of the window is a center: every later frame meets it.
            const float *c = rows + p * DP;
            if (tid < d) centers[(int64_t)nc * d + tid] = c[tid];
            if (tid < DP && nc - nc0 < kNew) kept[(nc - nc0) * DP + tid] = c[tid];
            if (tid <= p)
                alive = false;
            else if (!(rs_sqdist<DP>(x, c) >= t2))
                alive = false;
            ++nc;
        }
        __syncthreads();  // rows are rewritten, kept rows and centers are read by the next window
    }
    if (tid == 0) {
        state[kRsCount] = nc;
        state[kRsStop] = stop;
    }
}

// d > 32: windows of 256 listed frames, eight per warp, distances by
// warp_sqdist_exact; the centers added within the chunk are named by their
// frames (added[], read past L1) and read from X.
constexpr int kRsWideThreads = 1024;
constexpr int kRsWidePer = 8;

__global__ void __launch_bounds__(kRsWideThreads) regspace_walk_wide_kernel(
    const float *__restrict__ X, int64_t a, int64_t b, int d, const uint32_t *__restrict__ bits, float t2,
    int max_centers, float *__restrict__ centers, int32_t *__restrict__ list, int32_t *__restrict__ added,
    int32_t *__restrict__ state) {
    constexpr int kWarps = kRsWideThreads / 32;
    constexpr int kWindow = kWarps * kRsWidePer;
    __shared__ uint32_t masks[2][32];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int nc0 = state[kRsCount];
    int nc = nc0, stop = 0, slot = 0;
    const int m = rs_list<kRsWideThreads>(bits, b - a, list);
    __syncthreads();
    const DenseRows rows{X, d};
    for (int w0 = 0; w0 < m && !stop; w0 += kWindow) {
        // Frames w0 + 8 warp + q of the list; bit q of alive: q still stands.
        const int q0 = w0 + warp * kRsWidePer;
        const int cnt = max(0, min(kRsWidePer, m - q0));
        unsigned alive = (1u << cnt) - 1u;
        const int32_t mine = lane < cnt ? list[q0 + lane] : 0;
        for (int j = 0; j < nc - nc0 && alive; ++j) {
            const float *c = X + (a + __ldcg(added + j)) * d;
            for (unsigned v = alive; v; v &= v - 1u) {
                const int q = __ffs(v) - 1;
                const int64_t i = a + __shfl_sync(0xffffffffu, mine, q);
                if (!(warp_sqdist_exact(rows, i, c, d, lane) >= t2)) alive &= ~(1u << q);
            }
        }
        for (;;) {
            if (lane == 0) masks[slot][warp] = alive;
            __syncthreads();
            const unsigned mk = masks[slot][lane];
            const unsigned any = __ballot_sync(0xffffffffu, mk != 0u);
            slot ^= 1;
            if (!any) break;
            if (nc == max_centers) {
                stop = 1;
                break;
            }
            const int w = __ffs(any) - 1;
            const int q = __ffs(__shfl_sync(0xffffffffu, mk, w)) - 1;
            const int32_t pf = list[w0 + w * kRsWidePer + q];
            const float *c = X + (a + pf) * d;
            for (int f = tid; f < d; f += kRsWideThreads) centers[(int64_t)nc * d + f] = __ldg(c + f);
            if (tid == 0) added[nc - nc0] = pf;
            if (warp < w)
                alive = 0u;
            else if (warp == w)
                alive &= ~((2u << q) - 1u);
            for (unsigned v = alive; v; v &= v - 1u) {
                const int t = __ffs(v) - 1;
                const int64_t i = a + __shfl_sync(0xffffffffu, mine, t);
                if (!(warp_sqdist_exact(rows, i, c, d, lane) >= t2)) alive &= ~(1u << t);
            }
            ++nc;
        }
        __syncthreads();
    }
    if (tid == 0) {
        state[kRsCount] = nc;
        state[kRsStop] = stop;
    }
}

template <int DP>
int rs_chunk(const float *X, int64_t a, int64_t b, int d, float t2, int max_centers, float *centers, uint32_t *bits,
             int32_t *list, int32_t *state, cudaStream_t s) {
    static bool attr_done[kDeviceSlots] = {};
    const int dev = current_device();
    if (dev < 0 || dev >= kDeviceSlots || !attr_done[dev]) {
        KM_CUDA(cudaFuncSetAttribute(regspace_walk_kernel<DP>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)rs_walk_smem(DP)));
        if (dev >= 0 && dev < kDeviceSlots) attr_done[dev] = true;
    }
    int64_t g = (b - a + kRsFilterThreads - 1) / kRsFilterThreads;
    const int64_t cap = (int64_t)num_sms() * 8;
    if (g > cap) g = cap;
    regspace_filter_kernel<DP><<<(unsigned)g, kRsFilterThreads, 0, s>>>(X, a, b, d, centers, t2, state, bits);
    KM_CUDA(cudaGetLastError());
    regspace_walk_kernel<DP><<<1, rs_threads(DP), rs_walk_smem(DP), s>>>(X, a, b, d, bits, t2, max_centers, centers,
                                                                        list, state);
    KM_CUDA(cudaGetLastError());
    return KM_OK;
}

int rs_chunk_narrow(const float *X, int64_t a, int64_t b, int d, float t2, int max_centers, float *centers,
                    uint32_t *bits, int32_t *list, int32_t *state, cudaStream_t s) {
    if (d <= 4) return rs_chunk<4>(X, a, b, d, t2, max_centers, centers, bits, list, state, s);
    if (d <= 8) return rs_chunk<8>(X, a, b, d, t2, max_centers, centers, bits, list, state, s);
    if (d <= 16) return rs_chunk<16>(X, a, b, d, t2, max_centers, centers, bits, list, state, s);
    return rs_chunk<32>(X, a, b, d, t2, max_centers, centers, bits, list, state, s);
}

struct RsWs {
    uint32_t *bits;
    int32_t *list;    // frames of the chunk that passed the filter
    int32_t *added;   // d > 32: frames of the chunk that became centers; also the filter's labels
    float *dist;      // d > 32: smallest squared distances of the chunk
    int32_t *state;
};

RsWs rs_carve(void *ws, int d, size_t *bytes) {
    Carver c(ws);
    RsWs w;
    const int64_t chunk = d <= 32 ? kRsChunk : kRsChunkWide;
    w.bits = c.take<uint32_t>((size_t)chunk / 32);
    w.list = c.take<int32_t>((size_t)chunk);
    w.added = c.take<int32_t>(d <= 32 ? 1 : (size_t)chunk);
    w.dist = c.take<float>(d <= 32 ? 1 : (size_t)chunk);
    w.state = c.take<int32_t>(2);
    if (bytes) *bytes = c.bytes();
    return w;
}

}  // namespace

}  // namespace km

using namespace km;

extern "C" {

size_t km_regspace_workspace_size(int32_t d) {
    if (d < 1 || d > kMaxD) return 0;
    size_t bytes = 0;
    rs_carve(nullptr, d, &bytes);
    return bytes;
}

int km_regspace(const float *X, int64_t n, int32_t d, double dmin, int32_t max_centers, float *centers,
                int32_t *n_centers, int32_t *converged, void *workspace, size_t workspace_bytes, void *stream) {
    if (!n_centers || !converged) {
        set_error("n_centers and converged must be non-NULL");
        return KM_ERR_BAD_SHAPE;
    }
    *n_centers = 0;
    *converged = 1;
    KM_TRY(check_shape(n, d, max_centers > 0 ? max_centers : 1));
    if (max_centers < 1 || !(dmin >= 0.0) || (n > 0 && (!X || !centers))) {
        set_error("km_regspace needs max_centers >= 1, dmin >= 0 and non-NULL X, centers");
        return KM_ERR_BAD_SHAPE;
    }
    KM_TRY(check_ws(workspace, workspace_bytes, km_regspace_workspace_size(d)));
    if (n == 0) return KM_OK;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    const RsWs w = rs_carve(workspace, d, nullptr);
    const float t2 = rs_threshold(dmin);
    KM_CUDA(cudaMemsetAsync(w.state, 0, 2 * sizeof(int32_t), s));
    int32_t h_state[2] = {0, 0};
    auto read_state = [&]() -> int {
        KM_CUDA(cudaMemcpyAsync(h_state, w.state, sizeof(h_state), cudaMemcpyDeviceToHost, s));
        KM_CUDA(cudaStreamSynchronize(s));
        return KM_OK;
    };
    int64_t chunk = kRsFirst;
    int since = 0;
    for (int64_t a = 0; a < n && !h_state[kRsStop];) {
        const int64_t b = a + chunk < n ? a + chunk : n;
        if (d <= 32) {
            KM_TRY(rs_chunk_narrow(X, a, b, d, t2, max_centers, centers, w.bits, w.list, w.state, s));
            if (b < n && ++since == kRsCheck) {  // a stopped walk leaves soon after
                KM_TRY(read_state());
                since = 0;
            }
        } else {
            // The exact assignment kernel needs the center count on the host.
            const bool any = h_state[kRsCount] > 0;
            if (any)
                KM_TRY(launch_assign_fp32(X + a * d, nullptr, nullptr, b - a, d, centers, h_state[kRsCount], w.added,
                                          w.dist, nullptr, s));
            int64_t g = (b - a + 255) / 256;
            const int64_t cap = (int64_t)num_sms() * 8;
            if (g > cap) g = cap;
            regspace_bits_kernel<<<(unsigned)g, 256, 0, s>>>(X + a * d, b - a, d, centers, h_state[kRsCount],
                                                             w.dist, t2, w.bits);
            KM_CUDA(cudaGetLastError());
            regspace_walk_wide_kernel<<<1, kRsWideThreads, 0, s>>>(X, a, b, d, w.bits, t2, max_centers, centers,
                                                                   w.list, w.added, w.state);
            KM_CUDA(cudaGetLastError());
            KM_TRY(read_state());
        }
        a = b;
        chunk = std::min<int64_t>(2 * chunk, d <= 32 ? kRsChunk : kRsChunkWide);
    }
    KM_TRY(read_state());
    *n_centers = h_state[0];
    *converged = h_state[1] ? 0 : 1;
    return KM_OK;
}

}  // extern "C"
