// The prediction sweep of the reference's study tool (c_codes/s2_many_prediction.cpp:164-464):
// every target of one predictor's loop nest is predicted from the original data with each of a
// set of coefficients, quantised, and summed into the tool's error figures. The QB streams then
// go through the library's histogram and tiled Huffman kernels.
//
// Floating point follows what GCC 13.3 makes of the reference under -Ofast -mfma (pinned against
// the reference's own dot functions and binary outputs): neighbour pairs summed in float; the
// 1D4R and 2D4R products of those sums with 0.25 -+ t are exact in double; 1D6R is
// fma(w, s1, fma(a, s5, b * s3)) with w = 0.5 - (a + b); e = pred - x; qb = llround(e * neg_2_eb);
// e2 = fma(-2 qb, abs_eb, e); the sums of e^2 and e2^2 are fused steps. The sums run per thread,
// per block and over blocks in a fixed order, so a launch is deterministic; the reference sums one
// target after the other, so the sums agree to rounding, while every QB is identical.
#include <algorithm>
#include <climits>
#include <type_traits>

#include "launch.h"

namespace asz {

namespace {

constexpr unsigned kSweepThreads = 256;
constexpr uint32_t kSeg = 16;  // positions of a line per work item when a thread walks lines

__device__ __forceinline__ double warp_sum(double v) {
    for (int o = 16; o; o >>= 1) v = __dadd_rn(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}

}  // namespace

// A thread takes kSweepCoefs coefficients at once: a target's index (two 64-bit divisions), its loads
// and its conversions are the same for all of them. With a coefficient a thread those cost more than
// the prediction itself (100x500x500, 13 coefficients: 1.30 -> 0.77 ms). Then a warp waits for its loads and
// conversions, at 16 warps an SM: three CTAs an SM, with a few spilled registers, take 0.61 ms.
constexpr uint32_t kSweepCoefs = 4;

// Running figures of one thread and one coefficient: the three sums and the QB extremes.
template <class Q>
struct SweepAcc {
    double se = 0.0, sr = 0.0, sa = 0.0;
    Q lo = std::is_same_v<Q, int32_t> ? (Q)INT_MAX : (Q)LLONG_MAX, hi = std::is_same_v<Q, int32_t> ? (Q)INT_MIN : (Q)LLONG_MIN;
};

// One target (index `it` of the (line, position) space) with kSweepCoefs coefficient sets, nc of
// them real. wide: a QB that Q does not hold.
template <class Q, bool SIX>
__device__ __forceinline__ void sweep_one(const float *__restrict__ d, const SweepGeom &g,
                                          const double (&w)[kSweepCoefs][SIX ? 3 : 2], uint32_t nc, double abs_eb,
                                          double neg_2_eb, Q *__restrict__ out, uint64_t qb_stride, uint64_t it,
                                          SweepAcc<Q> (&acc)[kSweepCoefs], bool &wide) {
    uint64_t i[3], j;
    if (!sweep_target(g, it, i, j)) return;
    const uint64_t pos = i[0] * (g.n[1] * g.n[2]) + i[1] * g.n[2] + i[2];
    const uint64_t d0 = g.dist[0];
    const double x = d[pos];
    double v[3];
    if constexpr (SIX) {  // compress_1d6r_dot (s2_many_prediction.cpp:67-87)
        v[0] = __fadd_rn(d[pos - d0], d[pos + d0]);
        v[1] = __fadd_rn(d[pos - 5 * d0], d[pos + 5 * d0]);
        v[2] = __fadd_rn(d[pos - 3 * d0], d[pos + 3 * d0]);
    } else {  // compress_1d4r_dot (:28-45): lo and the far pair; compress_2d4r_dot (:47-65): lo and the second axis
        const uint64_t d1 = g.kind == 0 ? 3 * d0 : g.dist[1];
        v[0] = __fadd_rn(d[pos - d1], d[pos + d1]);
        v[1] = __fadd_rn(d[pos - d0], d[pos + d0]);
    }
#pragma unroll
    for (uint32_t c = 0; c < kSweepCoefs; c++) {
        SweepAcc<Q> &a = acc[c];
        double pred;
        if constexpr (SIX) pred = __fma_rn(w[c][0], v[0], __fma_rn(w[c][1], v[1], __dmul_rn(w[c][2], v[2])));
        else pred = __dadd_rn(__dmul_rn(w[c][0], v[0]), __dmul_rn(w[c][1], v[1]));
        const double e = __dsub_rn(pred, x);
        a.sr = __fma_rn(e, e, a.sr);
        a.sa = __dadd_rn(a.sa, fabs(e));
        const int64_t q = lround_d(__dmul_rn(e, neg_2_eb));
        const Q qs = (Q)q;
        wide |= qs != q;
        if (c < nc) out[c * qb_stride + j] = qs;
        const double e2 = __fma_rn(-(double)(q * 2), abs_eb, e);
        a.se = __fma_rn(e2, e2, a.se);
        a.lo = min(a.lo, qs);
        a.hi = max(a.hi, qs);
    }
}

// grid (x: CTAs over the work items, y: groups of kSweepCoefs coefficients). Writes the QB stream of
// coefficient k at qb + k * qb_stride, the CTA's three partial sums at part[(k * gridDim.x + blockIdx.x) * 3],
// and folds the stream's extremes into mm[2k], mm[2k + 1]; a QB that Q does not hold makes them the
// extremes of int64, and the caller repeats the launch with 64-bit QBs. They are nearly always held by
// 32 bits, which halves what this kernel writes and the two after it read.
//
// When the QB order runs along the contiguous axis, neighbouring threads take neighbouring
// positions of a line. When it runs along axis 0 or 1, a work item is a segment of kSeg positions
// of one line, with neighbouring items on neighbouring lines: a warp then reads neighbouring lines
// (adjacent along axis 2), and each thread writes its segment's QB run in order.
template <class Q, bool SIX>
__global__ void __launch_bounds__(kSweepThreads, 3)
    sweep_predict_kernel(const float *__restrict__ d, SweepGeom g, const SweepCoef *__restrict__ coef, uint32_t ncoef,
                         double abs_eb, double neg_2_eb, Q *__restrict__ qb, uint64_t qb_stride, double *__restrict__ part,
                         long long *__restrict__ mm) {
    const uint32_t k0 = blockIdx.y * kSweepCoefs, nc = min(kSweepCoefs, ncoef - k0);
    double cw[kSweepCoefs][SIX ? 3 : 2];
#pragma unroll
    for (uint32_t c = 0; c < kSweepCoefs; c++) {
        const SweepCoef &C = coef[k0 + min(c, nc - 1)];
        if constexpr (SIX) {
            cw[c][0] = C.w;
            cw[c][1] = C.c0;
            cw[c][2] = C.c1;
        } else {
            cw[c][0] = C.lo;
            cw[c][1] = C.hi;
        }
    }
    Q *out = qb + (uint64_t)k0 * qb_stride;
    const uint64_t gtid = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x, gstride = (uint64_t)gridDim.x * blockDim.x;
    SweepAcc<Q> acc[kSweepCoefs];
    bool wide = false;
    if (g.line_per_thread) {
        const uint64_t items = g.lines * ((g.per_line + kSeg - 1) / kSeg);
        for (uint64_t item = gtid; item < items; item += gstride) {
            const uint64_t line = item % g.lines, p0 = (item / g.lines) * kSeg;
            const uint64_t p1 = min(p0 + kSeg, g.per_line);
            for (uint64_t k = p0; k < p1; k++)
                sweep_one<Q, SIX>(d, g, cw, nc, abs_eb, neg_2_eb, out, qb_stride, line * g.per_line + k, acc, wide);
        }
    } else {
        const uint64_t total = g.lines * g.per_line;
        for (uint64_t it = gtid; it < total; it += gstride)
            sweep_one<Q, SIX>(d, g, cw, nc, abs_eb, neg_2_eb, out, qb_stride, it, acc, wide);
    }
    constexpr unsigned kWarps = kSweepThreads / 32;
    __shared__ double red[kSweepCoefs][3][kWarps];
    __shared__ Q rlo[kSweepCoefs][kWarps], rhi[kSweepCoefs][kWarps];
    const unsigned w = threadIdx.x >> 5;
#pragma unroll
    for (uint32_t c = 0; c < kSweepCoefs; c++) {
        const double se = warp_sum(acc[c].se), sr = warp_sum(acc[c].sr), sa = warp_sum(acc[c].sa);
        Q lo = acc[c].lo, hi = acc[c].hi;
        for (int o = 16; o; o >>= 1) {
            lo = min(lo, __shfl_xor_sync(0xffffffffu, lo, o));
            hi = max(hi, __shfl_xor_sync(0xffffffffu, hi, o));
        }
        if ((threadIdx.x & 31) == 0) {
            red[c][0][w] = se;
            red[c][1][w] = sr;
            red[c][2][w] = sa;
            rlo[c][w] = lo;
            rhi[c][w] = hi;
        }
    }
    wide = __syncthreads_or(wide);
    if (threadIdx.x < 32) {
        const uint32_t c = threadIdx.x / 3, f = threadIdx.x % 3;
        if (c < nc) {
            double s = 0.0;
            for (unsigned k = 0; k < kWarps; k++) s = __dadd_rn(s, red[c][f][k]);
            part[((uint64_t)(k0 + c) * gridDim.x + blockIdx.x) * 3 + f] = s;
        }
    } else if (threadIdx.x < 32 + nc) {
        const uint32_t c = threadIdx.x - 32;
        Q l = rlo[c][0], h = rhi[c][0];
        for (unsigned k = 1; k < kWarps; k++) {
            l = min(l, rlo[c][k]);
            h = max(h, rhi[c][k]);
        }
        if (wide || l <= h) {
            atomicMin(mm + 2 * (k0 + c), wide ? LLONG_MIN : (long long)l);
            atomicMax(mm + 2 * (k0 + c) + 1, wide ? LLONG_MAX : (long long)h);
        }
    }
}

// One CTA per coefficient: the partial sums of its nparts CTAs, in a fixed order.
__global__ void __launch_bounds__(kSweepThreads)
    sweep_sums_kernel(const double *__restrict__ part, uint32_t nparts, double *__restrict__ sums) {
    __shared__ double red[3][kSweepThreads / 32];
    const double *p = part + (uint64_t)blockIdx.x * nparts * 3;
    double s[3] = {0.0, 0.0, 0.0};
    for (uint32_t i = threadIdx.x; i < nparts; i += kSweepThreads)
        for (int c = 0; c < 3; c++) s[c] = __dadd_rn(s[c], p[(uint64_t)i * 3 + c]);
    for (int c = 0; c < 3; c++) s[c] = warp_sum(s[c]);
    if ((threadIdx.x & 31) == 0)
        for (int c = 0; c < 3; c++) red[c][threadIdx.x >> 5] = s[c];
    __syncthreads();
    if (threadIdx.x < 3) {
        double t = 0.0;
        for (unsigned k = 0; k < kSweepThreads / 32; k++) t = __dadd_rn(t, red[threadIdx.x][k]);
        sums[(uint64_t)blockIdx.x * 3 + threadIdx.x] = t;
    }
}

// Histograms and first positions of each symbol of the streams (hist[] preset to zero, first[] to all
// ones), stream blockIdx.y of n symbols at s + blockIdx.y * n. A CTA takes one contiguous chunk of its
// stream. With at most kStatsShared symbols, it counts and keeps first positions (relative to its chunk)
// in shared memory and folds them into the global tables once; a wider alphabet goes to the global
// tables directly. Reading a first position before lowering it skips the atomic for all but the
// earliest positions of a symbol. One launch for all streams, with 32-bit QBs: 0.35 -> 0.16 ms
// of thirteen streams of 12.5M.
constexpr uint32_t kStatsShared = 4096;

template <class Q>
__global__ void __launch_bounds__(kSweepThreads)
    sweep_stats_kernel(const Q *__restrict__ qb, uint64_t n, const SweepStream *__restrict__ streams,
                       unsigned long long *__restrict__ hists, unsigned long long *__restrict__ firsts) {
    __shared__ uint32_t hsh[kStatsShared], fsh[kStatsShared];
    const SweepStream E = streams[blockIdx.y];
    const Q *s = qb + (uint64_t)blockIdx.y * n;
    unsigned long long *hist = hists + E.at, *first = firsts + E.at;
    const uint64_t chunk = (n + gridDim.x - 1) / gridDim.x;
    const uint64_t c0 = blockIdx.x * chunk, c1 = min(n, c0 + chunk);
    if (E.range <= kStatsShared) {
        const uint32_t range = (uint32_t)E.range;
        for (uint32_t i = threadIdx.x; i < range; i += kSweepThreads) {
            hsh[i] = 0u;
            fsh[i] = 0xffffffffu;
        }
        __syncthreads();
        for (uint64_t j = c0 + threadIdx.x; j < c1; j += kSweepThreads) {
            const uint32_t v = (uint32_t)((int64_t)s[j] - E.offset), r = (uint32_t)(j - c0);
            atomicAdd(&hsh[v], 1u);
            if (fsh[v] > r) atomicMin(&fsh[v], r);
        }
        __syncthreads();
        for (uint32_t i = threadIdx.x; i < range; i += kSweepThreads)
            if (hsh[i]) {
                atomicAdd(&hist[i], (unsigned long long)hsh[i]);
                atomicMin(&first[i], (unsigned long long)(c0 + fsh[i]));
            }
        return;
    }
    for (uint64_t j = c0 + threadIdx.x; j < c1; j += kSweepThreads) {
        const uint64_t v = (uint64_t)((int64_t)s[j] - E.offset);
        atomicAdd(&hist[v], 1ull);
        unsigned long long *slot = first + v;
        if (__ldcg(slot) > j) atomicMin(slot, (unsigned long long)j);
    }
}

uint32_t sweep_predict_grid(const SweepGeom &g) {
    const uint64_t total = g.line_per_thread ? g.lines * ((g.per_line + kSeg - 1) / kSeg) : g.lines * g.per_line;
    const uint64_t want = (total + kSweepThreads - 1) / kSweepThreads;
    return (uint32_t)(want < 148 * 8 ? (want ? want : 1) : 148 * 8);
}

template <class Q>
cudaError_t launch_sweep_predict(const float *d, const SweepGeom &g, const SweepCoef *coef, uint32_t ncoef, double abs_eb,
                                 double neg_2_eb, Q *qb, uint64_t qb_stride, double *part, long long *mm, cudaStream_t st) {
    if (ncoef == 0) return cudaSuccess;
    const dim3 grid(sweep_predict_grid(g), (ncoef + kSweepCoefs - 1) / kSweepCoefs);
    if (g.kind == 2)
        sweep_predict_kernel<Q, true><<<grid, kSweepThreads, 0, st>>>(d, g, coef, ncoef, abs_eb, neg_2_eb, qb, qb_stride, part, mm);
    else
        sweep_predict_kernel<Q, false><<<grid, kSweepThreads, 0, st>>>(d, g, coef, ncoef, abs_eb, neg_2_eb, qb, qb_stride, part, mm);
    count_launch();
    return cudaGetLastError();
}
template cudaError_t launch_sweep_predict<int32_t>(const float *, const SweepGeom &, const SweepCoef *, uint32_t, double, double,
                                                   int32_t *, uint64_t, double *, long long *, cudaStream_t);
template cudaError_t launch_sweep_predict<int64_t>(const float *, const SweepGeom &, const SweepCoef *, uint32_t, double, double,
                                                   int64_t *, uint64_t, double *, long long *, cudaStream_t);

cudaError_t launch_sweep_sums(const double *part, uint32_t nparts, uint32_t ncoef, double *sums, cudaStream_t st) {
    if (ncoef == 0) return cudaSuccess;
    sweep_sums_kernel<<<ncoef, kSweepThreads, 0, st>>>(part, nparts, sums);
    count_launch();
    return cudaGetLastError();
}

template <class Q>
cudaError_t launch_sweep_stats(const Q *qb, uint64_t n, uint32_t ns, const SweepStream *streams, unsigned long long *hists,
                               unsigned long long *firsts, cudaStream_t st) {
    if (n == 0 || ns == 0) return cudaSuccess;
    // Chunks of at least 4096 symbols, so the shared tables' set-up and fold stay small beside them, and
    // of less than 2^32, whose positions the tables hold; about twice the CTAs that are resident.
    const uint64_t want = (n + 4095) / 4096, share = std::max<uint64_t>(148 * 12 / ns, 8);
    const uint64_t x = std::max(std::min(want, share), (n >> 31) + 1);
    sweep_stats_kernel<<<dim3((unsigned)x, ns), kSweepThreads, 0, st>>>(qb, n, streams, hists, firsts);
    count_launch();
    return cudaGetLastError();
}
template cudaError_t launch_sweep_stats<int32_t>(const int32_t *, uint64_t, uint32_t, const SweepStream *, unsigned long long *,
                                                 unsigned long long *, cudaStream_t);
template cudaError_t launch_sweep_stats<int64_t>(const int64_t *, uint64_t, uint32_t, const SweepStream *, unsigned long long *,
                                                 unsigned long long *, cudaStream_t);

}  // namespace asz
