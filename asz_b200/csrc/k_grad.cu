// Differentiable per-block coefficient tuning: a relaxed form of the reference's H1-PSNR proxy
// (get_h_psnr.tpp:6-31) as a function of a continuous t, its derivative, and a tuner that replaces
// the 5-candidate scan (compress.tpp:91-144) by a few projected steps on it.
//
// Samples. Group (block b, round l), indexed b * layers + l like the t stream, has the AB-map
// sample lattice of get_AB_map (get_AB_map.tpp:13-15), but the samples are read OPEN LOOP, from
// the original field: A = (x-1 + x1) - (x-3 + x3) and B = (float)fma(x-3 + x3 + x-1 + x1, 0.25, -x)
// along the round axis, in the reference's float steps (get_AB_map.tpp:18-21). The interior 1D4R
// prediction error is then r(t) = A t + B. Open loop means every round's groups exist at once, so
// one launch covers all of them.
//
// Relaxed proxy of a group (n samples, layer error bound eb, slope from the layer's default slope,
// value range R), to be minimised:
//   q_s = clamp(r_s / (2 eb), -256, 256)                   bin coordinate of sample s
//   p_k = (1/n) sum_s w(q_s - k), w the unit triangle       soft histogram over integer bins
//   H   = -sum_k p_k log2(p_k + 1e-6)                       soft entropy (bits)
//   m   = (1/n) sum_s r_s^2                                 open-loop squared residual
//   mse = m c / (m + c), c = eb^2 / 3                      -> m for small residuals, -> the
//                                                            uniform quantisation noise eb^2/3
//   J   = slope * H - 10 log10(R^2 / mse)                   minus the relaxed score
// dJ/dt follows from dq_s/dt = A_s / (2 eb) (0 where clamped) and dm/dt = (2/n) sum r_s A_s; the
// triangle kernel gives dH/dq_s = (h'(p_{k0+1}) - h'(p_{k0})) / n with k0 = floor(q_s) and
// h'(p) = -(log2(p + 1e-6) + p / ((p + 1e-6) ln 2)).
//
// A warp per group in the forward and backward kernels (a CTA for the largest groups and in the
// tuner), its soft histogram (513 bins) in shared memory; sums in double.
#include <cuda_runtime.h>

#include "dev_common.cuh"
#include "launch.h"
#include "tsel_fast.cuh"

namespace asz {
namespace grad {

constexpr int kHalfBins = 256;              // bins -256..256
constexpr int kBins = 2 * kHalfBins + 2;    // one spare
constexpr float kEps = 1e-6f;
constexpr double kTenOverLn10 = 4.3429448190325175;  // 10 / ln 10
constexpr float kInvLn2 = 1.4426950408889634f;

struct Meta {
    float eb, stat_eb, neg_2_stat_eb, slope;
};

// Bin coordinate, its clamp flag and the lower bin index (0-based in the window).
__device__ __forceinline__ void bin_of(float r, float inv2eb, float &f, int &k0, bool &clamped) {
    float q = r * inv2eb;
    clamped = !(q > -(float)kHalfBins && q < (float)kHalfBins);
    q = fminf(fmaxf(q, -(float)kHalfBins), (float)kHalfBins);
    float fl = floorf(q);
    if (fl >= (float)kHalfBins) fl = (float)kHalfBins - 1.0f;
    f = q - fl;
    k0 = (int)fl + kHalfBins;
}

struct Sums {
    double m, ra, H;  // mean r^2, sum r*A / n, soft entropy
    int klo, khi;     // lowest and highest bin with weight
};

// One CTA (the team: 32 to kMaxTeam threads, 256 by default) per group at a time. Its shared words
// (the soft histogram, h' values, or the judge's counts) are all zero between uses: every pass
// clears what it wrote, and only the bins a group touches are visited.
constexpr int kTeam = 256;
constexpr int kMaxTeam = 512;
constexpr int kTeamWarps = kMaxTeam / 32;
constexpr int kJudgeBins = 2048;              // judge window (quantised-error values)
constexpr uint32_t kMaxJudgeWindows = 128;    // beyond 128 * 2048 bins the judge keeps the default

struct PassShared {
    float hist[kBins];   // soft histogram
    float hp[kBins];     // h'(p) per bin
    double red[kTeamWarps][4];
    int imn[kTeamWarps], imx[kTeamWarps];
};

struct TeamShared : PassShared {
    uint32_t counts[2][kJudgeBins];  // judge: one window of quantised-error counts per candidate
    long long lmn[kTeamWarps], lmx[kTeamWarps];
};

// Sums over the team in a fixed order (warp tree, then warps by index): every thread gets them.
__device__ void team_sum4(TeamShared &sh, double (&v)[4]) {
    for (int o = 16; o; o >>= 1)
        for (int i = 0; i < 4; i++) v[i] += __shfl_xor_sync(0xffffffffu, v[i], o);
    const int w = threadIdx.x >> 5;
    if ((threadIdx.x & 31) == 0)
        for (int i = 0; i < 4; i++) sh.red[w][i] = v[i];
    __syncthreads();
    for (int i = 0; i < 4; i++) v[i] = 0.0;
    for (int k = 0; k < (int)(blockDim.x >> 5); k++)
        for (int i = 0; i < 4; i++) v[i] += sh.red[k][i];
    __syncthreads();
}

__device__ void team_sum3(PassShared &sh, double &a, double &b, double &c) {
    for (int o = 16; o; o >>= 1) {
        a += __shfl_xor_sync(0xffffffffu, a, o);
        b += __shfl_xor_sync(0xffffffffu, b, o);
        c += __shfl_xor_sync(0xffffffffu, c, o);
    }
    const int w = threadIdx.x >> 5;
    if ((threadIdx.x & 31) == 0) {
        sh.red[w][0] = a;
        sh.red[w][1] = b;
        sh.red[w][2] = c;
    }
    __syncthreads();
    a = b = c = 0.0;
    for (int i = 0; i < (int)(blockDim.x >> 5); i++) {
        a += sh.red[i][0];
        b += sh.red[i][1];
        c += sh.red[i][2];
    }
    __syncthreads();
}

template <class T>
__device__ void team_minmax(T (&mn)[kTeamWarps], T (&mx)[kTeamWarps], T &lo, T &hi) {
    for (int o = 16; o; o >>= 1) {
        const T l2 = __shfl_xor_sync(0xffffffffu, lo, o), h2 = __shfl_xor_sync(0xffffffffu, hi, o);
        lo = l2 < lo ? l2 : lo;
        hi = h2 > hi ? h2 : hi;
    }
    const int w = threadIdx.x >> 5;
    if ((threadIdx.x & 31) == 0) {
        mn[w] = lo;
        mx[w] = hi;
    }
    __syncthreads();
    for (int i = 0; i < (int)(blockDim.x >> 5); i++) {
        lo = mn[i] < lo ? mn[i] : lo;
        hi = mx[i] > hi ? mx[i] : hi;
    }
    __syncthreads();
}

// Soft histogram of the group's samples at t and the sums. keep: leave the histogram for
// group_grad (which clears it); otherwise it is cleared here.
__device__ Sums group_pass(PassShared &sh, const float *__restrict__ A, const float *__restrict__ B, uint32_t n,
                           const Meta &mt, float t, bool keep) {
    const float inv2eb = 0.5f / mt.eb;
    double m = 0.0, ra = 0.0, H = 0.0;
    int klo = kBins, khi = -1;
    for (uint32_t s = threadIdx.x; s < n; s += blockDim.x) {
        const float a = A[s], r = fmaf(a, t, B[s]);
        float f;
        int k0;
        bool cl;
        bin_of(r, inv2eb, f, k0, cl);
        atomicAdd(&sh.hist[k0], 1.0f - f);
        atomicAdd(&sh.hist[k0 + 1], f);
        klo = min(klo, k0);
        khi = max(khi, k0 + 1);
        m += (double)r * r;
        ra += (double)r * a;
    }
    team_minmax(sh.imn, sh.imx, klo, khi);  // its barriers also complete the histogram
    const float inv_n = 1.0f / (float)n;
    for (int i = klo + (int)threadIdx.x; i <= khi; i += blockDim.x) {
        const float p = sh.hist[i] * inv_n;
        const float l2 = log2f(p + kEps);
        if (p > 0.0f) H -= (double)p * (double)l2;
        if (keep) sh.hp[i] = -(l2 + p / (p + kEps) * kInvLn2);  // h'(p) for group_grad
        sh.hist[i] = 0.0f;
    }
    team_sum3(sh, m, ra, H);
    return Sums{m / n, ra / n, H, klo, khi};
}

__device__ __forceinline__ double objective(const Sums &S, const Meta &mt, float R2) {
    const double c = (double)mt.eb * mt.eb / 3.0;
    const double mse = fmax(S.m * c / (S.m + c), 1e-300);
    return (double)mt.slope * S.H - 10.0 * log10((double)R2 / mse);
}

// dJ/dt from the sums and the samples' sum of dH/dq dq/dt.
__device__ __forceinline__ double gradient(const Sums &S, double gh, uint32_t n, const Meta &mt) {
    const double c = (double)mt.eb * mt.eb / 3.0;
    const double dlog = S.m > 0.0 ? c / (S.m * (S.m + c)) : 0.0;
    return (double)mt.slope * (gh / n) + kTenOverLn10 * dlog * 2.0 * S.ra;
}

// dJ/dt after group_pass(keep) at the same t, from the h' values it left (the barriers of its
// final reduction made them visible).
__device__ double group_grad(PassShared &sh, const float *__restrict__ A, const float *__restrict__ B, uint32_t n,
                             const Meta &mt, float t, const Sums &S) {
    const float inv2eb = 0.5f / mt.eb;
    double gh = 0.0, u0 = 0.0, u1 = 0.0;
    for (uint32_t s = threadIdx.x; s < n; s += blockDim.x) {
        const float a = A[s], r = fmaf(a, t, B[s]);
        float f;
        int k0;
        bool cl;
        bin_of(r, inv2eb, f, k0, cl);
        if (!cl) gh += (double)(sh.hp[k0 + 1] - sh.hp[k0]) * (double)(a * inv2eb);
    }
    team_sum3(sh, gh, u0, u1);  // its barriers end the reads of h'
    return gradient(S, gh, n, mt);
}

__device__ __forceinline__ Meta load_meta(const float4 *meta, uint64_t g) {
    const float4 v = meta[g];
    Meta m{v.x, v.y, v.z, v.w};
    if (!isfinite(m.slope)) m.slope = 0.0f;
    return m;
}

__device__ __forceinline__ void team_clear(TeamShared &sh) {
    for (int i = threadIdx.x; i < kBins; i += blockDim.x) sh.hist[i] = 0.0f;
    for (int i = threadIdx.x; i < 2 * kJudgeBins; i += blockDim.x) (&sh.counts[0][0])[i] = 0u;
    __syncthreads();
}

// J (kGrad false) or dJ/dt times its incoming gradient (true) of every group, a warp per group.
//
// A group is 3 to 1600 samples in the plans met in use: a CTA of 256 threads spent its time at the
// barriers between its passes, ten groups one after another, and on float atomics in shared memory,
// which are compare-and-swap loops (256^3 field, 12k groups, 38 MB of samples: 100 us forward, 122
// backward). A warp per group needs no barrier and has 40 groups an SM under way; the histogram is in
// whole numbers, whose atomics are single instructions and whose sums are exact in any order: 35 us
// forward, 51 backward. It is the latency of a group's chain of loads (of 8 and 16 loads in flight a lane and
// 4 to 8 CTAs an SM, sixteen and five were the best). Above kWarpMost samples a group is a CTA's.
//
// The weights are those that a float has, and more. A bin has two words: how many samples begin in it
// and the sum of their fractions f, of which a sample weighs 1 - f in its bin and f in the next. f is
// taken in steps of 2^-T: the sum's leading bits are in one word, its last ones below the count in the
// other, so that 4095 samples leave T = 28, and 2047 and fewer 31. A coordinate of 1/32 and more, or a
// negative one (rounded when it moves up to its bin), is a whole number of such steps already; what
// the ones between 0 and 1/32 have below a step is summed beside them. (One word a bin, of steps of 2^-20 in
// the largest groups, took 31 and 47 us, and where samples weigh a millionth of a bin, the gradient was off by
// 200 times what a float's rounding explains.)
constexpr uint32_t kWarpMost = 4095;
constexpr int kProxyThreads = 256;
constexpr int kInFlight = 8;  // samples a lane loads ahead (two words each)

// The words of a bin for groups of n samples.
struct FracWords {
    int frac, low;  // bits of the fractions' leading part, below the counts too, and of their last part
    __device__ __forceinline__ explicit FracWords(uint32_t n) {
        frac = __clz(n);
        low = min(2 * frac - 32, 31 - frac);
    }
    // n < 2^(32 - frac): the counts fit above 2^frac, n last parts (at most 2^low) below it, and n
    // leading parts (at most 2^frac) a word.
    __device__ __forceinline__ float one() const { return __uint_as_float((uint32_t)(127 + frac + low) << 23); }
    __device__ __forceinline__ long long sum(uint32_t count, uint32_t lead) const {  // of the fractions, in steps
        return ((long long)lead << low) + (count & ((1u << frac) - 1));
    }
    __device__ __forceinline__ long long samples(uint32_t count) const { return (long long)(count >> frac) << (frac + low); }
};

template <bool kGrad>
__device__ double warp_proxy(uint32_t *counts, uint32_t *leads, const float *__restrict__ A, const float *__restrict__ B, uint32_t n,
                             const Meta &mt, float t, float R2) {
    const int lane = threadIdx.x & 31;
    const float inv2eb = 0.5f / mt.eb;
    const FracWords F(n);
    const float one = F.one();
    const uint32_t low_mask = (1u << F.low) - 1;
    const uint32_t unit = 1u << F.frac;
    double m = 0.0, ra = 0.0, H = 0.0;
    float below = 0.0f;
    int klo = kBins, khi = -1;
    for (uint32_t s0 = lane; s0 < n; s0 += 32 * kInFlight) {
        float a[kInFlight], b[kInFlight];
#pragma unroll
        for (int i = 0; i < kInFlight; i++) {
            const uint32_t s = s0 + 32 * i;
            a[i] = s < n ? A[s] : 0.0f;
            b[i] = s < n ? B[s] : 0.0f;
        }
#pragma unroll
        for (int i = 0; i < kInFlight; i++) {
            if (s0 + 32 * i >= n) break;
            const float r = fmaf(a[i], t, b[i]);
            float f;
            int k0;
            bool cl;
            bin_of(r, inv2eb, f, k0, cl);
            const uint32_t w = __float2uint_rn(f * one);
            if (k0 == kHalfBins && f < 0x1p-5f) below += f * one - (float)w;
            atomicAdd(&counts[k0], unit + (w & low_mask));
            atomicAdd(&leads[k0], w >> F.low);
            klo = min(klo, k0);
            khi = max(khi, k0 + 1);
            m = fma((double)r, (double)r, m);
            ra = fma((double)r, (double)a[i], ra);
        }
    }
    klo = __reduce_min_sync(0xffffffffu, klo);
    khi = __reduce_max_sync(0xffffffffu, khi);
    if (__any_sync(0xffffffffu, below != 0.0f))
        for (int o = 16; o; o >>= 1) below += __shfl_xor_sync(0xffffffffu, below, o);
    __syncwarp();
    const float inv = 1.0f / ((float)n * one);
    // From the last bins on, as a bin takes the fractions of the one before.
    for (int i0 = klo + (khi - klo) / 32 * 32; i0 >= klo; i0 -= 32) {
        const int i = i0 + lane;
        float w = 0.0f;
        if (i <= khi) {
            const uint32_t c = counts[i];
            long long v = F.samples(c) - F.sum(c, leads[i]);
            if (i > klo) v += F.sum(counts[i - 1], leads[i - 1]);
            w = __ll2float_rn(v);
            if (i == kHalfBins) w -= below;
            if (i == kHalfBins + 1) w += below;
        }
        __syncwarp();
        if (i <= khi) {
            const float p = w * inv;
            const float l2 = log2f(p + kEps);
            H -= (double)p * (double)l2;
            // h'(p) takes the count's place until the gradient's pass
            counts[i] = kGrad ? __float_as_uint(-(l2 + p / (p + kEps) * kInvLn2)) : 0u;
            leads[i] = 0u;
        }
    }
    for (int o = 16; o; o >>= 1) {
        m += __shfl_xor_sync(0xffffffffu, m, o);
        ra += __shfl_xor_sync(0xffffffffu, ra, o);
        if (!kGrad) H += __shfl_xor_sync(0xffffffffu, H, o);
    }
    const Sums S{m / n, ra / n, H, klo, khi};
    __syncwarp();
    if (!kGrad) return objective(S, mt, R2);
    double gh = 0.0;
    for (uint32_t s0 = lane; s0 < n; s0 += 32 * kInFlight) {
        float a[kInFlight], b[kInFlight];
#pragma unroll
        for (int i = 0; i < kInFlight; i++) {
            const uint32_t s = s0 + 32 * i;
            a[i] = s < n ? A[s] : 0.0f;
            b[i] = s < n ? B[s] : 0.0f;
        }
#pragma unroll
        for (int i = 0; i < kInFlight; i++) {
            if (s0 + 32 * i >= n) break;
            float f;
            int k0;
            bool cl;
            bin_of(fmaf(a[i], t, b[i]), inv2eb, f, k0, cl);
            if (!cl)
                gh = fma((double)(__uint_as_float(counts[k0 + 1]) - __uint_as_float(counts[k0])), (double)(a[i] * inv2eb), gh);
        }
    }
    for (int o = 16; o; o >>= 1) gh += __shfl_xor_sync(0xffffffffu, gh, o);
    __syncwarp();
    for (int i = klo + lane; i <= khi; i += 32) counts[i] = 0u;
    __syncwarp();
    return gradient(S, gh, n, mt);
}

template <bool kGrad>
__global__ void __launch_bounds__(kProxyThreads, 5)
    proxy_kernel(const float *__restrict__ A, const float *__restrict__ B, const uint32_t *__restrict__ off,
                 const float4 *__restrict__ meta, float R2, const float *__restrict__ t, const float *__restrict__ gJ,
                 uint64_t groups, float *__restrict__ out) {
    constexpr uint32_t kWarps = kProxyThreads / 32;
    __shared__ union Both {
        uint32_t warp[kWarps][2][kBins];
        PassShared team;
        __device__ Both() {}
    } sh;
    const uint32_t w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int i = lane; i < 2 * kBins; i += 32) sh.warp[w][0][i] = 0u;
    __syncwarp();
    for (uint64_t g = blockIdx.x * (uint64_t)kWarps + w; g < groups; g += (uint64_t)gridDim.x * kWarps) {
        const uint32_t o = off[g], n = off[g + 1] - o;
        if (n > kWarpMost) continue;
        double v = 0.0;
        if (n) v = warp_proxy<kGrad>(sh.warp[w][0], sh.warp[w][1], A + o, B + o, n, load_meta(meta, g), t[g], R2);
        if (lane == 0) out[g] = n == 0 ? 0.0f : kGrad ? (float)(v * (double)gJ[g]) : (float)v;
    }
    bool cleared = false;
    for (uint64_t g = blockIdx.x; g < groups; g += gridDim.x) {
        const uint32_t o = off[g], n = off[g + 1] - o;
        if (n <= kWarpMost) continue;
        if (!cleared) {
            __syncthreads();
            for (int i = threadIdx.x; i < kBins; i += blockDim.x) sh.team.hist[i] = 0.0f;
            __syncthreads();
            cleared = true;
        }
        const Meta mt = load_meta(meta, g);
        const Sums S = group_pass(sh.team, A + o, B + o, n, mt, t[g], kGrad);
        const double v = kGrad ? group_grad(sh.team, A + o, B + o, n, mt, t[g], S) * (double)gJ[g] : objective(S, mt, R2);
        if (threadIdx.x == 0) out[g] = (float)v;
    }
}

// The reference's proxy scores -slope * h1 + psnr of candidates t[0] and t[1] (get_h_psnr.tpp:6-31
// on the keys of get_AB_map.tpp:18-21), with order-free double sums. One pass computes both
// candidates' errors and counts them in a window placed on sample 0's bin; a candidate whose
// errors spread beyond it is counted again window by window. Returns false when some candidate's
// errors span more than kMaxJudgeWindows windows.
__device__ bool exact_scores(TeamShared &sh, const float *__restrict__ A, const float *__restrict__ B, uint32_t n,
                             const Meta &mt, float R2, const float (&t)[2], double (&score)[2]) {
    const float neg_eb = __fdiv_rn(0.5f, mt.eb), eb2 = __fadd_rn(mt.eb, mt.eb);
    const float t2[2] = {__fadd_rn(t[0], t[0]), __fadd_rn(t[1], t[1])};
    long long w0[2], lo[2] = {LLONG_MAX, LLONG_MAX}, hi[2] = {LLONG_MIN, LLONG_MIN};
    {
        float af, bf;
        bool nz;
        fastsel::keys_of_ab(A[0], B[0], mt.neg_2_stat_eb, af, bf, nz);
        for (int c = 0; c < 2; c++)
            w0[c] = lround_f(__fmul_rn(fastsel::cand_err(af, bf, t2[c], mt.stat_eb), neg_eb)) - kJudgeBins / 2;
    }
    double acc[4] = {0.0, 0.0, 0.0, 0.0};  // mse[0], mse[1], h1[0], h1[1]
    for (uint32_t s = threadIdx.x; s < n; s += blockDim.x) {
        float af, bf;
        bool nz;
        fastsel::keys_of_ab(A[s], B[s], mt.neg_2_stat_eb, af, bf, nz);
        for (int c = 0; c < 2; c++) {
            const float err = fastsel::cand_err(af, bf, t2[c], mt.stat_eb);
            const long long q = lround_f(__fmul_rn(err, neg_eb));
            const float de = __fmaf_rn(-__ll2float_rn(q), eb2, err);
            acc[c] += (double)de * de;
            lo[c] = q < lo[c] ? q : lo[c];
            hi[c] = q > hi[c] ? q : hi[c];
            if (q >= w0[c] && q - w0[c] < kJudgeBins) atomicAdd(&sh.counts[c][q - w0[c]], 1u);
        }
    }
    for (int c = 0; c < 2; c++) team_minmax(sh.lmn, sh.lmx, lo[c], hi[c]);
    bool ok = true;
    for (int c = 0; c < 2; c++) {
        uint32_t *cnt = sh.counts[c];
        const bool fits = lo[c] >= w0[c] && hi[c] - w0[c] < kJudgeBins;
        if (fits) {
            for (int i = (int)(lo[c] - w0[c]) + threadIdx.x; i <= (int)(hi[c] - w0[c]); i += blockDim.x) {
                const uint32_t k = cnt[i];
                if (k) {
                    const double p = (double)k / n;
                    acc[2 + c] -= p * log2(p);
                    cnt[i] = 0u;
                }
            }
            continue;
        }
        for (int i = threadIdx.x; i < kJudgeBins; i += blockDim.x) cnt[i] = 0u;
        __syncthreads();
        if ((unsigned long long)(hi[c] - lo[c]) / kJudgeBins >= kMaxJudgeWindows) {
            ok = false;
            continue;
        }
        for (long long w = lo[c]; w <= hi[c]; w += kJudgeBins) {
            for (uint32_t s = threadIdx.x; s < n; s += blockDim.x) {
                float af, bf;
                bool nz;
                fastsel::keys_of_ab(A[s], B[s], mt.neg_2_stat_eb, af, bf, nz);
                const long long q = lround_f(__fmul_rn(fastsel::cand_err(af, bf, t2[c], mt.stat_eb), neg_eb));
                if (q >= w && q - w < kJudgeBins) atomicAdd(&cnt[q - w], 1u);
            }
            __syncthreads();
            const int top = (int)min((long long)kJudgeBins - 1, hi[c] - w);
            for (int i = threadIdx.x; i <= top; i += blockDim.x) {
                const uint32_t k = cnt[i];
                if (k) {
                    const double p = (double)k / n;
                    acc[2 + c] -= p * log2(p);
                    cnt[i] = 0u;
                }
            }
            __syncthreads();
        }
    }
    team_sum4(sh, acc);
    for (int c = 0; c < 2; c++) {
        const double psnr = acc[c] > 0.0 ? 10.0 * log10((double)R2 * n / acc[c]) : INFINITY;
        score[c] = -(double)mt.slope * acc[2 + c] + psnr;
    }
    return ok;
}

// All of a group's tuning in one CTA: `steps` projected sign-gradient steps on J from t = 1/4 with
// step sizes step0 * 2^-k, inside [t_min, t_max]; the result snapped to the t grid; then the
// reference's proxy judges the snapped t against the default 1/4 and keeps the default unless
// the snapped t scores higher (the acceptance test of compress.tpp:136-140).
// stats: [0] groups tuned, [1] snapped t accepted, [2] quantised errors spread over more than
// kMaxJudgeWindows * kJudgeBins bins, so the judge kept the default.
// The steps see at most kStage samples of a group, staged in shared memory: every k-th sample,
// k = ceil(n / step_cap) (step_cap <= kStage; 0 means kStage). The judge sees all of them.
constexpr uint32_t kStage = 1024;

__global__ void __launch_bounds__(kMaxTeam)
    tune_kernel(const float *__restrict__ A, const float *__restrict__ B, const uint32_t *__restrict__ off,
                const float4 *__restrict__ meta, float R2, uint64_t groups, float t_min, float t_max, int32_t tp,
                uint32_t steps, float step0, uint32_t step_cap, int64_t *__restrict__ t_codes,
                float *__restrict__ t_relaxed, uint32_t *__restrict__ stats) {
    __shared__ TeamShared sh;
    __shared__ float sA[kStage], sB[kStage];
    if (step_cap == 0 || step_cap > kStage) step_cap = kStage;
    team_clear(sh);
    const int64_t code_lo = lround_f(__fmul_rn(t_min, (float)tp)), code_hi = lround_f(__fmul_rn(t_max, (float)tp));
    const int64_t code_def = lround_f(__fmul_rn(0.25f, (float)tp));
    for (uint64_t g = blockIdx.x; g < groups; g += gridDim.x) {
        const uint32_t o = off[g], n = off[g + 1] - o;
        if (n == 0) {
            if (threadIdx.x == 0) {
                t_codes[g] = code_def;
                if (t_relaxed) t_relaxed[g] = 0.25f;
            }
            continue;
        }
        const Meta mt = load_meta(meta, g);
        // The steps read their samples many times: stage them.
        const uint32_t stride = (n + step_cap - 1) / step_cap, ns = (n + stride - 1) / stride;
        __syncthreads();  // the previous group's passes are done with sA, sB
        for (uint32_t s = threadIdx.x; s < ns; s += blockDim.x) {
            sA[s] = A[o + s * stride];
            sB[s] = B[o + s * stride];
        }
        __syncthreads();
        float t = 0.25f, step = step0;
        for (uint32_t k = 0; k < steps; k++, step *= 0.5f) {
            const Sums S = group_pass(sh, sA, sB, ns, mt, t, true);
            const double d = group_grad(sh, sA, sB, ns, mt, t, S);
            if (d > 0.0) t -= step;
            else if (d < 0.0) t += step;
            t = fminf(fmaxf(t, t_min), t_max);
        }
        int64_t code = lround_f(__fmul_rn(t, (float)tp));
        code = code < code_lo ? code_lo : (code > code_hi ? code_hi : code);
        int64_t chosen = code_def;
        if (code != code_def) {
            const float cand[2] = {0.25f, (float)code / (float)tp};
            double sc[2];
            const bool ok = exact_scores(sh, A + o, B + o, n, mt, R2, cand, sc);
            if (!ok) {
                if (threadIdx.x == 0) atomicAdd(&stats[2], 1u);
            } else if (sc[1] - sc[0] > 0.0) {
                chosen = code;
                if (threadIdx.x == 0) atomicAdd(&stats[1], 1u);
            }
        }
        if (threadIdx.x == 0) {
            atomicAdd(&stats[0], 1u);
            t_codes[g] = chosen;
            if (t_relaxed) t_relaxed[g] = t;
        }
    }
}

// Open-loop AB samples of every group (see the file comment). One CTA per group; positions as in
// the fast selection (origin 0). err: bit 0 when a group's lattice does not hold off[] samples.
__global__ void __launch_bounds__(256)
    gather_kernel(FieldGeom fg, const RoundGeom *__restrict__ rounds, const ClassInfo *__restrict__ classes,
                  const float *__restrict__ x, const uint32_t *__restrict__ off, uint64_t groups, float *__restrict__ A,
                  float *__restrict__ B, uint32_t *err) {
    const uint32_t L = fg.layer_num;
    for (uint64_t gid = blockIdx.x; gid < groups; gid += gridDim.x) {
        const uint32_t o = off[gid], n = off[gid + 1] - o;
        if (n == 0) continue;
        const uint64_t g = gid / L, l = gid - g * L;
        const RoundGeom &rg = rounds[l];
        const uint64_t b2 = g % fg.block_num[2], b1 = (g / fg.block_num[2]) % fg.block_num[1],
                       b0 = g / (fg.block_num[1] * fg.block_num[2]);
        const uint64_t bb[3] = {b0, b1, b2};
        const int cls = (fastsel::class_of(b0, fg.block_num[0]) * 3 + fastsel::class_of(b1, fg.block_num[1])) * 3 +
                        fastsel::class_of(b2, fg.block_num[2]);
        const ClassInfo ci = classes[27 * l + cls];
        fastsel::FastSampleGeo sg;
        uint32_t cnt[3];
        const int d = rg.dir;
        for (int a = 0; a < 3; a++) {
            uint64_t lo = bb[a] * fg.block_shape[a];
            uint64_t hi = min((bb[a] + 1) * fg.block_shape[a] + 1, fg.n[a]);
            if (a != d && lo != 0) lo += rg.stride[a];
            if (a == d) {
                lo += 3 * rg.stride[a] / 2;
                hi -= 3 * rg.stride[a] / 2;
            }
            sg.lo[a] = lo;
            sg.step[a] = rg.stride[a] * ci.ss;
            cnt[a] = (uint32_t)((hi - lo + sg.step[a] - 1) / sg.step[a]);
        }
        if ((uint64_t)cnt[0] * cnt[1] * cnt[2] != n) {
            if (threadIdx.x == 0) atomicOr(err, 1u);
            continue;
        }
        sg.cnt2 = cnt[2];
        sg.c2 = fastsel::small_div(cnt[2]);
        sg.c12 = fastsel::small_div(cnt[1] * cnt[2]);
        for (uint32_t s = threadIdx.x; s < n; s += blockDim.x) {
            const uint64_t p = fastsel::fast_sample_pos(sg, s, fg.n[1], fg.n[2]), dd = rg.dist;
            const float m1 = x[p - dd], m3 = x[p - 3 * dd], p1 = x[p + dd], p3 = x[p + 3 * dd];
            A[o + s] = __fsub_rn(__fadd_rn(m1, p1), __fadd_rn(m3, p3));
            const float S4 = __fadd_rn(__fadd_rn(p1, p3), __fadd_rn(m1, m3));
            B[o + s] = __double2float_rn(__fma_rn((double)S4, 0.25, -(double)x[p]));
        }
    }
}

unsigned grid_for(uint64_t items, unsigned per_cta) {
    uint64_t b = (items + per_cta - 1) / per_cta;
    const uint64_t cap = 148ull * 8;
    return (unsigned)(b < 1 ? 1 : (b > cap ? cap : b));
}

// Grid of the forward and backward kernels: a group a warp, eight CTAs an SM.
unsigned proxy_grid(uint64_t groups) { return grid_for(groups, kProxyThreads / 32); }

// Grid of the gather and the tuner: one group per CTA at a time, up to 16 CTAs per SM.
unsigned group_grid(uint64_t groups) {
    const uint64_t cap = 148ull * 16;
    return (unsigned)(groups < 1 ? 1 : (groups > cap ? cap : groups));
}

}  // namespace grad

cudaError_t launch_grad_gather(const FieldGeom &fg, const RoundGeom *rounds, const ClassInfo *classes, const float *x,
                               const uint32_t *off, uint64_t groups, float *A, float *B, uint32_t *err, cudaStream_t st) {
    if (groups == 0) return cudaSuccess;
    grad::gather_kernel<<<grad::group_grid(groups), 256, 0, st>>>(fg, rounds, classes, x, off, groups, A, B, err);
    count_launch();
    return cudaGetLastError();
}

}  // namespace asz

using namespace asz;

extern "C" int asz_grad_forward(const float *A, const float *B, const uint32_t *offsets, const float *meta, float R2,
                                const float *t, uint64_t groups, float *J, void *cuda_stream) {
    if (groups == 0) return 0;
    if (!A || !B || !offsets || !meta || !t || !J) return 1;
    grad::proxy_kernel<false><<<grad::proxy_grid(groups), grad::kProxyThreads, 0, (cudaStream_t)cuda_stream>>>(
        A, B, offsets, (const float4 *)meta, R2, t, nullptr, groups, J);
    count_launch();
    return cudaGetLastError() == cudaSuccess ? 0 : 7;
}

extern "C" int asz_grad_backward(const float *A, const float *B, const uint32_t *offsets, const float *meta, float R2,
                                 const float *t, const float *grad_J, uint64_t groups, float *grad_t, void *cuda_stream) {
    if (groups == 0) return 0;
    if (!A || !B || !offsets || !meta || !t || !grad_J || !grad_t) return 1;
    grad::proxy_kernel<true><<<grad::proxy_grid(groups), grad::kProxyThreads, 0, (cudaStream_t)cuda_stream>>>(
        A, B, offsets, (const float4 *)meta, R2, t, grad_J, groups, grad_t);
    count_launch();
    return cudaGetLastError() == cudaSuccess ? 0 : 7;
}

extern "C" int asz_grad_tune(const float *A, const float *B, const uint32_t *offsets, const float *meta, float R2,
                             uint64_t groups, float t_min, float t_max, int32_t t_precision, uint32_t steps, float step0,
                             uint32_t step_cap, uint32_t team, int64_t *t_codes, float *t_relaxed, uint32_t *stats,
                             void *cuda_stream) {
    if (groups == 0) return 0;
    if (team == 0) team = grad::kTeam;
    if (!A || !B || !offsets || !meta || !t_codes || !stats || t_precision <= 0 || !(t_min <= t_max) || team % 32 ||
        team > (uint32_t)grad::kMaxTeam)
        return 1;
    grad::tune_kernel<<<grad::group_grid(groups), team, 0, (cudaStream_t)cuda_stream>>>(
        A, B, offsets, (const float4 *)meta, R2, groups, t_min, t_max, t_precision, steps, step0, step_cap, t_codes, t_relaxed,
        stats);
    count_launch();
    return cudaGetLastError() == cudaSuccess ? 0 : 7;
}
