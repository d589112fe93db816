// Plan search (c_codes/asz_core/generate_config.tpp:444-678) on the device: the sampled open-loop
// compression of every candidate predictor of a layer in one launch, and the candidates' squared
// error sums in the reference's sequential order.
#include <cuda_runtime.h>

#include "dev_common.cuh"
#include "float_chain.cuh"
#include "launch.h"

namespace asz {
namespace {

// dot_sample_compress (generate_config.tpp:227-254) as GCC emits it for the reference build: the
// edge stencils below, the interior 1D4R in double with a float product in between, the residual
// quantised in float (diff * neg_2_eb) and e = fmaf(-eb, (float)(2 * qb), diff) for the error sum.
//
// A row of CTAs per candidate (grid y), so the loop nest's divisors are the CTA's own and the QB
// extremes are reduced in the CTA before they reach the candidate's two words: one pair of atomics
// a CTA. Every thread's own pair, on the same two words, was most of the kernel (100x500x500, the
// search's 14 layers, nine candidates of 0.5 M samples in the first: 11.1 ms with it, 0.24 without).
// The QBs are counted on the way, in a window of kPlanWin bins around zero (hist: a window a
// candidate, zero before); a candidate whose counts do not add up has QBs outside it and is counted
// by the host's own launch. A window's set-up and fold are 4096 shared words a CTA, so a CTA has some
// thousand samples.
constexpr int kSampleThreads = 256;

__global__ void __launch_bounds__(kSampleThreads)
    plan_sample_kernel(const float *__restrict__ d, uint64_t n1, uint64_t n2, const PlanCand *__restrict__ cands,
                       int32_t *__restrict__ qb_out, float *__restrict__ e_out, int32_t *__restrict__ qb_range,
                       unsigned long long *__restrict__ hist) {
    __shared__ uint32_t hsh[kPlanWin];
    __shared__ int32_t rlo[kSampleThreads / 32], rhi[kSampleThreads / 32];
    const PlanCand &c = cands[blockIdx.y];
    const uint64_t n = c.cnt[0] * c.cnt[1] * c.cnt[2];
    const int a0 = c.ax[0], a1 = c.ax[1], a2 = c.ax[2];  // loop nest: outer to inner
    const uint64_t c2 = c.cnt[a2], c1 = c.cnt[a1];
    const uint64_t lo0 = c.lo[a0], lo1 = c.lo[a1], lo2 = c.lo[a2], st0 = c.st[a0], st1 = c.st[a1], st2 = c.st[a2];
    auto extent = [&](int a) { return a == 0 ? n1 * n2 : a == 1 ? n2 : (uint64_t)1; };
    const uint64_t x0 = extent(a0), x1 = extent(a1), x2 = extent(a2);
    const int dir = c.dir;
    const double td = (double)c.t;
    const float neg_2_eb = c.neg_2_eb, eb = c.eb;
    int32_t *const qb = qb_out + c.off;
    float *const eo = e_out + c.off;
    const uint64_t hs = c.hs, right = c.right, dist = c.dist;
    const bool narrow = n < (1ull << 32);
    for (uint32_t i = threadIdx.x; i < kPlanWin; i += blockDim.x) hsh[i] = 0u;
    __syncthreads();
    int32_t lo = INT32_MAX, hi = INT32_MIN;
    for (uint64_t kl = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; kl < n; kl += (uint64_t)gridDim.x * blockDim.x) {
        uint64_t k0, k1, k2;
        if (narrow) {  // 32-bit divisions
            const uint32_t r = (uint32_t)kl / (uint32_t)c2;
            k2 = (uint32_t)kl - r * (uint32_t)c2;
            k0 = r / (uint32_t)c1;
            k1 = r - (uint32_t)k0 * (uint32_t)c1;
        } else {
            const uint64_t r = kl / c2;
            k2 = kl - r * c2;
            k0 = r / c1;
            k1 = r - k0 * c1;
        }
        const uint64_t i0 = lo0 + k0 * st0, i1 = lo1 + k1 * st1, i2 = lo2 + k2 * st2;
        const uint64_t pos = i0 * x0 + i1 * x1 + i2 * x2;
        const uint64_t i = dir == a0 ? i0 : dir == a1 ? i1 : i2;
        const float xm1 = d[pos - dist];
        float pred;
        if (i <= hs) {
            if (i + hs >= right) pred = xm1;
            else if (i + 3 * hs >= right) pred = __fmul_rn(__fadd_rn(d[pos + dist], xm1), 0.5f);
            else pred = __fmul_rn(__fmaf_rn(d[pos + dist], 6.0f, __fmaf_rn(xm1, 3.0f, -d[pos + 3 * dist])), 0.125f);
        } else {
            const float xm3 = d[pos - 3 * dist];
            if (i + hs >= right) {
                pred = __fmul_rn(__fmaf_rn(xm1, 3.0f, -xm3), 0.5f);
            } else if (i + 3 * hs >= right) {
                pred = __fmul_rn(__fsub_rn(__fmaf_rn(xm1, 6.0f, __fmul_rn(d[pos + dist], 3.0f)), xm3), 0.125f);
            } else {
                const float s1 = __fadd_rn(d[pos + dist], xm1), s3 = __fadd_rn(xm3, d[pos + 3 * dist]);
                const float p1 = __double2float_rn(__dmul_rn((double)s3, __dsub_rn(0.25, td)));
                pred = __double2float_rn(__fma_rn(__dadd_rn(0.25, td), (double)s1, (double)p1));
            }
        }
        const float diff = __fsub_rn(pred, d[pos]);
        const int32_t q = (int32_t)lround_f(__fmul_rn(diff, neg_2_eb));
        const float q2 = __int2float_rn((int32_t)((uint32_t)q * 2u));
        qb[kl] = q;
        eo[kl] = __fmaf_rn(-eb, q2, diff);
        lo = min(lo, q);
        hi = max(hi, q);
        const uint32_t bin = (uint32_t)q + kPlanWin / 2;
        if (bin < kPlanWin) atomicAdd(&hsh[bin], 1u);
    }
    lo = __reduce_min_sync(0xffffffffu, lo);
    hi = __reduce_max_sync(0xffffffffu, hi);
    if ((threadIdx.x & 31) == 0) {
        rlo[threadIdx.x >> 5] = lo;
        rhi[threadIdx.x >> 5] = hi;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < kSampleThreads / 32; w++) {
            lo = min(lo, rlo[w]);
            hi = max(hi, rhi[w]);
        }
        if (lo <= hi) {
            atomicMin(&qb_range[2 * blockIdx.y], lo);
            atomicMax(&qb_range[2 * blockIdx.y + 1], hi);
        }
    }
    for (uint32_t i = threadIdx.x; i < kPlanWin; i += blockDim.x)
        if (hsh[i]) atomicAdd(&hist[(uint64_t)blockIdx.y * kPlanWin + i], (unsigned long long)hsh[i]);
}

// mse = fmaf(e, e, mse) over each candidate's samples in loop order, the reference's float sum
// (generate_config.tpp:227-254), bit for bit: a CTA per candidate over batches of 8192 terms
// (float_chain.cuh). For the same 14 layers a warp per candidate with batches of 256 took 3.6 ms,
// a CTA each takes 0.56: what is left is the scan and two barriers a batch, and one more pass for
// each of the sum's binades.
constexpr int kMsePer = 8;

__global__ void __launch_bounds__(1024) plan_mse_kernel(const PlanCand *__restrict__ cands, const float *__restrict__ e,
                                                        float *__restrict__ mse_out) {
    __shared__ ChainShared sh;
    const PlanCand &c = cands[blockIdx.x];
    const uint64_t n = c.cnt[0] * c.cnt[1] * c.cnt[2];
    const float *p = e + c.off;  // off is a multiple of kPlanAlign
    const float mse = block_chain<kMsePer>(
        sh, 0.0f, n,
        [&](uint64_t k, float (&x)[kMsePer]) {
            if (k + kMsePer <= n) {
                const float4 u = *reinterpret_cast<const float4 *>(p + k), v = *reinterpret_cast<const float4 *>(p + k + 4);
                x[0] = u.x, x[1] = u.y, x[2] = u.z, x[3] = u.w;
                x[4] = v.x, x[5] = v.y, x[6] = v.z, x[7] = v.w;
            } else {
                for (int i = 0; i < kMsePer; i++) x[i] = k + i < n ? p[k + i] : 0.0f;
            }
        },
        [](float s, float x) { return __fmaf_rn(x, x, s); });
    if (threadIdx.x == 0) mse_out[blockIdx.x] = mse;
}

}  // namespace

cudaError_t launch_plan_sample(const float *d, uint64_t n1, uint64_t n2, const PlanCand *cands, uint32_t ncands, uint64_t most,
                               int32_t *qb, float *e, int32_t *qb_range, unsigned long long *hist, cudaStream_t st) {
    if (most == 0 || ncands == 0) return cudaSuccess;
    // CTAs a candidate: 1024 samples each, and about 8 an SM over all candidates.
    const uint64_t want = (most + 4 * kSampleThreads - 1) / (4 * kSampleThreads), share = (148 * 8 + ncands - 1) / ncands;
    plan_sample_kernel<<<dim3((unsigned)(want < share ? want : share), ncands), kSampleThreads, 0, st>>>(d, n1, n2, cands, qb, e,
                                                                                                        qb_range, hist);
    count_launch();
    return cudaGetLastError();
}

cudaError_t launch_plan_mse(const PlanCand *cands, uint32_t ncands, const float *e, float *mse, cudaStream_t st) {
    if (ncands == 0) return cudaSuccess;
    plan_mse_kernel<<<ncands, 1024, 0, st>>>(cands, e, mse);
    count_launch();
    return cudaGetLastError();
}

}  // namespace asz
