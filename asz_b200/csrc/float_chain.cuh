// A serial float sum of non-negative terms, evaluated bit for bit by many threads.
//
// The reference adds its error and entropy terms one after the other into one float. While that
// running sum s stays in one binade [2^E, 2^(E+1)), with ulp u = 2^(E-23) and s = m u (m an integer
// in [2^23, 2^24)), adding a term x gives (m + rint(x / u)) u: the nearest multiple of u, whatever
// m is, unless x / u lies half way between two integers (round-half-even then looks at m) or the
// sum leaves the binade. So a batch of terms needs no order: each thread rounds its own x / u, a
// scan gives the running sums, and the batch is accepted up to the first thread whose terms tie or
// leave the binade. That thread takes its terms one by one, and the rest of the batch follows in
// the new binade. A sum crosses each binade once, so there are about log2(sum / first term) such
// steps.
//
// The tie test keeps a margin of 2^-20: a term known to a relative 2^-52, or an addition that is
// rounded to double before it is rounded to float, moves x / u by less than 2^-27 (x / u < 2^24),
// so neither can bring it across a half from outside the margin. A term that is negative or not
// finite fails the test too and is added by itself.
#pragma once
#include <cstdint>

namespace asz {

// The running sum as an integer multiple of its ulp.
struct ChainSum {
    float s;
    uint32_t m;
    double inv_u;
    int ex;
    bool normal;  // far enough above the smallest floats for the products below
    __device__ __forceinline__ explicit ChainSum(float v) : s(v), m(0), inv_u(0.0), ex(0), normal(v >= 0x1p-100f && v < 0x1p120f) {
        if (normal) {
            ex = (int)(__float_as_uint(v) >> 23) - 126;  // v = f 2^ex, f in [1/2, 1): ulp 2^(ex - 24)
            m = (__float_as_uint(v) & 0x7fffffu) | 0x800000u;
            inv_u = __longlong_as_double((long long)(1023 + 24 - ex) << 52);
        }
    }
    // The sum after `add` more ulps (m + add < 2^24).
    __device__ __forceinline__ float after(uint32_t add) const {
        return add == 0 ? s : __uint_as_float(((uint32_t)(ex + 126) << 23) | ((m + add) & 0x7fffffu));
    }
    // Rounded ulps of one term, added to `ulps` (saturating well above 2^24); false if the term
    // has to be added by itself.
    __device__ __forceinline__ bool take(double x, uint32_t &ulps) const {
        if (!normal) return x == 0.0 && s >= 0.0f;
        const double t = __dmul_rn(x, inv_u);
        if (!(t >= 0.0 && t < 0x1p24)) return false;
        const double r = rint(t);
        const double half = fabs(__dsub_rn(t, r));  // exact
        ulps = min(ulps + (uint32_t)__double2uint_rn(r), 1u << 25);
        return half < 0.5 - 0x1p-20;
    }
};

// One warp: the chain over terms 0..n-1, `per` consecutive terms a lane. term(k) is term k in
// double, step(s, k) the reference's own addition. Every lane gets the sum.
template <int kPer, class Term, class Step>
__device__ float warp_chain(float s, int n, const Term &term, const Step &step) {
    const int lane = threadIdx.x & 31;
    for (int b = 0; b < n; b += 32 * kPer) {
        const int k0 = b + lane * kPer, k1 = min(k0 + kPer, n);
        double x[kPer];
#pragma unroll
        for (int i = 0; i < kPer; i++) x[i] = k0 + i < n ? term(k0 + i) : 0.0;
        int from = 0;  // lanes below are done
        while (true) {
            const ChainSum c(s);
            uint32_t ulps = 0;
            bool ok = true;
            if (lane >= from) {
#pragma unroll
                for (int i = 0; i < kPer; i++) ok = c.take(x[i], ulps) && ok;
            }
            ulps = min(ulps, 1u << 24);
            uint32_t incl = ulps;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += y;
            }
            ok = ok && (!c.normal || c.m + incl < (1u << 24));
            const unsigned bad = __ballot_sync(0xffffffffu, !ok);
            const int f = bad ? __ffs(bad) - 1 : 31;
            const float upto = c.normal ? c.after(__shfl_sync(0xffffffffu, bad ? incl - ulps : incl, f)) : s;
            if (!bad) {
                s = upto;
                break;
            }
            float v = upto;
            if (lane == f)
                for (int k = k0; k < k1; k++) v = step(v, k);
            s = __shfl_sync(0xffffffffu, v, f);
            from = f + 1;
            if (from == 32) break;
        }
    }
    return s;
}

// Scratch of block_chain, in shared memory.
struct ChainShared {
    uint32_t total[2][32], first[2][32];
    float s;
};

// A CTA of 1024 threads: as warp_chain, with a batch of 1024 kPer terms (load(k0, x) fetches the
// terms from k0 on, zero past the end). Two barriers a batch, three where a thread steps by itself.
template <int kPer, class Load, class Step>
__device__ float block_chain(ChainShared &sh, float s, uint64_t n, const Load &load, const Step &step) {
    constexpr uint32_t kT = 1024;
    const uint32_t tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    uint32_t parity = 0;
    float next[kPer];
    load((uint64_t)tid * kPer, next);
    for (uint64_t b = 0; b < n; b += (uint64_t)kT * kPer) {
        const uint64_t k0 = b + (uint64_t)tid * kPer;
        float x[kPer];
#pragma unroll
        for (int i = 0; i < kPer; i++) x[i] = next[i];
        load(k0 + (uint64_t)kT * kPer, next);  // in flight over this batch
        uint32_t from = 0;
        while (true) {
            const ChainSum c(s);
            uint32_t ulps = 0;
            bool ok = true;
            if (tid >= from) {
#pragma unroll
                for (int i = 0; i < kPer; i++) ok = c.take(__dmul_rn((double)x[i], (double)x[i]), ulps) && ok;
            }
            ulps = min(ulps, 1u << 24);
            uint32_t incl = ulps;
#pragma unroll
            for (uint32_t o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += y;
            }
            if (lane == 31) sh.total[parity][w] = min(incl, 1u << 24);
            __syncthreads();
            uint32_t wt = sh.total[parity][lane];  // running totals of the warps (32 of them)
#pragma unroll
            for (uint32_t o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(0xffffffffu, wt, o);
                if (lane >= o) wt += y;
            }
            const uint32_t all = __shfl_sync(0xffffffffu, wt, 31);
            const uint32_t before = w ? __shfl_sync(0xffffffffu, wt, w - 1) : 0u;
            ok = ok && (!c.normal || c.m + before + incl < (1u << 24));
            const unsigned bad = __ballot_sync(0xffffffffu, !ok);
            if (lane == 0) sh.first[parity][w] = bad ? w * 32 + (uint32_t)__ffs(bad) - 1 : kT;
            __syncthreads();
            const uint32_t f = __reduce_min_sync(0xffffffffu, sh.first[parity][lane]);
            parity ^= 1;
            if (f == kT) {
                if (c.normal) s = c.after(all);
                break;
            }
            if (tid == f) {
                float v = c.normal ? c.after(before + incl - ulps) : s;
#pragma unroll
                for (int i = 0; i < kPer; i++)
                    if (k0 + i < n) v = step(v, x[i]);
                sh.s = v;
            }
            __syncthreads();
            s = sh.s;
            from = f + 1;
            if (from == kT) break;
        }
    }
    return s;
}

}  // namespace asz
