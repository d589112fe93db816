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
    int ex;
    double inv_u;
    bool normal;  // well inside the normal floats
    __device__ __forceinline__ explicit ChainSum(float v) : s(v), m(0), ex(0), inv_u(0.0), normal(v >= 0x1p-100f && v < 0x1p120f) {
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
    // Rounded ulps of one term; false if the term has to be added by itself.
    __device__ __forceinline__ bool ulps(double x, uint32_t &r) const {
        r = 0;
        if (!normal) return x == 0.0 && s >= 0.0f;
        const double t = __dmul_rn(x, inv_u);
        if (!(t >= 0.0 && t < 0x1p24)) return false;
        const double w = rint(t);
        r = (uint32_t)__double2uint_rn(w);
        return fabs(__dsub_rn(t, w)) < 0.5 - 0x1p-20;  // the difference is exact
    }
};

// Terms of warp_chain lie in its batches' order: four consecutive ones a lane, without bank
// conflicts.
constexpr int kChainPer = 4, kChainBatch = 32 * kChainPer, kChainHead = 12;
__device__ __forceinline__ int chain_slot(int k) {
    return (k & ~(kChainBatch - 1)) + (k & (kChainPer - 1)) * 32 + ((k & (kChainBatch - 1)) / kChainPer);
}
__host__ __device__ constexpr uint32_t chain_slots(uint32_t n) {
    return (n + kChainBatch - 1) / kChainBatch * kChainBatch;
}

// One warp: the chain over n terms, term k at x[chain_slot(k)]. step(s, k) is the reference's own
// addition. Every lane gets the sum. A pass takes what is left of the batch up to the first term
// that leaves the binade or ties, and that term.
template <class Step>
__device__ __forceinline__ float warp_chain(const double *x, int n, const Step &step) {
    const int lane = threadIdx.x & 31;
    float s = 0.0f;
    // The sum leaves its binade at every other of the first terms: those are added as they are.
    const int head = min(n, kChainHead);
    for (int k = 0; k < head; k++) s = step(s, k);
    for (int b = 0; b < n; b += kChainBatch) {
        double v[kChainPer];
#pragma unroll
        for (int i = 0; i < kChainPer; i++) v[i] = b + lane * kChainPer + i < n ? x[b + i * 32 + lane] : 0.0;
        int done = b == 0 ? head : 0;  // terms of the batch already added
        while (true) {
            const ChainSum c(s);
            uint32_t r[kChainPer], sum = 0;
            bool ok[kChainPer];
#pragma unroll
            for (int i = 0; i < kChainPer; i++) {
                ok[i] = c.ulps(v[i], r[i]);
                // What is added already, and places past the last term, which a sum that is not a
                // number would reject.
                if (lane * kChainPer + i < done || b + lane * kChainPer + i >= n) ok[i] = true, r[i] = 0;
                sum += r[i];  // r <= 2^24
            }
            uint32_t incl = sum;  // <= 32 * 2^26
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += y;
            }
            // Within the lane: the first term that cannot be taken, and the sum before it.
            uint32_t acc = incl - sum;
            int at = kChainPer;
#pragma unroll
            for (int i = 0; i < kChainPer; i++) {
                if (at != kChainPer) continue;
                if (!ok[i] || (c.normal && c.m + acc + r[i] >= (1u << 24))) at = i;
                else acc += r[i];
            }
            const unsigned bad = __ballot_sync(0xffffffffu, at != kChainPer);
            const int f = bad ? __ffs(bad) - 1 : 31;
            s = c.after(__shfl_sync(0xffffffffu, acc, f));
            if (!bad) break;
            const int k = f * kChainPer + __shfl_sync(0xffffffffu, at, f);
            s = step(s, b + k);  // the same on every lane
            done = k + 1;
            if (b + done >= n) break;
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
                for (int i = 0; i < kPer; i++) {
                    uint32_t r;
                    ok = c.ulps(__dmul_rn((double)x[i], (double)x[i]), r) && ok;
                    ulps += r;
                }
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
                s = c.after(all);
                break;
            }
            if (tid == f) {
                float v = c.after(before + incl - ulps);
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
