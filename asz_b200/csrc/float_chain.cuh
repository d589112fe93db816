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
// steps. The subnormal floats and the first binade above them have one ulp and count as one binade
// (m from 0 on), so sums of terms of any size, also none but zeros, are taken this way. An infinite
// sum and one that is not a number stay what they are.
//
// Ties are common in the sums of a field of whole numbers or of few significant bits, once the sum's
// ulp is twice the squares' last place: most terms tie then. Where a batch had one, block_chain
// gives each thread's sum for an even and for an odd m, and scans the pairs, so that no tie ends a pass;
// warp_chain, whose batches are short, adds what is left of a batch term by term after kChainTies of
// them. The plan search of 100x500x500 bytes at 5e-2, with a pass for each thread that had a tie, took
// 62 ms, now 4.1; of values of 1e-25, with every term rejected while the sum was below 2^-100, 220, now 7.
//
// The tie test of warp_chain keeps a margin of 2^-20: a term known to a relative 2^-52, or an addition
// that is rounded to double before it is rounded to float, moves x / u by less than 2^-27
// (x / u < 2^24), so neither can bring it across a half from outside the margin. block_chain's terms
// are squares, exact in double, and its step rounds once: its ties are exact. A term that is negative
// or not finite fails the test too and is added by itself.
#pragma once
#include <cstdint>

namespace asz {

// The running sum as an integer multiple of its ulp.
struct ChainSum {
    float s;
    uint32_t m;
    double inv_u;
    bool regular;  // finite and not negative
    __device__ __forceinline__ explicit ChainSum(float v) : s(v), m(0), inv_u(0.0), regular(v >= 0.0f && v <= 0x1.fffffep127f) {
        if (regular) {
            const uint32_t bits = __float_as_uint(v) & 0x7fffffffu, e = max(bits >> 23, 1u);
            m = bits - ((e - 1) << 23);  // v = m 2^(e - 150)
            inv_u = __longlong_as_double((long long)(1023 + 150 - (int)e) << 52);
        }
    }
    // The sum after `add` more ulps (m + add < 2^24): the floats of a binade are consecutive integers.
    __device__ __forceinline__ float after(uint32_t add) const { return add == 0 ? s : __uint_as_float(__float_as_uint(s) + add); }
    // A sum that no term of this kind changes.
    __device__ __forceinline__ bool absorbs(double x) const { return s != s || (s > 0.0f && !regular && x >= 0.0); }
    // Rounded ulps of one term; false if the term has to be added by itself.
    __device__ __forceinline__ bool ulps(double x, uint32_t &r) const {
        r = 0;
        if (!regular) return absorbs(x);
        const double t = __dmul_rn(x, inv_u);
        if (!(t >= 0.0 && t < 0x1p24)) return false;
        const double w = rint(t);
        r = (uint32_t)__double2uint_rn(w);
        return fabs(__dsub_rn(t, w)) < 0.5 - 0x1p-20;  // the difference is exact
    }
    // Adds one exactly known term's ulps to the sums from an even (even) and from an odd m.
    __device__ __forceinline__ bool ulps2(double x, uint32_t &even, uint32_t &odd) const {
        if (!regular) return absorbs(x);
        const double t = __dmul_rn(x, inv_u);
        if (!(t >= 0.0 && t < 0x1p24)) return false;
        const double w = rint(t);
        const uint32_t r = (uint32_t)__double2uint_rn(w);
        if (fabs(__dsub_rn(t, w)) == 0.5) {  // to the even one of the two sums around it
            const uint32_t low = r - (w > t);
            even += low + ((even + low) & 1u);
            odd += low + ((odd + low + 1u) & 1u);
        } else {
            even += r;
            odd += r;
        }
        return true;
    }
};

// Terms of warp_chain lie in its batches' order: four consecutive ones a lane, without bank
// conflicts.
constexpr int kChainPer = 4, kChainBatch = 32 * kChainPer, kChainHead = 12, kChainTies = 8;
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
        for (int steps = 0;; steps++) {
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
                if (!ok[i] || (c.regular && c.m + acc + r[i] >= (1u << 24))) at = i;
                else acc += r[i];
            }
            const unsigned bad = __ballot_sync(0xffffffffu, at != kChainPer);
            const int f = bad ? __ffs(bad) - 1 : 31;
            s = c.after(__shfl_sync(0xffffffffu, acc, f));
            if (!bad) break;
            const int k = f * kChainPer + __shfl_sync(0xffffffffu, at, f);
            s = step(s, b + k);  // the same on every lane
            done = k + 1;
            if (steps == kChainTies)
                for (; done < kChainBatch && b + done < n; done++) s = step(s, b + done);
            if (done == kChainBatch || b + done >= n) break;
        }
    }
    return s;
}

// Increments of m over some terms, from an even and from an odd m.
struct ChainInc {
    uint32_t even, odd;
    __device__ __forceinline__ uint32_t from(uint32_t m) const { return m & 1u ? odd : even; }
    // These terms, then those of b. Sums above 2^24 need not be right, only above 2^24.
    __device__ __forceinline__ ChainInc then(const ChainInc &b) const {
        return ChainInc{even + b.from(even), odd + b.from(odd + 1u)};
    }
};

// Scratch of block_chain, in shared memory.
struct ChainShared {
    ChainInc total[2][32];
    uint32_t first[2][32];
    float s;
};

template <bool kTies>
struct ChainTies {
    static constexpr bool value = kTies;
};

// Inclusive scan over the warp; without ties the two increments are one.
template <bool kTies>
__device__ __forceinline__ ChainInc chain_scan(ChainInc v) {
    const uint32_t lane = threadIdx.x & 31;
#pragma unroll
    for (uint32_t o = 1; o < 32; o <<= 1) {
        const uint32_t e = __shfl_up_sync(0xffffffffu, v.even, o);
        if (kTies) {
            const uint32_t d = __shfl_up_sync(0xffffffffu, v.odd, o);
            if (lane >= o) v = ChainInc{e, d}.then(v);
        } else if (lane >= o) {
            v.even += e;
        }
    }
    return v;
}

// A CTA of 1024 threads: as warp_chain, with a batch of 1024 kPer terms, squares of x (load(k0, x) fetches
// the values from k0 on, zero past the end; step is exact but for one rounding). Two barriers a pass,
// three where a thread steps by itself. A batch's first pass stops at a tie, the others take ties as well.
template <int kPer, class Load, class Step>
__device__ float block_chain(ChainShared &sh, float s, uint64_t n, const Load &load, const Step &step) {
    constexpr uint32_t kT = 1024, kFull = 1u << 24;
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
        auto pass = [&](auto kTies) {  // true: the batch is done
            constexpr bool kWithTies = decltype(kTies)::value;
            const ChainSum c(s);
            ChainInc mine{0, 0};
            bool ok = true;
            if (tid >= from) {
#pragma unroll
                for (int i = 0; i < kPer; i++) {
                    const double t = __dmul_rn((double)x[i], (double)x[i]);
                    if (kWithTies) {
                        ok = c.ulps2(t, mine.even, mine.odd) && ok;
                    } else {
                        uint32_t r;
                        ok = c.ulps(t, r) && ok;
                        mine.even += r;
                    }
                }
            }
            auto cap = [&](ChainInc v) { return ChainInc{min(v.even, kFull), min(v.odd, kFull)}; };
            const ChainInc incl = chain_scan<kWithTies>(cap(mine));
            if (lane == 31) sh.total[parity][w] = cap(incl);
            __syncthreads();
            const ChainInc wt = chain_scan<kWithTies>(sh.total[parity][lane]);  // of the warps (32 of them)
            // The sum before this thread's warp, before this thread and after it, and after all.
            const uint32_t run = kWithTies ? wt.from(c.m) : wt.even;
            const uint32_t all = __shfl_sync(0xffffffffu, run, 31), warps = __shfl_sync(0xffffffffu, run, (int)w - 1);
            const uint32_t before_warp = w ? warps : 0u;
            const uint32_t in_warp = kWithTies ? incl.from(c.m + before_warp) : incl.even;
            const uint32_t lanes = __shfl_up_sync(0xffffffffu, in_warp, 1);
            const uint32_t before = before_warp + (lane ? lanes : 0u);
            ok = ok && (!c.regular || c.m + before_warp + in_warp < kFull);
            const unsigned bad = __ballot_sync(0xffffffffu, !ok);
            if (lane == 0) sh.first[parity][w] = bad ? w * 32 + (uint32_t)__ffs(bad) - 1 : kT;
            __syncthreads();
            const uint32_t f = __reduce_min_sync(0xffffffffu, sh.first[parity][lane]);
            parity ^= 1;
            if (f == kT) {
                s = c.after(all);
                return true;
            }
            if (tid == f) {
                float v = c.after(before);
#pragma unroll
                for (int i = 0; i < kPer; i++)
                    if (k0 + i < n) v = step(v, x[i]);
                sh.s = v;
            }
            __syncthreads();
            s = sh.s;
            from = f + 1;
            return from == kT;
        };
        if (pass(ChainTies<false>())) continue;
        while (!pass(ChainTies<true>())) {}
    }
    return s;
}

}  // namespace asz
