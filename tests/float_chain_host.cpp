// float_chain.cuh on the host: a fiber per CUDA thread, switched at every warp or CTA collective, so
// that the device functions themselves run, one thread at a time, with what they read counted.
#include <ucontext.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstring>
#include <functional>
#include <memory>
#include <vector>

#define __device__
#define __host__
#define __forceinline__ inline
using std::fabs;
using std::max;
using std::min;
using std::rint;

static struct {
    unsigned x;
} threadIdx;

namespace emu {
struct Meeting {  // values of `size` threads, twice: nobody overwrites what another still reads
    uint64_t v[2][1024];
    uint64_t arrived = 0;
};
static std::vector<ucontext_t> fibers;
static std::vector<uint64_t> epochs[2];  // of a thread: warp collectives, barriers
static std::vector<Meeting> warps;
static Meeting cta;
static ucontext_t home;
static unsigned current, live;
static std::vector<char> done;
static uint64_t barriers;
static std::function<void()> body;

static void next_fiber() {
    const unsigned from = current;
    for (unsigned k = 1; k <= fibers.size(); k++) {
        const unsigned to = (from + k) % fibers.size();
        if (done[to]) continue;
        if (to == from) return;
        current = threadIdx.x = to;
        swapcontext(&fibers[from], &fibers[to]);
        return;
    }
}
static const uint64_t *meet(Meeting &m, unsigned kind, unsigned slot, unsigned size, uint64_t v) {
    const uint64_t e = epochs[kind][threadIdx.x]++;
    m.v[e & 1][slot] = v;
    m.arrived++;
    while (m.arrived < size * (e + 1)) next_fiber();
    return m.v[e & 1];
}
static const uint64_t *warp_meet(uint64_t v) { return meet(warps[threadIdx.x / 32], 0, threadIdx.x % 32, 32, v); }
static const uint64_t *cta_meet(uint64_t v) {
    if (threadIdx.x == 0) barriers++;
    return meet(cta, 1, threadIdx.x, (unsigned)fibers.size(), v);
}
static void entry() {
    body();
    done[current] = 1;
    if (--live == 0) setcontext(&home);
    const unsigned from = current;
    for (unsigned k = 1;; k++) {
        const unsigned to = (from + k) % fibers.size();
        if (done[to]) continue;
        current = threadIdx.x = to;
        setcontext(&fibers[to]);
    }
}
static void run(unsigned threads, std::function<void()> f) {
    constexpr size_t kStack = 64 << 10;
    body = std::move(f);
    fibers.assign(threads, ucontext_t{});
    epochs[0].assign(threads, 0);
    epochs[1].assign(threads, 0);
    warps.assign(threads / 32, Meeting{});
    cta.arrived = barriers = 0;
    done.assign(threads, 0);
    live = threads;
    std::unique_ptr<char[]> stacks(new char[kStack * threads]);
    for (unsigned t = 0; t < threads; t++) {
        getcontext(&fibers[t]);
        fibers[t].uc_stack.ss_sp = stacks.get() + kStack * t;
        fibers[t].uc_stack.ss_size = kStack;
        makecontext(&fibers[t], entry, 0);
    }
    current = threadIdx.x = 0;
    swapcontext(&home, &fibers[0]);
}
}  // namespace emu

static uint32_t __float_as_uint(float v) {
    uint32_t u;
    std::memcpy(&u, &v, 4);
    return u;
}
static float __uint_as_float(uint32_t u) {
    float v;
    std::memcpy(&v, &u, 4);
    return v;
}
static double __longlong_as_double(long long u) {
    double v;
    std::memcpy(&v, &u, 8);
    return v;
}
static double __dmul_rn(double a, double b) { return a * b; }
static double __dsub_rn(double a, double b) { return a - b; }
static uint32_t __double2uint_rn(double v) { return (uint32_t)rint(v); }
static int __ffs(unsigned v) { return __builtin_ffs((int)v); }
template <class T>
static T __shfl_sync(unsigned, T v, int lane) {
    return (T)emu::warp_meet((uint64_t)v)[lane & 31];
}
template <class T>
static T __shfl_up_sync(unsigned, T v, unsigned o) {
    const unsigned lane = threadIdx.x % 32;
    const uint64_t *all = emu::warp_meet((uint64_t)v);
    return lane >= o ? (T)all[lane - o] : v;
}
static unsigned __ballot_sync(unsigned, bool p) {
    const uint64_t *all = emu::warp_meet(p);
    unsigned r = 0;
    for (int l = 0; l < 32; l++) r |= (unsigned)all[l] << l;
    return r;
}
static uint32_t __reduce_min_sync(unsigned, uint32_t v) {
    const uint64_t *all = emu::warp_meet(v);
    return (uint32_t)*std::min_element(all, all + 32);
}
static void __syncthreads() { emu::cta_meet(0); }

#include "../asz_b200/csrc/float_chain.cuh"

// The error chains: s = (float)fma(cnt, d d, s) in double (warp), s = fmaf(d, d, s) (CTA).
extern "C" float serial_weighted(const float *d, const int *cnt, int n) {
    volatile float s = 0.0f;
    for (int k = 0; k < n; k++) s = (float)std::fma((double)cnt[k], (double)d[k] * d[k], (double)s);
    return s;
}
extern "C" float serial_square(const float *d, int n) {
    volatile float s = 0.0f;
    for (int k = 0; k < n; k++) s = std::fma(d[k], d[k], (float)s);
    return s;
}
// last: the largest index that the warp's steps were given; steps: how many they were.
extern "C" float warp_weighted(const float *d, const int *cnt, int n, int *last, int *steps) {
    std::vector<double> x(asz::chain_slots((uint32_t)n), NAN);
    for (int k = 0; k < n; k++) x[asz::chain_slot(k)] = (double)cnt[k] * ((double)d[k] * d[k]);
    float out = 0.0f;
    *last = *steps = 0;
    emu::run(32, [&] {
        const float s = asz::warp_chain(x.data(), n, [&](float v, int k) {
            if (threadIdx.x == 0) *last = max(*last, k), ++*steps;
            if (k >= n) return v;
            return (float)std::fma((double)cnt[k], (double)d[k] * d[k], (double)v);
        });
        if (threadIdx.x == 0) out = s;
    });
    return out;
}
extern "C" float block_square(const float *d, int n, int *barriers) {
    static asz::ChainShared sh;
    float out = 0.0f;
    emu::run(1024, [&] {
        const float s = asz::block_chain<8>(
            sh, 0.0f, (uint64_t)n, [&](uint64_t k, float(&x)[8]) { for (int i = 0; i < 8; i++) x[i] = k + i < (uint64_t)n ? d[k + i] : 0.0f; },
            [](float v, float x) { return std::fma(x, x, v); });
        if (threadIdx.x == 0) out = s;
    });
    *barriers = (int)emu::barriers;
    return out;
}
