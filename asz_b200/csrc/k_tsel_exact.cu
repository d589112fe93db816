// Exact per-(block, round) coefficient selection for the groups the fast path could not settle,
// and the default-slope proxies (c_codes/asz_core/compress.tpp:91-144, get_AB_map.tpp:7-24,
// get_h_psnr.tpp:6-31, get_default_slope.tpp:15-39).
//
// One CTA per group, all state in shared memory:
//  1. sample keys in get_AB_map's scan order;
//  2. de-duplicate them (shared hash table) and compact the distinct keys in first-occurrence order;
//  3. rebuild std::unordered_map's iteration order without replaying insertions one by one. Within
//     one rehash stage the list is a sequence of bucket runs: runs ordered by the time their bucket
//     was first filled (newest first), nodes within a run newest first. A node's "time" in a stage
//     is its position in the previous stage's list if it was present at the rehash, else its
//     insertion index. So each stage is a parallel rank computation (atomics, one scan);
//  4. per evaluation: quantised errors in map order, the qb_map's own order (same method, identity
//     hash), then the two order-dependent float sums.
// The result is the reference's float h1 and log10f argument bit for bit; the t decision then
// uses the same certified log10 step as the serial kernel.
//
// A launch has a few groups (tens in a round, three boxes for the default slope), so what counts is
// how long one group takes, and that is a chain of short dependent steps, not work. Hence:
// - the CTA splits into up to five teams of warps, an evaluation each, so a group takes as long as
//   one evaluation and not as five (as many teams as the shared memory holds the tables of);
// - tables are sized by the group and not by the largest group;
// - a rehash stage has the threads it needs: a warp up to 31 nodes, four (or the team's three) up to
//   127, and then a node a thread in registers;
// - the serial float sums go to a warp each (float_chain.cuh) instead of a thread, a step of which
//   takes a double fused add and two conversions in a row.
// Default slope of a 512^3 field (three boxes, ten evaluations): 84 -> 39 us; the nine rounds' groups
// of a 161x257x349 quintic field at 1e-4: 1.13 -> 0.52 ms; the plan search's AB maps at 100x500x500:
// 3.2 -> 0.79 ms. What is left of one group is spread over all phases (363 samples: sampling 4 us,
// map order 6, evaluation maps 6, sums 7), each a few dozen dependent shared-memory round trips.
#include <cuda_runtime.h>

#include "dev_common.cuh"
#include "float_chain.cuh"
#include "launch.h"
#include "listsim.cuh"
#include "tsel.cuh"

namespace asz {
namespace {

constexpr int kThreads = 512;
constexpr int kTeams = 5;      // evaluations side by side, where their tables fit
constexpr int kMaxEvals = 22;  // default slope: 11 t values x 2 error bounds

__device__ __forceinline__ int class_of(uint64_t b, uint64_t nb) { return b == 0 ? 0 : (b == nb - 1 ? 2 : 1); }

__device__ __forceinline__ uint64_t mix64(uint64_t x) {
    x ^= x >> 33;
    x *= 0xff51afd7ed558ccdull;
    x ^= x >> 33;
    x *= 0xc4ceb9fe1a85ec53ull;
    x ^= x >> 33;
    return x;
}

// A set of whole warps that synchronise on their own hardware barrier (bar 0 is the CTA's). A team
// of one warp needs none.
struct Team {
    int tid, size, bar;
    __device__ __forceinline__ void sync() const {
        if (size == 32) __syncwarp();
        else asm volatile("bar.sync %0, %1;" ::"r"(bar), "r"(size) : "memory");
    }
};

__device__ __forceinline__ int warp_incl_scan(int v) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o) v += y;
    }
    return v;
}

// Exclusive scan of one value per team thread; total in *tot. warp_sums holds 32 ints.
__device__ int team_excl_scan(const Team &T, int v, int *warp_sums, int *tot) {
    const int lane = T.tid & 31, w = T.tid >> 5, nw = T.size >> 5;
    const int x = warp_incl_scan(v);
    if (nw == 1) {
        if (tot) *tot = __shfl_sync(0xffffffffu, x, 31);
        return x - v;
    }
    if (lane == 31) warp_sums[w] = x;
    T.sync();
    const int s = warp_incl_scan(lane < nw ? warp_sums[lane] : 0);  // every warp, so no second barrier
    const int base = w ? __shfl_sync(0xffffffffu, s, w - 1) : 0, total = __shfl_sync(0xffffffffu, s, nw - 1);
    T.sync();
    if (tot) *tot = total;
    return base + x - v;
}

// Exclusive scan of a[0..n) in place; returns the total.
__device__ int team_scan_array(const Team &T, int *a, int n, int *warp_sums) {
    const int per = (n + T.size - 1) / T.size;
    const int beg = T.tid * per, end = min(beg + per, n);
    int local = 0;
    for (int i = beg; i < end; i++) local += a[i];
    int tot;
    int off = team_excl_scan(T, local, warp_sums, &tot);
    for (int i = beg; i < end; i++) {
        int v = a[i];
        a[i] = off;
        off += v;
    }
    T.sync();
    return tot;
}

// Working arrays of one map's order: heads (one int a bucket), next, after, first, rank, moved (one a
// node).
struct OrderScratch {
    int *heads, *next, *after, *first, *rank, *moved;
};

// h mod the stage's bucket count: the quotient by the reciprocal is at most two short.
__device__ __forceinline__ int bucket_of(uint64_t h, uint32_t beta, uint64_t magic) {
    uint64_t r = h - __umul64hi(h, magic) * beta;
    if (r >= beta) r -= beta;
    if (r >= beta) r -= beta;
    return (int)r;
}

// A bucket's chain from `head`, as times of its nodes in no order: the first of them, how many they
// are, and how many are later than t.
__device__ __forceinline__ void walk(const int *next, int head, int t, int limit, int &first, int &count, int &later) {
    first = t;
    count = later = 0;
    for (int x = head; x >= 0 && count < limit; x = next[x]) {
        first = min(first, x);
        count++;
        later += x > t;
    }
}

// One rehash stage over nodes [0, end): ord[] is the list before it for the first `fresh` nodes (the
// others come in the order of their index) and the list after it at the end. A node's time is its
// place in that sequence, thread or iteration t has the node of time t, and its new place is the
// number of nodes in runs opened after its own plus those of its run that are later than it.
__device__ __forceinline__ void map_stage(const Team T, int stage, int end, int fresh, const uint64_t *hash, const OrderScratch S,
                                       int *ord, int *warp_sums) {
    const uint32_t beta = (uint32_t)sched_bkt(stage);
    const uint64_t magic = sched_magic(stage);
    const int lane = T.tid & 31, w = T.tid >> 5, nw = T.size >> 5;
    for (uint32_t b = T.tid; b < beta; b += T.size) S.heads[b] = -1;
    if (end <= T.size) {  // a node a thread, in registers
        const int t = T.tid;
        const bool in = t < end;
        const int e = t < fresh ? ord[t] : t;
        const int b = in ? bucket_of(hash[e], beta, magic) : 0;
        T.sync();
        if (in) S.next[t] = atomicExch(&S.heads[b], t);
        T.sync();
        int first = t, count = 0, later = 0;
        if (in) walk(S.next, S.heads[b], t, end, first, count, later);
        const int opened = first == t ? count : 0;  // the run's nodes, at the time it was opened
        int sum = opened;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_down_sync(0xffffffffu, sum, o);
            if (lane + o < 32) sum += y;
        }
        int behind = 0;
        if (nw > 1) {
            if (lane == 0) warp_sums[w] = sum;
            T.sync();
            behind = __reduce_add_sync(0xffffffffu, lane > w && lane < nw ? warp_sums[lane] : 0);
        }
        if (in && opened) S.after[t] = behind + sum - opened;
        T.sync();
        if (in) ord[S.after[first] + later] = e;
        T.sync();
        return;
    }
    T.sync();
    for (int t = T.tid; t < end; t += T.size) {
        const int e = t < fresh ? ord[t] : t;
        const int b = bucket_of(hash[e], beta, magic);
        S.moved[t] = e;
        S.rank[t] = b;
        S.next[t] = atomicExch(&S.heads[b], t);
    }
    T.sync();
    for (int t = T.tid; t < end; t += T.size) {
        int first, count, later;
        walk(S.next, S.heads[S.rank[t]], t, end, first, count, later);
        S.first[t] = first;
        S.rank[t] = later;
        S.after[end - 1 - t] = first == t ? count : 0;
    }
    T.sync();
    team_scan_array(T, S.after, end, warp_sums);
    for (int t = T.tid; t < end; t += T.size) ord[S.after[end - 1 - S.first[t]] + S.rank[t]] = S.moved[t];
    T.sync();
}

// Iteration order of a std::unordered_map filled by inserting distinct elements 0..m-1 (m >= 1) with
// the given hashes in order (stage method, see the file comment). Writes ord[m]. The stages of up to
// 31 nodes are the team's first warp's, those of up to 127 the first `few` threads', which
// synchronise on barrier `few_bar` (few == the team's size: on the team's).
__device__ __forceinline__ void map_order(const Team &T, int few, int few_bar, int m, const uint64_t *hash, const OrderScratch &S, int *ord,
                          int *warp_sums) {
    int had = 32;  // threads that have the list
    for (int stage = 0; stage < kSchedLen && sched_at(stage) <= (uint64_t)m; stage++) {
        const int fresh = stage == 0 ? 0 : (int)sched_at(stage) - 1;
        const int end = (stage + 1 < kSchedLen && sched_at(stage + 1) <= (uint64_t)m) ? (int)sched_at(stage + 1) - 1 : m;
        const Team U{T.tid, end < 32 ? 32 : end < 128 ? few : T.size, end < 128 ? few_bar : T.bar};
        if (T.tid >= U.size) continue;
        if (U.size != had) U.sync();
        had = U.size;
        map_stage(U, stage, end, fresh, hash, S, ord, warp_sums);
    }
    if (had != T.size) T.sync();
}

struct ExactGroup {
    SampleBox box;
    uint32_t n;
};

// Layout of the working set of a group of up to n samples with `teams` evaluations side by side
// (offsets in bytes), made on the host. The distinct entries and the AB map's order persist;
// sampling and de-duplication, the AB map's stages and the teams' tables follow one another in one
// region. In a team's slice, beside its distinct values, their counts and their order, one area
// holds its hash table, then its map's stages, then the terms of its sums.
struct Layout {
    uint32_t n, teams;
    uint32_t ekey, ecnt, ord;                 // persistent
    uint32_t key, tkey, tfirst, tcnt, sslot;  // phases 1-2
    uint32_t hash, order;                     // phase 3
    uint32_t team, team_stride;               // phase 4
    uint32_t qval, qc, qord, work;            // in a team's slice
    uint32_t qtab, qfirst, qsum, qslot;       // in its work area
    uint32_t total;
    __host__ Layout(uint32_t n_, uint32_t teams_) : n(n_), teams(teams_) {
        const uint32_t hcap = hash_slots(n);
        uint32_t off = 0, top = 0;
        auto take = [&](uint32_t bytes) {
            const uint32_t o = off;
            off += (bytes + 15) & ~15u;
            top = off > top ? off : top;
            return o;
        };
        ekey = take(8 * n);
        ecnt = take(4 * n);
        ord = take(4 * n);
        const uint32_t u = off;
        key = take(8 * n);
        tkey = take(8 * hcap);
        tfirst = take(4 * hcap);
        tcnt = take(4 * hcap);
        sslot = take(4 * n);
        off = u;
        hash = take(8 * n);
        order = take(order_bytes(n));
        off = 0;
        uint32_t own = top;
        top = 0;
        qval = take(8 * n);
        qc = take(4 * n);
        qord = take(4 * n);
        work = take(order_bytes(n));
        off = work;
        take(16 * chain_slots(n) + 12 * n);
        off = work;
        qtab = take(4 * hcap);
        qfirst = take(4 * hcap);
        qsum = take(4 * hcap);
        qslot = take(4 * n);
        team = u;
        team_stride = top;
        total = u + teams * team_stride > own ? u + teams * team_stride : own;
    }
    __host__ __device__ static uint32_t hash_slots(uint32_t n) { return n + n / 2 + 16; }
    __host__ static uint32_t order_bytes(uint32_t n) {
        return 4 * (5 * ((n + 3) & ~3u) + (uint32_t)sched_buckets(n));
    }
    __device__ OrderScratch order_at(uint8_t *p) const {
        const uint32_t an = (n + 3) & ~3u;
        int *q = (int *)p;
        return OrderScratch{q + 5 * an, q, q + an, q + 2 * an, q + 3 * an, q + 4 * an};
    }
};

// The layout of a launch whose groups have up to n samples, in `bytes` of memory: five teams of
// three warps, two of eight, or the whole CTA. The last fits where exact_smem_bytes(n) does.
Layout exact_layout(uint32_t n, uint64_t bytes) {
    if (n < kExactFullMost)
        for (uint32_t teams : {(uint32_t)kTeams, 2u}) {
            const Layout l(n, teams);
            if (l.total <= bytes) return l;
        }
    return Layout(n, 1);
}

// Quantised error of an entry for one evaluation (get_h_psnr.tpp:14-19 as emitted).
__device__ __forceinline__ void entry_err(uint64_t kk, float t2, float stat_eb, float neg, float eb2, int &q, float &d) {
    float af = __ll2float_rn((int64_t)(int32_t)(uint32_t)(kk >> 32)), bf = __ll2float_rn((int64_t)(int32_t)(uint32_t)kk);
    float err = __fmul_rn(__fmaf_rn(bf, 2.0f, __fmul_rn(af, t2)), stat_eb);
    int64_t q64 = lround_f(__fmul_rn(err, neg));
    q = (int)q64;
    d = __fmaf_rn(-__ll2float_rn(q64), eb2, err);
}

__device__ __forceinline__ uint32_t hash_slot(uint64_t k, uint32_t cap) { return __umulhi((uint32_t)(mix64(k) >> 32), cap); }

// Evaluations of one group: h1 and the log10f argument for each (t, abs_eb), in the working set at
// `mem`. Returns false if the group is larger than the layout or has keys outside int32.
__device__ bool exact_eval(const ExactGroup &eg, const float *__restrict__ ref, const float *__restrict__ x0, uint64_t n1n2,
                           uint64_t n2, const ProxyEval *evals, int n_evals, float R2, const float *__restrict__ log2tab,
                           uint8_t *mem, const Layout &Lo, float *h1_out, float *x_out, uint32_t *m_out) {
    const uint32_t n = eg.n, hcap = Layout::hash_slots(n);
    if (n > Lo.n || blockDim.x != (unsigned)kThreads) return false;
    const int teams = (int)Lo.teams;
    __shared__ int warp_sums[kTeams][32], all_sums[32];
    __shared__ int flag_wide;
    const Team all{(int)threadIdx.x, (int)blockDim.x, 0};
    uint64_t *key = (uint64_t *)(mem + Lo.key), *tkey = (uint64_t *)(mem + Lo.tkey), *ekey = (uint64_t *)(mem + Lo.ekey);
    int *tfirst = (int *)(mem + Lo.tfirst), *tcnt = (int *)(mem + Lo.tcnt), *sslot = (int *)(mem + Lo.sslot);
    int *ecnt = (int *)(mem + Lo.ecnt), *ord = (int *)(mem + Lo.ord);
    if (threadIdx.x == 0) flag_wide = 0;
    const uint64_t EMPTY = 0x8000000000000000ull;  // a = INT32_MIN: rejected below, so never a key
    for (uint32_t i = threadIdx.x; i < hcap; i += blockDim.x) {
        tkey[i] = EMPTY;
        tfirst[i] = INT32_MAX;
        tcnt[i] = 0;
    }
    all.sync();
    // 1. Sample keys in get_AB_map's scan order, into the hash table: first occurrence and count
    // per distinct key.
    const SampleBox &b = eg.box;
    uint32_t c[3];
    for (int a = 0; a < 3; a++) c[a] = b.hi[a] > b.lo[a] ? (uint32_t)((b.hi[a] - b.lo[a] + b.step[a] - 1) / b.step[a]) : 0;
    for (uint32_t s = threadIdx.x; s < n; s += blockDim.x) {
        uint32_t k2 = s % c[2], k1 = (s / c[2]) % c[1], k0 = s / (c[1] * c[2]);
        uint64_t p = (b.lo[0] + k0 * b.step[0]) * n1n2 + (b.lo[1] + k1 * b.step[1]) * n2 + (b.lo[2] + k2 * b.step[2]);
        const uint64_t d = b.dist;
        float m1 = ref[p - d], m3 = ref[p - 3 * d], p1 = ref[p + d], p3 = ref[p + 3 * d];
        float Af = __fsub_rn(__fadd_rn(m1, p1), __fadd_rn(m3, p3));
        float S4 = __fadd_rn(__fadd_rn(p1, p3), __fadd_rn(m1, m3));
        float Bf = __double2float_rn(__fma_rn((double)S4, 0.25, -(double)x0[p]));
        int64_t ak = lround_f(__fmul_rn(Af, b.neg_2_stat_eb)), bk = lround_f(__fmul_rn(Bf, b.neg_2_stat_eb));
        if (ak <= INT32_MIN || ak > INT32_MAX || bk < INT32_MIN || bk > INT32_MAX) {
            flag_wide = 1;
            sslot[s] = 0;
            continue;
        }
        const uint64_t k = ((uint64_t)(uint32_t)(int32_t)ak << 32) | (uint32_t)(int32_t)bk;
        key[s] = k;
        uint32_t slot = hash_slot(k, hcap);
        for (uint32_t probe = 0; probe < hcap; probe++) {
            unsigned long long prev = atomicCAS((unsigned long long *)&tkey[slot], (unsigned long long)EMPTY, (unsigned long long)k);
            if (prev == EMPTY || prev == k) break;
            if (++slot == hcap) slot = 0;
        }
        sslot[s] = (int)slot;
        atomicMin(&tfirst[slot], (int)s);
        atomicAdd(&tcnt[slot], 1);
    }
    all.sync();
    if (flag_wide) return false;
    // 2. Distinct keys in first-occurrence order.
    int m;
    {
        const uint32_t per = (n + blockDim.x - 1) / blockDim.x, beg = threadIdx.x * per, end = min(beg + per, n);
        int local = 0;
        for (uint32_t s = beg; s < end; s++) local += tfirst[sslot[s]] == (int)s;
        int off = team_excl_scan(all, local, all_sums, &m);
        for (uint32_t s = beg; s < end; s++)
            if (tfirst[sslot[s]] == (int)s) {
                ekey[off] = key[s];
                ecnt[off] = tcnt[sslot[s]];
                off++;
            }
    }
    all.sync();
    // hash = a*1145141919810 + b (asz_param.hpp:22-40); its array lies over the hash table
    uint64_t *hash = (uint64_t *)(mem + Lo.hash);
    for (int e = threadIdx.x; e < m; e += blockDim.x) {
        const uint64_t k = ekey[e];
        hash[e] = (uint64_t)(int64_t)(int32_t)(uint32_t)(k >> 32) * 1145141919810ull + (uint64_t)(int64_t)(int32_t)(uint32_t)k;
    }
    all.sync();
    if (m_out && threadIdx.x == 0) *m_out = (uint32_t)m;
    if (m == 0) return true;
    // 3. AB map order.
    map_order(all, 128, kTeams + 1, m, (const uint64_t *)(mem + Lo.hash), Lo.order_at(mem + Lo.order), ord, all_sums);
    // 4. Evaluations, a team each; the warps past the last whole team have none.
    const float nf = __ull2float_rn((uint64_t)n), rn = __fdiv_rn(1.0f, nf);
    const int team_size = (kThreads / 32 / teams) * 32, t = threadIdx.x / team_size;
    if (t < teams) {
        const Team qt{(int)threadIdx.x - t * team_size, team_size, t + 1};
        const int few = min(team_size, 128), few_bar = team_size > 128 ? kTeams + 2 + t : qt.bar;
        uint8_t *const tm = mem + Lo.team + t * Lo.team_stride;
        int *qtab = (int *)(tm + Lo.qtab), *qfirst = (int *)(tm + Lo.qfirst), *qsum = (int *)(tm + Lo.qsum),
            *qslot = (int *)(tm + Lo.qslot), *qc = (int *)(tm + Lo.qc), *qord = (int *)(tm + Lo.qord);
        uint64_t *qval = (uint64_t *)(tm + Lo.qval);  // sign-extended: the identity hash
        double *xh = (double *)(tm + Lo.work), *xm = xh + chain_slots(n);
        float2 *pl = (float2 *)(xm + chain_slots(n));
        float *dev = (float *)(pl + n);
        for (int j = t; j < n_evals; j += teams) {
            const ProxyEval ev = evals[j];
            const float neg = __fdiv_rn(0.5f, ev.abs_eb), t2 = __fadd_rn(ev.t, ev.t), eb2 = __fadd_rn(ev.abs_eb, ev.abs_eb);
            for (uint32_t i = qt.tid; i < hcap; i += qt.size) {
                qtab[i] = INT32_MIN;
                qfirst[i] = INT32_MAX;
                qsum[i] = 0;
            }
            qt.sync();
            // Distinct q values, first occurrence in map order, summed counts.
            for (int k = qt.tid; k < m; k += qt.size) {
                const int e = ord[k];
                int q;
                float dv;
                entry_err(ekey[e], t2, b.stat_eb, neg, eb2, q, dv);
                uint32_t slot = hash_slot((uint64_t)(uint32_t)q, hcap);
                for (uint32_t probe = 0; probe < hcap; probe++) {
                    int prev = atomicCAS(&qtab[slot], INT32_MIN, q);
                    if (prev == INT32_MIN || prev == q) break;
                    if (++slot == hcap) slot = 0;
                }
                qslot[k] = (int)slot;
                atomicMin(&qfirst[slot], k);
                atomicAdd(&qsum[slot], ecnt[e]);
            }
            qt.sync();
            int mq;
            {
                const int per = (m + qt.size - 1) / qt.size, beg = qt.tid * per, end = min(beg + per, m);
                int local = 0;
                for (int k = beg; k < end; k++) local += qfirst[qslot[k]] == k;
                int off = team_excl_scan(qt, local, warp_sums[t], &mq);
                for (int k = beg; k < end; k++)
                    if (qfirst[qslot[k]] == k) {
                        qval[off] = (uint64_t)(int64_t)qtab[qslot[k]];
                        qc[off] = qsum[qslot[k]];
                        off++;
                    }
            }
            qt.sync();
            map_order(qt, few, few_bar, mq, qval, Lo.order_at(tm + Lo.work), qord, warp_sums[t]);
            // The terms of both sums in their order (the stages' arrays are free now).
            for (int k = qt.tid; k < m; k += qt.size) {
                const int e = ord[k];
                int q;
                float dv;
                entry_err(ekey[e], t2, b.stat_eb, neg, eb2, q, dv);
                dev[k] = dv;
                xm[chain_slot(k)] = __dmul_rn((double)ecnt[e], __dmul_rn((double)dv, (double)dv));
            }
            for (int k = qt.tid; k < mq; k += qt.size) {
                const int cnt = qc[qord[k]];
                const float2 v = make_float2(__fmul_rn(__ull2float_rn((uint64_t)cnt), rn), log2tab[cnt]);
                pl[k] = v;
                xh[chain_slot(k)] = __dmul_rn(-(double)v.x, (double)v.y);
            }
            qt.sync();
            const int w = qt.tid >> 5;
            if (w == 0) {
                // h1 chain (get_h_psnr.tpp:23-28).
                const float h1 = warp_chain(xh, mq, [&](float s, int k) { return __fmaf_rn(-pl[k].x, pl[k].y, s); });
                if (qt.tid == 0) h1_out[j] = h1;
            } else if (w == 1) {
                // mse chain (get_h_psnr.tpp:12-22) in map order.
                const float mse = warp_chain(xm, m, [&](float s, int k) {
                    const double dd = (double)dev[k];
                    return __double2float_rn(__fma_rn((double)ecnt[ord[k]], __dmul_rn(dd, dd), (double)s));
                });
                if (qt.tid == 32) x_out[j] = __fmul_rn(__fdiv_rn(R2, mse), nf);
            }
            qt.sync();
        }
    }
    all.sync();
    return true;
}

__device__ __forceinline__ float step_ulps(float v, int k) {
    int32_t b = __float_as_int(v);
    if (v == 0.0f) return k > 0 ? __int_as_float(k) : -__int_as_float(-k);
    if (b >= 0) return __int_as_float(b + k);
    return __int_as_float(b - k);
}

struct Band {
    float mid, lo, hi;
};
__device__ Band psnr_band(float x) {
    Band p;
    if (!(x > 0.0f) || isinf(x) || isnan(x)) {
        float l = (x == 0.0f) ? -INFINITY : (isinf(x) ? INFINITY : __int_as_float(0x7fc00000));
        p.mid = p.lo = p.hi = __fmul_rn(10.0f, l);
        return p;
    }
    float l = __double2float_rn(log10((double)x));
    p.mid = __fmul_rn(10.0f, l);
    p.lo = __fmul_rn(10.0f, step_ulps(l, -4));
    p.hi = __fmul_rn(10.0f, step_ulps(l, 4));
    return p;
}

}  // namespace

// Exact t selection for the listed groups of round l; groups that do not fit the arena go to
// `spill` for the serial kernel.
// Exact replay of group g of one field and round (compress.tpp:91-144 in the maps' order). The
// caller's spill(g) receives a group too large for shared memory (thread 0).
template <class Spill>
__device__ void exact_one(const FieldGeom &fg, const RoundGeom &rg, uint32_t l, const ClassInfo *__restrict__ classes,
                          const float *__restrict__ rec, const float *__restrict__ orig, const float *__restrict__ log2arena,
                          float R2, float t_default, float *__restrict__ tval, int64_t *__restrict__ t_int, uint32_t *fb_count,
                          AmbiguousRecord *amb, uint32_t amb_cap, uint32_t *amb_count, const uint32_t *__restrict__ overrides,
                          uint32_t n_overrides, float *__restrict__ proxies, uint64_t g, uint8_t *smem,
                          const Layout &Lo, float *h1v, float *xv, uint32_t &m_sh, const Spill &spill) {
    const uint64_t nblocks = fg.block_num[0] * fg.block_num[1] * fg.block_num[2];
    const float cand[5] = {1.0f / 16, 1.0f / 4, 9.0f / 32, 5.0f / 16, 11.0f / 32};
    if (g >= nblocks) return;
    const uint64_t b2 = g % fg.block_num[2], b1 = (g / fg.block_num[2]) % fg.block_num[1],
                   b0 = g / (fg.block_num[1] * fg.block_num[2]);
    const uint64_t bb[3] = {b0, b1, b2};
    const int cls = (class_of(b0, fg.block_num[0]) * 3 + class_of(b1, fg.block_num[1])) * 3 + class_of(b2, fg.block_num[2]);
    const ClassInfo ci = classes[cls];
    const int d = rg.dir;
    ExactGroup eg;
    for (int a = 0; a < 3; a++) {
        uint64_t lo = fg.origin[a] + bb[a] * fg.block_shape[a];
        uint64_t hi = min(fg.origin[a] + (bb[a] + 1) * fg.block_shape[a] + 1, fg.n[a]);
        if (a != d && lo != 0) lo += rg.stride[a];
        if (a == d) {
            lo += 3 * rg.stride[a] / 2;
            hi -= 3 * rg.stride[a] / 2;
        }
        eg.box.lo[a] = lo;
        eg.box.hi[a] = hi;
        eg.box.step[a] = rg.stride[a] * ci.ss;
    }
    eg.box.dist = rg.dist;
    eg.box.neg_2_stat_eb = rg.neg_2_stat_eb;
    eg.box.stat_eb = rg.stat_eb;
    eg.n = ci.n;
    __shared__ ProxyEval ev[5];
    __shared__ Band band[5];
    if (threadIdx.x < 5) ev[threadIdx.x] = ProxyEval{cand[threadIdx.x], rg.eb};
    if (threadIdx.x == 0) m_sh = 0;
    __syncthreads();
    bool ok = exact_eval(eg, rec, orig, fg.n[1] * fg.n[2], fg.n[2], ev, 5, R2, log2arena + ci.log2_off, smem, Lo, h1v,
                         xv, &m_sh);
    __syncthreads();
    if (ok && threadIdx.x < 5) band[threadIdx.x] = psnr_band(xv[threadIdx.x]);
    __syncthreads();
    if (!ok) {
        if (threadIdx.x == 0) spill(g);
        __syncthreads();
        return;
    }
    if (threadIdx.x == 0) {
        float best_t = t_default;
        bool fb = m_sh == 0;
        bool forced = false;
        for (uint32_t i = 0; i < n_overrides; i++)
            if (overrides[3 * i] == (uint32_t)g && overrides[3 * i + 1] == l) {
                forced = true;
                best_t = __uint_as_float(overrides[3 * i + 2]);
            }
        if (!fb && !forced) {
            if (proxies)
                for (int c = 0; c < 5; c++) {
                    proxies[g * 10 + c] = h1v[c];
                    proxies[g * 10 + 5 + c] = xv[c];
                }
            int best = 1;
            bool ambiguous = false;
            for (int c = 0; c < 5; c++) {
                if (cand[c] == cand[best]) continue;
                float d_h1 = __fsub_rn(h1v[best], h1v[c]);
                bool accept;
                if (__float_as_uint(xv[c]) == __float_as_uint(xv[best]) && isfinite(xv[c]) && xv[c] > 0.0f) {
                    accept = __fmaf_rn(d_h1, rg.slope, 0.0f) > 0.0f;
                } else {
                    const Band pc = band[c], pb = band[best];
                    float s_mid = __fmaf_rn(d_h1, rg.slope, __fsub_rn(pc.mid, pb.mid));
                    float s_lo = __fmaf_rn(d_h1, rg.slope, __fsub_rn(pc.lo, pb.hi));
                    float s_hi = __fmaf_rn(d_h1, rg.slope, __fsub_rn(pc.hi, pb.lo));
                    if (!((s_lo > 0.0f) || !(s_hi > 0.0f))) ambiguous = true;
                    accept = s_mid > 0.0f;
                }
                if (accept) best = c;
            }
            best_t = cand[best];
            if (ambiguous) {
                uint32_t k = atomicAdd(amb_count, 1u);
                if (k < amb_cap) {
                    AmbiguousRecord &r = amb[k];
                    r.block = (uint32_t)g;
                    r.round = l;
                    r.provisional = (int32_t)lround_f(__fmul_rn(best_t, (float)fg.t_precision));
                    for (int c = 0; c < 5; c++) {
                        r.h1[c] = h1v[c];
                        r.x[c] = xv[c];
                    }
                }
            }
        }
        if (fb) atomicAdd(fb_count, 1u);
        tval[g] = best_t;
        t_int[g * fg.layer_num + l] = lround_f(__fmul_rn(best_t, (float)fg.t_precision));
    }
    __syncthreads();
}

struct ListSpill {
    uint32_t *list, *count;
    __device__ void operator()(uint64_t g) const { list[atomicAdd(count, 1u)] = (uint32_t)g; }
};

__global__ void __launch_bounds__(kThreads, 1)
    tsel_exact_kernel(FieldGeom fg, RoundGeom rg, uint32_t l, const ClassInfo *__restrict__ classes,
                      const float *__restrict__ rec, const float *__restrict__ orig, const float *__restrict__ log2arena,
                      float R2, float t_default, float *__restrict__ tval, int64_t *__restrict__ t_int,
                      uint32_t *__restrict__ fb_count, AmbiguousRecord *amb, uint32_t amb_cap, uint32_t *amb_count,
                      const uint32_t *__restrict__ overrides, uint32_t n_overrides, float *__restrict__ proxies,
                      const uint32_t *__restrict__ list, const uint32_t *__restrict__ list_count, uint32_t *spill,
                      uint32_t *spill_count, const __grid_constant__ Layout Lo) {
    extern __shared__ __align__(16) uint8_t smem[];
    const uint32_t items = *list_count;
    __shared__ float h1v[kMaxEvals], xv[kMaxEvals];
    __shared__ uint32_t m_sh;
    const ListSpill sp{spill, spill_count};
    for (uint32_t it = blockIdx.x; it < items; it += gridDim.x)
        exact_one(fg, rg, l, classes, rec, orig, log2arena, R2, t_default, tval, t_int, fb_count, amb, amb_cap, amb_count,
                  overrides, n_overrides, proxies, list[it], smem, Lo, h1v, xv, m_sh, sp);
}

// Batched form: the (field << 32 | group) entries that the batched fast path handed off, for all
// fields of a batch at once; spills go to one list of entries of the same form.
struct PairSpill {
    unsigned long long *list;
    uint32_t *count;
    uint32_t f;
    __device__ void operator()(uint64_t g) const { list[atomicAdd(count, 1u)] = ((unsigned long long)f << 32) | g; }
};

__global__ void __launch_bounds__(kThreads, 1)
    tsel_exact_batch_kernel(const BatchField *__restrict__ F, uint32_t l, const float *__restrict__ log2arena,
                            float t_default, const unsigned long long *__restrict__ list, const uint32_t *__restrict__ list_count,
                            unsigned long long *spill, uint32_t *spill_count, const __grid_constant__ Layout Lo) {
    extern __shared__ __align__(16) uint8_t smem[];
    const uint32_t items = *list_count;
    __shared__ float h1v[kMaxEvals], xv[kMaxEvals];
    __shared__ uint32_t m_sh;
    for (uint32_t it = blockIdx.x; it < items; it += gridDim.x) {
        const unsigned long long e = list[it];
        const uint32_t f = (uint32_t)(e >> 32);
        const BatchField &B = F[f];
        const uint64_t nb = B.fg.block_num[0] * B.fg.block_num[1] * B.fg.block_num[2];
        const PairSpill sp{spill, spill_count, f};
        exact_one(B.fg, B.rounds[l], l, B.classes + 27 * l, B.rec, B.in, log2arena, B.R2, t_default, B.tval, B.tint, &B.cnt->fb,
                  B.amb, B.amb_cap, &B.cnt->amb_count, nullptr, 0, B.proxies ? B.proxies + nb * l * 10 : nullptr,
                  e & 0xffffffffull, smem, Lo, h1v, xv, m_sh, sp);
    }
}

// Batched form of tsel_exact_global_kernel: the entries the batched exact kernel spilled (groups
// above its shared-memory capacity), a CTA per group in its slice of global scratch; what this
// cannot take (keys outside int32) goes on to `spill` for the serial kernel.
__global__ void __launch_bounds__(kThreads, 1)
    tsel_exact_global_batch_kernel(const BatchField *__restrict__ F, uint32_t l, const float *__restrict__ log2arena,
                                   float t_default, const unsigned long long *__restrict__ list,
                                   const uint32_t *__restrict__ list_count, unsigned long long *spill, uint32_t *spill_count,
                                   uint8_t *scratch, uint64_t stride, const __grid_constant__ Layout Lo) {
    uint8_t *mine = scratch + blockIdx.x * stride;
    const uint32_t items = *list_count;
    __shared__ float h1v[kMaxEvals], xv[kMaxEvals];
    __shared__ uint32_t m_sh;
    for (uint32_t it = blockIdx.x; it < items; it += gridDim.x) {
        const unsigned long long e = list[it];
        const uint32_t f = (uint32_t)(e >> 32);
        const BatchField &B = F[f];
        const uint64_t nb = B.fg.block_num[0] * B.fg.block_num[1] * B.fg.block_num[2];
        const PairSpill sp{spill, spill_count, f};
        exact_one(B.fg, B.rounds[l], l, B.classes + 27 * l, B.rec, B.in, log2arena, B.R2, t_default, B.tval, B.tint, &B.cnt->fb,
                  B.amb, B.amb_cap, &B.cnt->amb_count, nullptr, 0, B.proxies ? B.proxies + nb * l * 10 : nullptr,
                  e & 0xffffffffull, mine, Lo, h1v, xv, m_sh, sp);
    }
}

// Box blockIdx.x, evaluations [kTeams * blockIdx.y, + kTeams): each CTA rebuilds the box's map and runs
// one batch of evaluations side by side.
__device__ __forceinline__ void slope_box(const SampleBox *__restrict__ boxes, const ProxyEval *__restrict__ evals,
                                          uint32_t n_evals, const float *__restrict__ orig, uint64_t n1n2, uint64_t n2,
                                          const float *__restrict__ log2arena, float R2, float *__restrict__ h1_out,
                                          float *__restrict__ x_out, uint32_t *__restrict__ m_out,
                                          uint32_t *__restrict__ err_word, const Layout &Lo) {
    extern __shared__ __align__(16) uint8_t smem[];
    __shared__ float h1v[kMaxEvals], xv[kMaxEvals];
    const uint32_t g = blockIdx.x, e0 = kTeams * blockIdx.y;
    if (e0 >= n_evals) return;
    const uint32_t ne = min((uint32_t)kTeams, n_evals - e0);
    ExactGroup eg;
    eg.box = boxes[g];
    eg.n = eg.box.n;
    uint32_t m = 0;
    bool ok = exact_eval(eg, orig, orig, n1n2, n2, evals + e0, (int)ne, R2, log2arena + eg.box.log2_off, smem, Lo,
                         h1v, xv, &m);
    __syncthreads();
    if (!ok) {
        if (threadIdx.x == 0) atomicOr(err_word, 2u);
        return;
    }
    if (threadIdx.x == 0 && blockIdx.y == 0) m_out[g] = m;
    for (uint32_t e = threadIdx.x; e < ne; e += blockDim.x) {
        h1_out[g * n_evals + e0 + e] = h1v[e];
        x_out[g * n_evals + e0 + e] = xv[e];
    }
}

__global__ void __launch_bounds__(kThreads, 1)
    slope_exact_kernel(const SampleBox *__restrict__ boxes, const ProxyEval *__restrict__ evals, uint32_t n_evals,
                       const float *__restrict__ orig, uint64_t n1n2, uint64_t n2, const float *__restrict__ log2arena,
                       float R2, float *__restrict__ h1_out, float *__restrict__ x_out, uint32_t *__restrict__ m_out,
                       uint32_t *__restrict__ err_word, const __grid_constant__ Layout Lo) {
    slope_box(boxes, evals, n_evals, orig, n1n2, n2, log2arena, R2, h1_out, x_out, m_out, err_word, Lo);
}

// The fields of a batch (z): eight fields of 16 MB each 0.26 -> 0.04 ms, and a wait of the host for
// all of them instead of one each.
__global__ void __launch_bounds__(kThreads, 1)
    slope_batch_kernel(const SlopeField *__restrict__ fields, uint32_t n_evals, const float *__restrict__ log2arena,
                       SlopeOut *__restrict__ out, const __grid_constant__ Layout Lo) {
    const SlopeField &f = fields[blockIdx.z];
    SlopeOut &o = out[blockIdx.z];
    slope_box(f.boxes, f.evals, n_evals, f.orig, f.n1n2, f.n2, log2arena, f.R2, o.h1, o.x, o.m, &o.err, Lo);
}

// The same exact replay for groups larger than shared memory holds: each CTA works in its own
// slice of a global scratch arena (stride bytes, L2-resident) instead of shared memory, so a group
// of up to `cap` samples is still replayed by a whole CTA rather than by one thread. Groups it
// cannot take (more samples than cap, keys outside int32) go to `spill` for the serial kernel.
__global__ void __launch_bounds__(kThreads, 1)
    tsel_exact_global_kernel(FieldGeom fg, RoundGeom rg, uint32_t l, const ClassInfo *__restrict__ classes,
                             const float *__restrict__ rec, const float *__restrict__ orig,
                             const float *__restrict__ log2arena, float R2, float t_default, float *__restrict__ tval,
                             int64_t *__restrict__ t_int, uint32_t *__restrict__ fb_count, AmbiguousRecord *amb,
                             uint32_t amb_cap, uint32_t *amb_count, const uint32_t *__restrict__ overrides,
                             uint32_t n_overrides, float *__restrict__ proxies, const uint32_t *__restrict__ list,
                             const uint32_t *__restrict__ list_count, uint32_t *spill, uint32_t *spill_count,
                             uint8_t *scratch, uint64_t stride, const __grid_constant__ Layout Lo) {
    uint8_t *mine = scratch + blockIdx.x * stride;
    const uint32_t items = *list_count;
    __shared__ float h1v[kMaxEvals], xv[kMaxEvals];
    __shared__ uint32_t m_sh;
    const ListSpill sp{spill, spill_count};
    for (uint32_t it = blockIdx.x; it < items; it += gridDim.x)
        exact_one(fg, rg, l, classes, rec, orig, log2arena, R2, t_default, tval, t_int, fb_count, amb, amb_cap, amb_count,
                  overrides, n_overrides, proxies, list[it], mine, Lo, h1v, xv, m_sh, sp);
}

__global__ void __launch_bounds__(kThreads, 1)
    slope_exact_global_kernel(const SampleBox *__restrict__ boxes, const ProxyEval *__restrict__ evals, uint32_t n_evals,
                              const float *__restrict__ orig, uint64_t n1n2, uint64_t n2,
                              const float *__restrict__ log2arena, float R2, float *__restrict__ h1_out,
                              float *__restrict__ x_out, uint32_t *__restrict__ m_out, uint32_t *__restrict__ err_word,
                              uint8_t *scratch, uint64_t stride, const __grid_constant__ Layout Lo) {
    __shared__ float h1v[kMaxEvals], xv[kMaxEvals];
    const uint32_t g = blockIdx.x, e0 = kTeams * blockIdx.y;  // as slope_exact_kernel
    if (e0 >= n_evals) return;
    const uint32_t ne = min((uint32_t)kTeams, n_evals - e0);
    ExactGroup eg;
    eg.box = boxes[g];
    eg.n = eg.box.n;
    uint32_t m = 0;
    bool ok = exact_eval(eg, orig, orig, n1n2, n2, evals + e0, (int)ne, R2, log2arena + eg.box.log2_off,
                         scratch + (blockIdx.y * gridDim.x + g) * stride, Lo, h1v, xv, &m);
    __syncthreads();
    if (!ok) {
        if (threadIdx.x == 0) atomicOr(err_word, 2u);
        return;
    }
    if (threadIdx.x == 0 && blockIdx.y == 0) m_out[g] = m;
    for (uint32_t e = threadIdx.x; e < ne; e += blockDim.x) {
        h1_out[g * n_evals + e0 + e] = h1v[e];
        x_out[g * n_evals + e0 + e] = xv[e];
    }
}

// Working-set bytes of groups of up to n samples: with one evaluation at a time (what a kernel
// needs at least), and with as many side by side as are worth having.
uint32_t exact_smem_bytes(uint32_t n) { return Layout(n, 1).total; }
uint32_t exact_full_bytes(uint32_t n) { return Layout(n, kTeams).total; }
uint32_t slope_batches(uint32_t n_evals) { return (n_evals + kTeams - 1) / kTeams; }

namespace {

// Shared memory of a launch whose largest group has `most` samples and whose kernel takes groups of
// up to `cap`: the side-by-side tables where they fit. The kernel's limit is the most that any launch
// uses: it is one for all threads of the process, and for launches that a graph keeps.
cudaError_t exact_shared(const void *kernel, uint32_t cap, uint32_t most, Layout &lo) {
    int dev = 0, lim = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&lim, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    if (e != cudaSuccess) return e;
    const uint32_t limit = (uint32_t)lim - kExactStatic;
    lo = exact_layout(most < cap ? most : cap, limit);
    return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)limit);
}

}  // namespace

cudaError_t launch_tsel_exact_global(const FieldGeom &fg, const RoundGeom &rg, uint32_t l, const ClassInfo *classes,
                                     const float *rec, const float *orig, const float *log2arena, float R2, float t_default,
                                     float *tval, int64_t *t_int, uint32_t *fb_count, AmbiguousRecord *amb, uint32_t amb_cap,
                                     uint32_t *amb_count, const uint32_t *overrides, uint32_t n_overrides, float *proxies,
                                     const uint32_t *list, const uint32_t *list_count, uint32_t *spill, uint32_t *spill_count,
                                     uint8_t *scratch, uint64_t stride, uint32_t cap, unsigned grid, cudaStream_t st) {
    if (grid == 0) return cudaSuccess;
    tsel_exact_global_kernel<<<grid, kThreads, 0, st>>>(fg, rg, l, classes, rec, orig, log2arena, R2, t_default, tval, t_int,
                                                        fb_count, amb, amb_cap, amb_count, overrides, n_overrides, proxies,
                                                        list, list_count, spill, spill_count, scratch, stride,
                                                        exact_layout(cap, stride));
    count_launch();
    return cudaGetLastError();
}

cudaError_t launch_slope_exact_global(const SampleBox *boxes, const ProxyEval *evals, uint32_t n_evals, const float *orig,
                                      uint64_t n1n2, uint64_t n2, const float *log2arena, float R2, float *h1, float *x,
                                      uint32_t *m_out, uint32_t *err, uint8_t *scratch, uint64_t stride, uint32_t cap,
                                      uint32_t nboxes, cudaStream_t st) {
    if (nboxes == 0) return cudaSuccess;
    slope_exact_global_kernel<<<dim3(nboxes, slope_batches(n_evals)), kThreads, 0, st>>>(boxes, evals, n_evals, orig, n1n2, n2, log2arena, R2, h1, x, m_out,
                                                           err, scratch, stride, exact_layout(cap, stride));
    count_launch();
    return cudaGetLastError();
}

cudaError_t launch_tsel_exact(const FieldGeom &fg, const RoundGeom &rg, uint32_t l, const ClassInfo *classes, const float *rec,
                              const float *orig, const float *log2arena, float R2, float t_default, float *tval,
                              int64_t *t_int, uint32_t *fb_count, AmbiguousRecord *amb, uint32_t amb_cap,
                              uint32_t *amb_count, const uint32_t *overrides, uint32_t n_overrides, float *proxies,
                              const uint32_t *list, const uint32_t *list_count, uint32_t *spill, uint32_t *spill_count,
                              uint32_t cap, uint32_t most, unsigned grid, cudaStream_t st) {
    Layout lo(1, 1);
    cudaError_t e = exact_shared((const void *)tsel_exact_kernel, cap, most, lo);
    if (e != cudaSuccess) return e;
    tsel_exact_kernel<<<grid, kThreads, lo.total, st>>>(fg, rg, l, classes, rec, orig, log2arena, R2, t_default, tval, t_int,
                                                     fb_count, amb, amb_cap, amb_count, overrides, n_overrides, proxies, list,
                                                     list_count, spill, spill_count, lo);
    count_launch();
    return cudaGetLastError();
}

cudaError_t launch_tsel_exact_global_batch(const BatchField *F, uint32_t l, const float *log2arena, float t_default,
                                           const unsigned long long *list, const uint32_t *list_count,
                                           unsigned long long *spill, uint32_t *spill_count, uint8_t *scratch, uint64_t stride,
                                           uint32_t cap, unsigned grid, cudaStream_t st) {
    if (grid == 0) return cudaSuccess;
    tsel_exact_global_batch_kernel<<<grid, kThreads, 0, st>>>(F, l, log2arena, t_default, list, list_count, spill, spill_count,
                                                              scratch, stride, exact_layout(cap, stride));
    count_launch();
    return cudaGetLastError();
}

cudaError_t launch_tsel_exact_batch(const BatchField *F, uint32_t l, const float *log2arena, float t_default,
                                    const unsigned long long *list, const uint32_t *list_count, unsigned long long *spill,
                                    uint32_t *spill_count, uint32_t cap, uint32_t most, unsigned grid, cudaStream_t st) {
    Layout lo(1, 1);
    cudaError_t e = exact_shared((const void *)tsel_exact_batch_kernel, cap, most, lo);
    if (e != cudaSuccess) return e;
    tsel_exact_batch_kernel<<<grid, kThreads, lo.total, st>>>(F, l, log2arena, t_default, list, list_count, spill, spill_count, lo);
    count_launch();
    return cudaGetLastError();
}

cudaError_t launch_slope_exact(const SampleBox *boxes, const ProxyEval *evals, uint32_t n_evals, const float *orig,
                               uint64_t n1n2, uint64_t n2, const float *log2arena, float R2, float *h1, float *x,
                               uint32_t *m_out, uint32_t *err, uint32_t cap, uint32_t most, uint32_t nboxes,
                               cudaStream_t st) {
    if (nboxes == 0) return cudaSuccess;
    Layout lo(1, 1);
    cudaError_t e = exact_shared((const void *)slope_exact_kernel, cap, most, lo);
    if (e != cudaSuccess) return e;
    const dim3 grid(nboxes, slope_batches(n_evals));
    slope_exact_kernel<<<grid, kThreads, lo.total, st>>>(boxes, evals, n_evals, orig, n1n2, n2, log2arena, R2, h1, x, m_out, err,
                                                      lo);
    count_launch();
    return cudaGetLastError();
}

cudaError_t launch_slope_batch(const SlopeField *fields, uint32_t nf, uint32_t n_evals, const float *log2arena, SlopeOut *out,
                               uint32_t cap, uint32_t most, cudaStream_t st) {
    Layout lo(1, 1);
    cudaError_t e = exact_shared((const void *)slope_batch_kernel, cap, most, lo);
    if (e != cudaSuccess) return e;
    slope_batch_kernel<<<dim3(3, slope_batches(n_evals), nf), kThreads, lo.total, st>>>(fields, n_evals, log2arena, out, lo);
    count_launch();
    return cudaGetLastError();
}

}  // namespace asz
