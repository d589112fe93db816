// Fused rounds along axis 2: whole plans of them compressed (e.g. "cubic2_012" on every level), and runs
// of consecutive ones decompressed.
//
// Compression. With all rounds on one axis, the pivot stride is 1 on the other two axes, so a block owns whole
// lines along axis 2 and every stencil read of a round stays on the target's own line. The lines of
// a "column" (the blocks sharing one (block0, block1) pair) can therefore be held in shared memory
// by one CTA for all rounds: the field is read and written once instead of once per round.
// Results are those of the per-round kernels (same stencils, same arithmetic, same QB indices);
// rounds run in the same order, and a round's coefficient selection sees the column after the
// previous round, as the per-round kernels do.
#include <cuda_runtime.h>

#include <algorithm>

#include "dev_common.cuh"
#include "geometry.cuh"
#include "launch.h"
#include "round_ops.cuh"
#include "tsel_fast.cuh"

namespace asz {
namespace {

constexpr uint32_t kMaxColumnBlocks = 64;  // blocks along axis 2 (the host checks the plan)

__host__ __device__ inline uint32_t column_count(uint32_t set, uint32_t nb0, uint32_t nb1) {
    if (set == kColumnsInterior) return (nb0 - 1) * (nb1 - 1);
    if (set == kColumnsEdge) return nb0 + nb1 - 1;
    return nb0 * nb1;
}

// The lines of column (b0, b1): coordinates [lo, lo + nl) on axes 0 and 1. A block's upper face is
// its own and its lower face the block below's, except at 0, so the columns' lines partition the
// (axis 0, axis 1) plane.
struct Column {
    uint32_t lo0, lo1, nl0, nl1;
};

__device__ __forceinline__ Column column_of(const FieldGeom &fg, uint32_t b0, uint32_t b1) {
    const uint32_t s0 = (uint32_t)fg.block_shape[0], s1 = (uint32_t)fg.block_shape[1];
    Column col;
    col.lo0 = b0 ? b0 * s0 + 1 : 0;
    col.lo1 = b1 ? b1 * s1 + 1 : 0;
    const uint32_t hi0 = (uint32_t)min((uint64_t)b0 * s0 + s0 + 1, fg.n[0]);
    const uint32_t hi1 = (uint32_t)min((uint64_t)b1 * s1 + s1 + 1, fg.n[1]);
    col.nl0 = hi0 > col.lo0 ? hi0 - col.lo0 : 0;
    col.nl1 = hi1 > col.lo1 ? hi1 - col.lo1 : 0;
    return col;
}

// Column sets of one launch: every column, the columns with b0 >= 1 and b1 >= 1 (at most
// block_shape[0] * block_shape[1] lines each), or the others (b0 == 0 or b1 == 0, one line more on
// each such axis). Splitting them lets the larger set run with less shared memory per CTA.
__device__ __forceinline__ void column_at(uint32_t set, uint32_t it, uint32_t nb1, uint32_t &b0, uint32_t &b1) {
    if (set == kColumnsInterior) {
        b0 = 1 + it / (nb1 - 1);
        b1 = 1 + it % (nb1 - 1);
    } else if (set == kColumnsEdge) {
        b0 = it < nb1 ? 0 : it - nb1 + 1;
        b1 = it < nb1 ? it : 0;
    } else {
        b0 = it / nb1;
        b1 = it % nb1;
    }
}

// Warp per line, coalesced along axis 2.
__device__ __forceinline__ void load_lines(const FieldGeom &fg, const Column &col, const float *__restrict__ g, float *s) {
    const uint32_t n2 = (uint32_t)fg.n[2], nl = col.nl0 * col.nl1;
    for (uint32_t line = threadIdx.x >> 5; line < nl; line += blockDim.x >> 5) {
        const uint32_t i0 = col.lo0 + line / col.nl1, i1 = col.lo1 + line % col.nl1;
        const float *src = g + ((uint64_t)i0 * fg.n[1] + i1) * n2;
        for (uint32_t x = threadIdx.x & 31; x < n2; x += 32) s[line * n2 + x] = src[x];
    }
}

__device__ __forceinline__ void store_lines(const FieldGeom &fg, const Column &col, const float *s, float *__restrict__ g) {
    const uint32_t n2 = (uint32_t)fg.n[2], nl = col.nl0 * col.nl1;
    for (uint32_t line = threadIdx.x >> 5; line < nl; line += blockDim.x >> 5) {
        const uint32_t i0 = col.lo0 + line / col.nl1, i1 = col.lo1 + line % col.nl1;
        float *dst = g + ((uint64_t)i0 * fg.n[1] + i1) * n2;
        for (uint32_t x = threadIdx.x & 31; x < n2; x += 32) dst[x] = s[line * n2 + x];
    }
}

__host__ __device__ constexpr size_t align16(size_t b) { return (b + 15) & ~size_t(15); }

// ---------------------------------------------------------------------------------------------
// Decompression: consecutive rounds along axis 2, a warp per line. Nothing crosses lines here (the t
// codes are given), so a line needs only its own known points: the warp loads them, runs the rounds
// in shared memory and stores the line once. decompress.tpp:34: value = fma(-qb, 2eb, pred) in
// double, t = t_int / t_precision.
//
// A launch per round reads and writes the line's sectors again in every round of stride up to 8, and
// costs a launch for the few targets of a coarse one. Here the traffic is the QBs read and the field
// written once, and what bounds it is the instructions issued per target, so the parts that are the
// same for a round or a line are kept out of the targets' loop and the QBs' offsets are 32-bit from
// the line's base. A round's first QBs are loaded during the round before. One value in 32 is
// padding: with it the lattices' power-of-two strides meet no bank twice. 512x512x512 in nine rounds:
// 1.70 -> 0.72 ms (a table for the one block too, and a line a warp: 1.04), 75% of the issue slots and
// 40% of the conversion units taken; 40x48x64 in five: 53 -> 13 us. Four CTAs of 64 registers: five
// of 48 spill (0.82 ms).
constexpr uint32_t kRunRounds = 16, kRunAhead = 4, kRunWarps = 8, kRunCtas = 4;
constexpr uint64_t kRunSmem = 227 * 1024, kRunSm = 228 * 1024;  // shared memory of a CTA, of an SM

struct RunRound {
    double eb2;
    uint64_t qoff, qb_total;  // the stream's first QB and its length
    uint64_t ent2;            // axis 2's entries
    uint32_t hs, count, first, total2, order, l;
    uint32_t cubics, quintics;  // one block: targets [1, 1 + cubics) are cubic, but [2, 2 + quintics) quintic
};
struct LineRun {
    RunRound r[kRunRounds];
    uint64_t ent0, ent1, total1, n1n2;
    uint32_t rounds, lines, T1, n2, nb1, nb2, layers, targets, known, step, tab_words, line_words;
    float tp;
};

__device__ __forceinline__ uint32_t padded(uint32_t i) { return i + (i >> 5); }

__device__ __forceinline__ float cubic(float m3, float m1, float p1, float p3, double c1, double c2) {
    const float a = __double2float_rn(__dmul_rn((double)__fadd_rn(m3, p3), c1));
    return __double2float_rn(__fma_rn(c2, (double)__fadd_rn(m1, p1), (double)a));
}

// The cases other than the cubic and the quintic one, without branches: neighbours that a case does
// not use are read from the target's own place.
__device__ __forceinline__ float predict_edge(const float *s, uint32_t i, uint32_t hs, uint32_t sc) {
    const bool has_p1 = sc != kStencilLeft1 && sc != kStencilRight1, right = sc >= kStencilRight1;
    const float m1 = s[padded(i - hs)], p1 = s[padded(has_p1 ? i + hs : i)], m3 = s[padded(right ? i - 3 * hs : i)],
                p3 = s[padded(sc == kStencilLeft3 ? i + 3 * hs : i)];
    float v = m1;
    if (sc == kStencilLeft2) v = __fmul_rn(__fadd_rn(m1, p1), 0.5f);
    if (sc == kStencilLeft3) v = __fmul_rn(__fsub_rn(__fmaf_rn(m1, 3.0f, __fmul_rn(p1, 6.0f)), p3), 0.125f);
    if (sc == kStencilRight1) v = __fmul_rn(__fmaf_rn(m1, 3.0f, -m3), 0.5f);
    if (sc == kStencilRight2) v = __fmul_rn(__fmaf_rn(p1, 3.0f, __fmaf_rn(m1, 6.0f, -m3)), 0.125f);
    return v;
}

// A line: its place in the field, its blocks, and the parts of its QBs' offsets that no round changes.
struct RunLine {
    AxisEntry e0, e1;
    float *g;
    uint64_t blk, base;
};

__device__ __forceinline__ RunLine run_line(const LineRun &R, const AxisEntry *ent, float *rec, uint32_t line) {
    RunLine l;
    const uint32_t k0 = line / R.T1;
    l.e0 = load_entry(ent + R.ent0 + k0);
    l.e1 = load_entry(ent + R.ent1 + (line - k0 * R.T1));
    l.g = rec + (uint64_t)l.e0.ii * R.n1n2 + (uint64_t)l.e1.ii * R.n2;
    l.blk = ((uint64_t)l.e0.bb * R.nb1 + l.e1.bb) * R.nb2;
    l.base = l.e0.pre * R.total1 + (uint64_t)l.e0.cc * l.e1.pre;
    return l;
}

// A line's QBs in a round: where its part of the stream starts, and the factors of a target's offset,
// mul * pre + (u * cc + jj) * w + x (get_qb_index).
struct LineQBs {
    const int32_t *q;
    uint32_t limit;  // QBs from q to the stream's end
    uint32_t mul, u, w, x;
};

__device__ __forceinline__ LineQBs line_qbs(const RunRound &m, const RunLine &l, const int32_t *qb) {
    LineQBs L;
    const uint64_t off = l.base * m.total2, left = off < m.qb_total ? m.qb_total - off : 0;
    L.mul = l.e0.cc * l.e1.cc;
    L.u = m.order == 2 ? l.e0.jj * l.e1.cc + l.e1.jj : m.order == 0 ? l.e1.jj : l.e0.jj;
    L.w = m.order == 2 ? 1 : m.order == 0 ? l.e0.cc : l.e1.cc;
    L.x = m.order == 2 ? 0 : m.order == 0 ? l.e0.jj : l.e1.jj;
    L.q = qb + m.qoff + off;
    L.limit = left < 0xffffffffu ? (uint32_t)left : 0xffffffffu;
    return L;
}

__device__ __forceinline__ float run_t(const LineRun &R, const int64_t *t_int, uint64_t blk, uint32_t r) {
    return __fdiv_rn(__ll2float_rn(__ldg(t_int + blk * R.layers + R.r[r].l)), R.tp);
}

// Several blocks along axis 2: a warp per line; the targets' block offsets, QB boxes and stencil cases
// come from a table in shared memory.
__global__ void __launch_bounds__(32 * kRunWarps, kRunCtas)
    lines_decompress_kernel(const __grid_constant__ LineRun R, const AxisEntry *__restrict__ ent, const int64_t *__restrict__ t_int,
                            const int32_t *__restrict__ qb, float *__restrict__ rec, uint32_t *err_word) {
    extern __shared__ __align__(16) uint32_t run_smem[];
    const uint32_t warps = blockDim.x >> 5, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    // Axis 2's entries of all targets: {pre | cc << 16, jj | stencil << 16 | bb << 19}.
    uint2 *tab = reinterpret_cast<uint2 *>(run_smem);
    float *s = reinterpret_cast<float *>(run_smem + R.tab_words + warp * R.line_words);
    float *ts = s + R.line_words - R.nb2 * R.rounds;
    for (uint32_t r = 0; r < R.rounds; r++)
        for (uint32_t k = threadIdx.x; k < R.r[r].count; k += blockDim.x) {
            const AxisEntry e = load_entry(ent + R.r[r].ent2 + k);
            tab[R.r[r].first + k] = make_uint2((uint32_t)e.pre | e.cc << 16, e.jj | e.stencil << 16 | e.bb << 19);
        }
    __syncthreads();
    for (uint32_t line = blockIdx.x * warps + warp; line < R.lines; line += gridDim.x * warps) {
        const RunLine l = run_line(R, ent, rec, line);
        auto load_qbs = [&](const LineQBs &L, uint32_t r, uint32_t k, int32_t (&q)[kRunAhead]) {
            const uint32_t count = R.r[r].count, first = R.r[r].first;
#pragma unroll
            for (uint32_t j = 0; j < kRunAhead; j++) {
                if (k + 32 * j >= count) break;
                const uint32_t i = k + 32 * j + lane;
                q[j] = 0;
                if (i >= count) continue;
                const uint2 e = tab[first + i];
                const uint32_t o = L.mul * (e.x & 0xffff) + (L.u * (e.x >> 16) + (e.y & 0xffff)) * L.w + L.x;
                if (o < L.limit) q[j] = __ldg(L.q + o);
                else atomicOr(err_word, 4u);
            }
        };
        int32_t q[kRunAhead];
        LineQBs L = line_qbs(R.r[0], l, qb);
        load_qbs(L, 0, 0, q);
        for (uint32_t k = lane; k < R.known; k += 32) s[padded(k * R.step)] = l.g[k * R.step];
        for (uint32_t k = lane; k < R.nb2 * R.rounds; k += 32) ts[k] = run_t(R, t_int, l.blk + k / R.rounds, k % R.rounds);
        __syncwarp();
        for (uint32_t r = 0; r < R.rounds; r++) {
            const uint32_t hs = R.r[r].hs, count = R.r[r].count, first = R.r[r].first;
            const double eb2 = R.r[r].eb2;
            for (uint32_t k = 0; k < count; k += 32 * kRunAhead) {
                int32_t next[kRunAhead];
                if (k + 32 * kRunAhead < count) {
                    load_qbs(L, r, k + 32 * kRunAhead, next);
                } else if (r + 1 < R.rounds) {
                    L = line_qbs(R.r[r + 1], l, qb);
                    load_qbs(L, r + 1, 0, next);
                }
#pragma unroll
                for (uint32_t j = 0; j < kRunAhead; j++) {
                    if (k + 32 * j >= count) break;
                    const uint32_t i = k + 32 * j + lane;
                    if (i >= count) continue;
                    const uint32_t ii = hs * (2 * i + 1), w = tab[first + i].y, sc = (w >> 16) & 7;
                    const float m1 = s[padded(ii - hs)];
                    float pred;
                    if (sc <= kStencilQuintic) {
                        const float p1 = s[padded(ii + hs)], m3 = s[padded(ii - 3 * hs)], p3 = s[padded(ii + 3 * hs)];
                        if (sc == kStencilCubic) {
                            const double td = (double)ts[(w >> 19) * R.rounds + r];
                            pred = cubic(m3, m1, p1, p3, __dsub_rn(0.25, td), __dadd_rn(0.25, td));
                        } else {
                            const StencilIn v{m1, p1, m3, p3, s[padded(ii - 5 * hs)], s[padded(ii + 5 * hs)]};
                            pred = predict_loaded(v, kStencilQuintic, 0.0f);
                        }
                    } else {
                        pred = predict_edge(s, ii, hs, sc);
                    }
                    s[padded(ii)] = __double2float_rn(__fma_rn(-(double)q[j], eb2, (double)pred));
                }
#pragma unroll
                for (uint32_t j = 0; j < kRunAhead; j++) q[j] = next[j];
            }
            __syncwarp();
        }
        const uint32_t hs = R.r[R.rounds - 1].hs;
        for (uint32_t i = lane * hs; i < R.n2; i += 32 * hs) l.g[i] = s[padded(i)];
        __syncwarp();
    }
}

// One block along axis 2: no table, everything follows from a target's index. kLanes lanes per line
// (16: two lines in a warp, which then share the coarse rounds' steps). A round's interior targets
// are 1 .. cubics; their shared-memory addresses move by a constant from step to step, because a step
// of kLanes targets is a multiple of 32 values. The targets at the line's ends (the first, and up to
// two last) are lanes 0 to 2's, in one step of their own.
template <uint32_t kLanes>
__global__ void __launch_bounds__(32 * kRunWarps, kRunCtas)
    lines_decompress_one_kernel(const __grid_constant__ LineRun R, const AxisEntry *__restrict__ ent,
                                const int64_t *__restrict__ t_int, const int32_t *__restrict__ qb, float *__restrict__ rec,
                                uint32_t *err_word) {
    extern __shared__ __align__(16) uint32_t run_smem[];
    constexpr uint32_t kPer = 32 / kLanes;
    const uint32_t groups = blockDim.x / kLanes, group = threadIdx.x / kLanes, lane = threadIdx.x & 31,
                   sub = threadIdx.x & (kLanes - 1);
    float *s = reinterpret_cast<float *>(run_smem + group * R.line_words);
    float *ts = s + R.line_words - R.rounds;
    const uint32_t step = gridDim.x * groups;
    for (uint32_t at = blockIdx.x * groups + group; at - group % kPer < R.lines; at += step) {
        const bool real = at < R.lines;  // a group past the last line works on that one and stores nothing
        const RunLine l = run_line(R, ent, rec, real ? at : R.lines - 1);
        auto end_target = [&](uint32_t r) { return sub == 0 ? 0 : R.r[r].cubics + sub; };  // lanes 0 to 2
        auto load = [&](const LineQBs &L, uint32_t o) {
            if (o < L.limit) return __ldg(L.q + o);
            atomicOr(err_word, 4u);
            return 0;
        };
        auto load_ends = [&](LineQBs &L, uint32_t r) {
            L.x += L.u * R.r[r].count * L.w;
            const uint32_t i = end_target(r);
            return sub < 3 && i < R.r[r].count ? load(L, i * L.w + L.x) : 0;
        };
        auto load_inner = [&](const LineQBs &L, uint32_t r, uint32_t k, int32_t (&q)[kRunAhead]) {
            const uint32_t cubics = R.r[r].cubics;
#pragma unroll
            for (uint32_t j = 0; j < kRunAhead; j++) {
                if (k + kLanes * j >= cubics) break;
                const uint32_t i = k + kLanes * j + sub;
                q[j] = i < cubics ? load(L, (i + 1) * L.w + L.x) : 0;
            }
        };
        int32_t q[kRunAhead], qe;
        LineQBs L = line_qbs(R.r[0], l, qb);
        qe = load_ends(L, 0);
        load_inner(L, 0, 0, q);
        for (uint32_t k = sub; k < R.known; k += kLanes) s[padded(k * R.step)] = l.g[k * R.step];
        for (uint32_t r = sub; r < R.rounds; r += kLanes) ts[r] = run_t(R, t_int, l.blk, r);
        __syncwarp();
        for (uint32_t r = 0; r < R.rounds; r++) {
            const uint32_t hs = R.r[r].hs, cubics = R.r[r].cubics, quintics = R.r[r].quintics;
            const double eb2 = R.r[r].eb2, td = (double)ts[r], c1 = __dsub_rn(0.25, td), c2 = __dadd_rn(0.25, td);
            const uint32_t ie = end_target(r);
            const int32_t q_end = qe;
            // Inner targets, from 1: addresses of the target and its neighbours.
            const uint32_t i0 = hs * (2 * sub + 3), move = 2 * hs * kLanes / 32 * 33;
            const float *a3 = s + padded(i0 - 3 * hs), *a1 = s + padded(i0 - hs), *b1 = s + padded(i0 + hs),
                        *b3 = s + padded(i0 + 3 * hs);
            float *c = s + padded(i0);
            uint32_t k = 0;
            do {
                int32_t next[kRunAhead];
                if (k + kLanes * kRunAhead < cubics) {
                    load_inner(L, r, k + kLanes * kRunAhead, next);
                } else if (r + 1 < R.rounds) {
                    L = line_qbs(R.r[r + 1], l, qb);
                    qe = load_ends(L, r + 1);
                    load_inner(L, r + 1, 0, next);
                }
#pragma unroll
                for (uint32_t j = 0; j < kRunAhead; j++) {
                    if (k + kLanes * j >= cubics) break;
                    const uint32_t i = k + kLanes * j + sub;
                    if (i < cubics) {
                        float pred;
                        if (i - 1 < quintics) {
                            const uint32_t ii = hs * (2 * i + 3);
                            const StencilIn v{*a1, *b1, *a3, *b3, s[padded(ii - 5 * hs)], s[padded(ii + 5 * hs)]};
                            pred = predict_loaded(v, kStencilQuintic, 0.0f);
                        } else {
                            pred = cubic(*a3, *a1, *b1, *b3, c1, c2);
                        }
                        *c = __double2float_rn(__fma_rn(-(double)q[j], eb2, (double)pred));
                    }
                    a3 += move;
                    a1 += move;
                    b1 += move;
                    b3 += move;
                    c += move;
                }
#pragma unroll
                for (uint32_t j = 0; j < kRunAhead; j++) q[j] = next[j];
                k += kLanes * kRunAhead;
            } while (k < cubics);
            if (sub < 3 && ie < R.r[r].count) {
                const uint32_t ii = hs * (2 * ie + 1);
                const float pred = predict_edge(s, ii, hs, stencil_case(ii, hs, R.n2, false));
                s[padded(ii)] = __double2float_rn(__fma_rn(-(double)q_end, eb2, (double)pred));
            }
            __syncwarp();
        }
        // The warp stores its lines one after another, whole sectors at a time.
        const uint32_t hs = R.r[R.rounds - 1].hs;
        for (uint32_t m = 0; m < kPer; m++) {
            float *g = reinterpret_cast<float *>(__shfl_sync(0xffffffffu, (unsigned long long)l.g, m * kLanes));
            if (!__shfl_sync(0xffffffffu, real, m * kLanes)) continue;
            const float *line = s + ((int)m - (int)(lane / kLanes)) * (int)R.line_words;
            for (uint32_t i = lane * hs; i < R.n2; i += 32 * hs) g[i] = line[padded(i)];
        }
        __syncwarp();
    }
}

// ---------------------------------------------------------------------------------------------
// Compression.

// Samples of a block read from its column's lines in shared memory (the original values from
// global memory). The positions are those of the per-round fast kernel along axis 2.
struct LineSrc {
    fastsel::FastSampleGeo sg;
    const float *lines;
    const float *orig;
    uint64_t n1;
    uint32_t n2, lo0, lo1, nl1, hs;
    float neg;
    __device__ __forceinline__ void keys(uint32_t s, float &af, float &bf, bool &nz) const {
        using namespace fastsel;
        const uint32_t k0 = div_small(s, sg.c12);
        const uint32_t r = s - k0 * sg.c12.d;
        const uint32_t k1 = div_small(r, sg.c2);
        const uint32_t k2 = r - k1 * sg.cnt2;
        const uint32_t i0 = (uint32_t)(sg.lo[0] + k0 * sg.step[0]), i1 = (uint32_t)(sg.lo[1] + k1 * sg.step[1]);
        const uint32_t x = (uint32_t)(sg.lo[2] + k2 * sg.step[2]);
        const float *ln = lines + ((i0 - lo0) * nl1 + (i1 - lo1)) * n2;
        keys_of(ln[x - hs], ln[x - 3 * hs], ln[x + hs], ln[x + 3 * hs], orig[((uint64_t)i0 * n1 + i1) * n2 + x], neg, af, bf,
                nz);
    }
};

struct CompShared {
    fastsel::GroupShared gs;
    float t[kMaxColumnBlocks];  // this round's t per block of the column
};

// Per column, from its first round (or its resume entry) to the last round: coefficient selection
// of each block (certified fast path, fastsel::fast_group) and the round's targets, all on the
// lines in shared memory. A block whose choice needs the exact path stops its column at that round:
// the lines go back to rec, the block is listed for the exact path (bail_blocks + round * nblocks,
// bail_count[round]) and the column for resumption (resume_out: column, round). A resumed column
// starts with the t of its first round already chosen (tval) for each of its blocks.
__global__ void __launch_bounds__(fastsel::kThreads, 6)
    lines_compress_kernel(FieldGeom fg, const RoundGeom *__restrict__ rounds, const AxisEntry *__restrict__ ent,
                          const uint64_t *__restrict__ qoff, const ClassInfo *__restrict__ classes,
                          const float *__restrict__ orig, float *__restrict__ rec, const float *__restrict__ log2arena,
                          float R2, float t_default, float *__restrict__ tval, int64_t *__restrict__ t_int,
                          uint32_t *__restrict__ fb_count, int32_t *__restrict__ qb, int32_t *__restrict__ qb_range,
                          const uint32_t *__restrict__ overrides, uint32_t n_overrides, uint32_t *__restrict__ why,
                          const uint32_t *__restrict__ resume_in, uint32_t n_resume, uint32_t *__restrict__ bail_blocks,
                          uint32_t *__restrict__ bail_count, uint32_t *__restrict__ resume_out,
                          uint32_t *__restrict__ resume_count, uint32_t set, uint32_t *err_word) {
    using namespace fastsel;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    CompShared &cs = *reinterpret_cast<CompShared *>(smem_raw);
    float *sl = reinterpret_cast<float *>(smem_raw + align16(sizeof(CompShared)));
    const uint32_t tid = threadIdx.x;
    const uint32_t nb0 = (uint32_t)fg.block_num[0], nb1 = (uint32_t)fg.block_num[1], nb2 = (uint32_t)fg.block_num[2];
    const uint64_t nblocks = (uint64_t)nb0 * nb1 * nb2;
    const uint32_t n2 = (uint32_t)fg.n[2], L = fg.layer_num;
    const uint32_t items = resume_in ? n_resume : column_count(set, nb0, nb1);
    for (int i = tid; i < 5 * kWinWords; i += kThreads) (&cs.gs.hist[0][0])[i] = 0;
    for (uint32_t it = blockIdx.x; it < items; it += gridDim.x) {
        uint32_t b0, b1;
        if (resume_in) column_at(kColumnsAll, resume_in[2 * it], nb1, b0, b1);  // entries hold column indices
        else column_at(set, it, nb1, b0, b1);
        const uint32_t c = b0 * nb1 + b1;
        const uint32_t start = resume_in ? resume_in[2 * it + 1] : 0;
        const Column col = column_of(fg, b0, b1);
        const uint32_t nl = col.nl0 * col.nl1;
        __syncthreads();
        load_lines(fg, col, rec, sl);
        __syncthreads();
        bool bailed = false;
        for (uint32_t l = start; l < L; l++) {
            const RoundGeom &rg = rounds[l];
            const ClassInfo *cls = classes + 27 * l;
            // ---- Coefficient selection for each block of the column (compress.tpp:91-144).
            for (uint32_t b2 = 0; b2 < nb2; b2++) {
                const uint64_t g = ((uint64_t)b0 * nb1 + b1) * nb2 + b2;
                float t = 0.0f;
                if (resume_in && l == start) {
                    t = tval[g];  // settled before this launch
                } else {
                    const int ccls = (class_of(b0, nb0) * 3 + class_of(b1, nb1)) * 3 + class_of(b2, nb2);
                    const ClassInfo ci = cls[ccls];
                    bool forced = false;
                    float forced_t = 0.0f;
                    for (uint32_t i = 0; i < n_overrides; i++)
                        if (overrides[3 * i] == (uint32_t)g && overrides[3 * i + 1] == l) {
                            forced = true;
                            forced_t = __uint_as_float(overrides[3 * i + 2]);
                        }
                    uint32_t code = kFastDecided;
                    if (ci.fallback || ci.n == 0 || forced) {
                        t = forced ? forced_t : t_default;
                        if (!forced && tid == 0) atomicAdd(fb_count, 1u);
                    } else if (ci.n > 0xffffu) {  // a bin count could overflow its 16-bit half word
                        code = kFastHandoff;
                        if (tid == 0) atomicAdd(&why[0], 1u);
                    } else {
                        const uint64_t bb[3] = {b0, b1, b2};
                        FastSampleGeo sg;
                        uint32_t cnt[3];
                        for (int a = 0; a < 3; a++) {
                            uint64_t lo = bb[a] * fg.block_shape[a];
                            uint64_t hi = min((bb[a] + 1) * fg.block_shape[a] + 1, fg.n[a]);
                            if (a != 2 && lo != 0) lo += rg.stride[a];
                            if (a == 2) {
                                lo += 3 * rg.stride[a] / 2;
                                hi -= 3 * rg.stride[a] / 2;
                            }
                            sg.lo[a] = lo;
                            sg.step[a] = rg.stride[a] * ci.ss;
                            cnt[a] = (uint32_t)((hi - lo + sg.step[a] - 1) / sg.step[a]);
                        }
                        sg.cnt2 = cnt[2];
                        sg.c2 = small_div(cnt[2]);
                        sg.c12 = small_div(cnt[1] * cnt[2]);
                        const LineSrc src{sg, sl, orig, fg.n[1], n2, col.lo0, col.lo1, col.nl1, (uint32_t)rg.hs,
                                          rg.neg_2_stat_eb};
                        code = fast_group(cs.gs, src, ci.n, rg, log2arena + ci.log2_off, R2, why, t);
                    }
                    if (code == kFastHandoff) {
                        if (tid == 0) bail_blocks[(uint64_t)l * nblocks + atomicAdd(&bail_count[l], 1u)] = (uint32_t)g;
                        bailed = true;
                    } else if (tid == 0) {
                        tval[g] = t;
                        t_int[g * L + l] = lround_f(__fmul_rn(t, (float)fg.t_precision));
                    }
                }
                if (tid == 0) cs.t[b2] = t;
            }
            __syncthreads();
            if (bailed) {
                // The rest of the column waits for the exact path: its state goes back to memory.
                store_lines(fg, col, sl, rec);
                if (tid == 0) {
                    const uint32_t k = atomicAdd(resume_count, 1u);
                    resume_out[2 * k] = c;
                    resume_out[2 * k + 1] = l;
                }
                break;
            }
            // ---- The round's targets (compress.tpp:35-37 as emitted along axis 2: divide).
            const double ebd = (double)rg.eb, eb2 = __dadd_rn(ebd, ebd), rinv = __ddiv_rn(1.0, ebd);
            const uint32_t T2 = (uint32_t)rg.tcount[2], hs = (uint32_t)rg.hs;
            const AxisEntry *e0t = ent + rg.ent_off[0], *e1t = ent + rg.ent_off[1], *e2t = ent + rg.ent_off[2];
            int32_t *qbl = qb + qoff[l + 1];
            int32_t lo = INT32_MAX, hi = INT32_MIN;
            const uint32_t work = nl * T2;
#pragma unroll 4
            for (uint32_t w = tid; w < work; w += blockDim.x) {
                const uint32_t line = w / T2, k = w - line * T2;
                const uint32_t r0 = line / col.nl1, i0 = col.lo0 + r0, i1 = col.lo1 + (line - r0 * col.nl1);
                const AxisEntry e0 = load_entry(e0t + i0), e1 = load_entry(e1t + i1), e2 = load_entry(e2t + k);
                const uint64_t qi = qb_index(rg, e0, e1, e2);
                if (qi >= rg.qb_total || e2.bb >= kMaxColumnBlocks) {
                    atomicOr(err_word, 4u);
                    continue;
                }
                float *ln = sl + line * n2;
                const float t = e2.stencil == kStencilCubic ? cs.t[e2.bb] : 0.0f;
                const float pred = predict_case(ln, e2.ii, hs, e2.stencil, t);
                const double pd = (double)pred;
                const double diff = __dsub_rn(pd, (double)orig[((uint64_t)i0 * fg.n[1] + i1) * n2 + e2.ii]);
                const int32_t v = (int32_t)lround_d(quot_for_lround(__dmul_rn(diff, 0.5), ebd, rinv));
                qbl[qi] = v;
                ln[e2.ii] = __double2float_rn(__fma_rn(-(double)v, eb2, pd));
                lo = min(lo, v);
                hi = max(hi, v);
            }
            for (int o = 16; o > 0; o >>= 1) {
                lo = min(lo, __shfl_xor_sync(0xffffffffu, lo, o));
                hi = max(hi, __shfl_xor_sync(0xffffffffu, hi, o));
            }
            if ((tid & 31) == 0 && lo <= hi) {
                atomicMin(&qb_range[2 * (l + 1)], lo);
                atomicMax(&qb_range[2 * (l + 1) + 1], hi);
            }
            __syncthreads();
        }
        if (!bailed) store_lines(fg, col, sl, rec);
    }
}

}  // namespace

uint32_t lines_smem_limit() { return 96 * 1024; }

// The launch's CTAs: the most warps on an SM, `per` lines each; of equals the wider CTA (fewer copies
// of the table), unless that leaves SMs without lines.
struct RunShape {
    uint32_t warps, ctas;  // of a CTA, of an SM
};
static RunShape run_shape(uint64_t tab_words, uint64_t line_words, uint32_t per, uint64_t lines) {
    RunShape s{1, 0};
    for (uint32_t w = kRunWarps; w >= 1; w /= 2) {
        const uint64_t bytes = 4 * (tab_words + w * per * line_words);
        if (bytes > kRunSmem) continue;
        const uint32_t c = (uint32_t)std::min<uint64_t>(kRunWarps * kRunCtas / w, kRunSm / (bytes + 1024));
        if (c * w > s.ctas * s.warps || (w >= 4 && lines < 148ull * 2 * w * per)) s = {w, c};
    }
    return s;
}

// Where a run goes line by line. A line costs its rounds' steps whatever its length, 1.1 ns in all at
// five rounds, so short lines are better off round by round, where a step holds several lines
// (512x512xn: n = 32 140 against 240 us, n = 64 260 against 298; 256x256x512 in nine rounds 510 against
// 185), unless they are so few that launches are what the rounds cost (24x20x17: 39 against 11 us). With
// a table, a CTA must also fit as often as its registers allow: with half of the warps the rounds are
// as fast (64x64x4096 in four rounds: 203 against 238 us; 256x256x512 in three: 362 against 199).
constexpr uint64_t kRunTargets = 96, kRunFewLines = 4096;

uint32_t lines_run_length(const FieldGeom &fg, const RoundGeom *rounds, uint32_t count) {
    uint32_t len = 0, used = 0;
    uint64_t targets = 0, lines = 0;
    for (; len < count && rounds[len].dir == 2; len++) {
        if (!rounds[len].targets) continue;
        used++;
        targets += rounds[len].tcount[2];
        lines = rounds[len].tcount[0] * rounds[len].tcount[1];
    }
    if (used < 2 || used > kRunRounds || (targets < kRunTargets && lines > kRunFewLines)) return 0;
    if (fg.origin[0] || fg.origin[1] || fg.origin[2] || fg.n[2] >= 65536) return 0;  // 16-bit entries
    // 32-bit offsets within a row of blocks' QBs.
    const uint64_t c0 = std::min(fg.block_shape[0] + 1, fg.n[0]), c1 = std::min(fg.block_shape[1] + 1, fg.n[1]);
    if (c0 * c1 >= (1ull << 31) / fg.n[2]) return 0;
    const bool one = fg.block_num[2] == 1;
    const RunShape s = run_shape(one ? 0 : 2 * targets, fg.n[2] + fg.n[2] / 32 + 1 + fg.block_num[2] * used, 1, lines);
    return s.ctas * s.warps >= (one ? 1 : kRunWarps * kRunCtas) ? len : 0;
}

cudaError_t launch_lines_decompress(const FieldGeom &fg, const RoundGeom *rounds, uint32_t len, uint32_t l0, const AxisEntry *ent,
                                    const uint64_t *qoff, const int64_t *t_int, const int32_t *qb, float *rec, uint32_t *err,
                                    cudaStream_t st) {
    LineRun R{};
    R.n1n2 = fg.n[1] * fg.n[2];
    R.n2 = (uint32_t)fg.n[2];
    for (uint32_t l = 0; l < len; l++) {
        const RoundGeom &rg = rounds[l];
        if (rg.targets == 0) continue;
        if (R.rounds == 0) {
            R.ent0 = rg.ent_off[0];
            R.ent1 = rg.ent_off[1];
            R.total1 = rg.total[1];
            R.lines = (uint32_t)(rg.tcount[0] * rg.tcount[1]);
            R.T1 = (uint32_t)rg.tcount[1];
            R.step = (uint32_t)(2 * rg.hs);
            R.known = (R.n2 + R.step - 1) / R.step;
        }
        RunRound &m = R.r[R.rounds++];
        m.eb2 = (double)rg.eb + (double)rg.eb;
        m.qoff = qoff[l0 + l + 1];
        m.qb_total = rg.qb_total;
        m.ent2 = rg.ent_off[2];
        m.hs = (uint32_t)rg.hs;
        m.count = (uint32_t)rg.tcount[2];
        m.first = R.targets;
        m.total2 = (uint32_t)rg.total[2];
        m.order = (uint32_t)rg.order;
        m.l = l0 + l;
        // Targets i >= 1 with (2 i + 1) hs + 3 hs < n2, and i >= 2 with (2 i + 1) hs + 5 hs < n2.
        auto below = [&](uint64_t reach, uint32_t from) {
            const uint64_t end = reach < R.n2 ? (R.n2 - reach + 2 * rg.hs - 1) / (2 * rg.hs) : 0;
            return end > from ? (uint32_t)(end - from) : 0u;
        };
        m.cubics = below(4 * rg.hs, 1);
        m.quintics = fg.quintic ? below(6 * rg.hs, 2) : 0;
        R.targets += m.count;
    }
    R.nb1 = (uint32_t)fg.block_num[1];
    R.nb2 = (uint32_t)fg.block_num[2];
    R.layers = fg.layer_num;
    R.tp = (float)fg.t_precision;
    const bool one = R.nb2 == 1;
    R.tab_words = one ? 0 : 2 * R.targets;
    R.line_words = R.n2 + R.n2 / 32 + 1 + R.nb2 * R.rounds;
    RunShape sh = run_shape(R.tab_words, R.line_words, 1, R.lines);
    uint32_t per = 1;
    if (one && R.lines >= 148 * 2 * 16) {
        // Two lines a warp where that leaves the SMs their warps.
        const RunShape two = run_shape(R.tab_words, R.line_words, 2, R.lines);
        if (two.warps * two.ctas == kRunWarps * kRunCtas) {
            sh = two;
            per = 2;
        }
    }
    const uint32_t warps = sh.warps, ctas = sh.ctas;
    const uint32_t smem = 4 * (R.tab_words + warps * per * R.line_words);
    auto kernel = !one ? lines_decompress_kernel : per == 2 ? lines_decompress_one_kernel<16> : lines_decompress_one_kernel<32>;
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kRunSmem);
    if (e != cudaSuccess) return e;
    const uint32_t grid = std::min((R.lines + warps * per - 1) / (warps * per), 148 * ctas);
    kernel<<<grid, 32 * warps, smem, st>>>(R, ent, t_int, qb, rec, err);
    count_launch();
    return cudaGetLastError();
}

cudaError_t launch_lines_compress(const FieldGeom &fg, const RoundGeom *rounds, const AxisEntry *ent, const uint64_t *qoff,
                                  const ClassInfo *classes, const float *orig, float *rec, const float *log2arena, float R2,
                                  float t_default, float *tval, int64_t *t_int, uint32_t *fb_count, int32_t *qb,
                                  int32_t *qb_range, const uint32_t *overrides, uint32_t n_overrides, uint32_t *why,
                                  const uint32_t *resume_in, uint32_t n_resume, uint32_t *bail_blocks, uint32_t *bail_count,
                                  uint32_t *resume_out, uint32_t *resume_count, uint32_t *err, uint32_t set,
                                  uint32_t line_bytes, cudaStream_t st) {
    const uint32_t items =
        resume_in ? n_resume : column_count(set, (uint32_t)fg.block_num[0], (uint32_t)fg.block_num[1]);
    if (items == 0) return cudaSuccess;
    if (fg.block_num[2] > kMaxColumnBlocks) return cudaErrorInvalidValue;
    const uint32_t smem = (uint32_t)(align16(sizeof(CompShared)) + line_bytes);
    cudaError_t e = cudaFuncSetAttribute(lines_compress_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)(align16(sizeof(CompShared)) + lines_smem_limit()));
    if (e != cudaSuccess) return e;
    int per_sm = 0;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, lines_compress_kernel, fastsel::kThreads, smem);
    if (e != cudaSuccess) return e;
    const uint64_t cap = 148ull * (per_sm > 0 ? per_sm : 1);
    lines_compress_kernel<<<(unsigned)(items < cap ? items : cap), fastsel::kThreads, smem, st>>>(
        fg, rounds, ent, qoff, classes, orig, rec, log2arena, R2, t_default, tval, t_int, fb_count, qb, qb_range, overrides,
        n_overrides, why, resume_in, n_resume, bail_blocks, bail_count, resume_out, resume_count, set, err);
    count_launch();
    return cudaGetLastError();
}

}  // namespace asz
