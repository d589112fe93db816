// Host side of the prediction sweep (asz_sweep in include/asz_b200.h): the GPU form of the
// reference's study tool c_codes/s2_many_prediction.cpp.
//
// Per relative error bound, the predictor's coefficients go through in batches sized to the
// device memory: one launch predicts and quantises every target for every coefficient of the
// batch (k_sweep.cu); histograms and first positions of the QB symbols follow on the device; the
// host builds each stream's Huffman code and H1; the streams are encoded, copied out and compressed
// one behind the other: while a stream is encoded the one before it crosses to the host, where
// libzstd level 3 takes those that are there, framed as huffman_encoder_class<int64_t>::save + encode,
// on the worker threads (lossless_encode_and_write_csv, :400-440).
//
// Host floating point restates the reference's forms under its -Ofast build and is compiled with
// -ffp-contract=off: the grid constants (a division in a loop becomes a product with the rounded
// reciprocal), H1 with p = freq * (1 / size) and H1 -= p log2 p fused, and the final figures with
// psnr = 10 log10((range^2 / mse_sum) * size).
#include <cuda_runtime.h>

#include <algorithm>
#include <chrono>
#include <climits>
#include <cmath>
#include <cstring>
#include <memory>
#include <mutex>
#include <string>
#include <unordered_map>
#include <utility>
#include <vector>

#include "../../../include/asz_b200.h"
#include "../launch.h"
#include "buffers.h"
#include "huffman_host.h"
#include "internal.h"
#include "zstd_api.h"

using namespace asz;
using asz::host::DevBuf;
using asz::host::PinnedBuf;

namespace {

using u64 = uint64_t;
using clk = std::chrono::steady_clock;

// Per stream in work at a time: the zstd output and a zstd context, kept across rows and calls so that
// their pages are mapped once (first writes to fresh pages cost as much as zstd).
struct WorkerScratch {
    std::vector<uint8_t> z;
    ZSTD_CCtx *cc = nullptr;
};

// Streams of fewer symbols are encoded and copied out together: below, a launch and a copy each cost
// more than the wait for the others.
constexpr u64 kGroupSymbols = 1ull << 22;

struct SweepState {
    DevBuf coef, qb, part, sums, mm, hist, first, tab, pay, enc;
    PinnedBuf small, counts, payload;
    std::vector<std::unique_ptr<WorkerScratch>> ws;
    cudaStream_t copies = nullptr;   // payloads on their way to the host
    std::vector<cudaEvent_t> events;  // two a group of streams: encoded, and there
    // Makes the copies' stream and at least n events.
    cudaError_t reserve_events(size_t n) {
        cudaError_t e = cudaSuccess;
        if (!copies) e = cudaStreamCreateWithFlags(&copies, cudaStreamNonBlocking);
        while (e == cudaSuccess && events.size() < n) {
            cudaEvent_t ev = nullptr;
            e = cudaEventCreateWithFlags(&ev, cudaEventDisableTiming);
            if (e == cudaSuccess) events.push_back(ev);
        }
        return e;
    }
};

// Whatever way a call returns, its copies no longer run: the buffers they use are the next call's.
struct CopiesEnd {
    cudaStream_t s;
    ~CopiesEnd() { cudaStreamSynchronize(s); }
};

struct Predictor {
    int kind = -1;  // 0: 1d4r, 1: 2d4r, 2: 1d6r
    int axis[2] = {-1, -1};
    int order = -1;
};

// Predictor names of s2_many_prediction.cpp:538-552: "<stencil>_xx<order>".
bool parse_predictor(const char *name, Predictor &p, std::string &err) {
    const std::string s = name ? name : "";
    err = "unknown predictor " + s;
    auto ax = [&](size_t i) { return i < s.size() && s[i] >= '0' && s[i] <= '2' ? s[i] - '0' : -1; };
    size_t i = 4;
    if (s.rfind("1d4r", 0) == 0) p.kind = 0;
    else if (s.rfind("2d4r", 0) == 0) p.kind = 1;
    else if (s.rfind("1d6r", 0) == 0) p.kind = 2;
    else return false;
    p.axis[0] = ax(i++);
    if (p.kind == 1) p.axis[1] = ax(i++);
    if (s.size() != i + 4 || s.compare(i, 3, "_xx") != 0) return false;
    p.order = ax(i + 3);
    if (p.axis[0] < 0 || p.order < 0) return false;
    if (p.kind == 1 && !(p.axis[1] > p.axis[0])) return false;
    return true;
}

// The target loops (stride 1). Legacy (s2_many_prediction.cpp:204-397): the two axes other than
// the QB order run outside in increasing order, the order axis inside; a 1D predictor's axis
// covers [m, n - m) every other point (m = 3 for 1D4R, 5 for 1D4R shared1d and for 1D6R), the
// other axes every point; 2D4R's two axes cover [1, n - 1), the third [0, n), every other point
// along axis 0 (pair 01), 1 (pair 02) or 2 (pair 12). Common (:126-149): [5, n - 5) on every
// axis, points with an odd coordinate sum.
bool sweep_geometry(const Predictor &p, const u64 n[3], const std::string &targets, SweepGeom &g) {
    std::memset(&g, 0, sizeof g);
    for (int a = 0; a < 3; a++) g.n[a] = n[a];
    auto dist = [&](int a) { return a == 0 ? n[1] * n[2] : a == 1 ? n[2] : (u64)1; };
    g.dist[0] = dist(p.axis[0]);
    g.dist[1] = p.kind == 1 ? dist(p.axis[1]) : 0;
    g.kind = (uint32_t)p.kind;
    int k = 0;
    for (int a = 0; a < 3; a++)
        if (a != p.order) g.axis[k++] = (uint32_t)a;
    g.axis[2] = (uint32_t)p.order;
    g.line_per_thread = p.order != 2;
    if (targets == "common") {
        g.common = 1;
        for (int l = 0; l < 3; l++) {
            const u64 m = n[g.axis[l]];
            g.start[l] = 5;
            g.step[l] = 1;
            g.count[l] = m > 10 ? m - 10 : 0;
        }
        const u64 c = g.count[2];
        g.inner_odd = (c + 1) / 2;  // 5, 7, ... below n - 5
        g.inner_even = c / 2;       // 6, 8, ...
        g.lines = g.count[0] * g.count[1];
        g.per_line = std::max(g.inner_odd, g.inner_even);
        const u64 L0 = g.count[0], L1 = g.count[1];
        const u64 q0 = (L0 + 1) / 2 * ((L1 + 1) / 2) + L0 / 2 * (L1 / 2);
        g.targets = q0 * g.inner_odd + (L0 * L1 - q0) * g.inner_even;
        return true;
    }
    const bool shared1d = targets == "shared1d";
    const int doubled = p.kind == 1 ? (p.axis[0] == 0 && p.axis[1] == 1 ? 0 : p.axis[0] == 0 ? 1 : 2) : p.axis[0];
    for (int l = 0; l < 3; l++) {
        const int a = (int)g.axis[l];
        const bool on = a == p.axis[0] || (p.kind == 1 && a == p.axis[1]);
        const u64 m = p.kind == 1 ? 1 : p.kind == 2 ? 5 : (shared1d ? 5 : 3);
        const u64 lo = on ? m : 0, hi = on ? (n[a] > m ? n[a] - m : 0) : n[a];
        g.start[l] = lo;
        g.step[l] = a == doubled ? 2 : 1;
        g.count[l] = hi > lo ? (hi - lo + g.step[l] - 1) / g.step[l] : 0;
    }
    g.lines = g.count[0] * g.count[1];
    g.per_line = g.count[2];
    g.targets = g.lines * g.per_line;
    return true;
}

// Coefficient grids (s2_many_prediction.cpp:89-124, :199-201, :264-266).
bool coef_grid(const Predictor &p, const std::string &six, std::vector<std::pair<double, double>> &g, std::string &err) {
    g.clear();
    if (p.kind == 0) {
        for (int i = 0; i <= 12; i++) g.push_back({(double)((float)i / 32.0f), 0.0});
        return true;
    }
    if (p.kind == 1) {  // i / 24 in float, as i times the float reciprocal of 24
        for (int i = -6; i <= 6; i++) g.push_back({(double)((float)i * (1.0f / 24.0f)), 0.0});
        return true;
    }
    if (six == "transition") {
        g.push_back({1.0 / 6, 1.0 / 6});
        g.push_back({3.0 / 256, -25.0 / 256});
        for (int i = 0; i <= 12; i++) g.push_back({0.0, (8 - i) / 32.0});
        g.push_back({137.0 / 1536, 53.0 / 1536});
        for (int i = 0; i <= 12; i++) {
            g.push_back({1.0 / 12, (40 - 3 * i) * (1.0 / 192.0)});
            g.push_back({3.0 / 512, (39 - 8 * i) / 512.0});
        }
        return true;
    }
    if (six != "legacy" && six != "augmented") {
        err = "six-reference grid must be legacy, augmented or transition";
        return false;
    }
    static const int k1[] = {0, 11, 22, 31, 41}, k2[] = {0, 113, 248, 341, 453, 567, 680, 793};
    for (int a : k1)
        for (int b : k2) g.push_back({1.0 / 6 - (double)((float)a / 186.0f), 1.0 / 6 - (double)((float)b / 1488.0f)});
    if (six == "augmented") {
        std::vector<std::pair<double, double>> exact = {{3.0 / 256, -25.0 / 256}};
        for (int i = 0; i <= 12; i++) exact.push_back({0.0, (8 - i) / 32.0});
        for (const auto &c : exact) {
            auto it = std::find_if(g.begin(), g.end(), [&](const std::pair<double, double> &q) {
                return std::fabs(q.first - c.first) < 1e-7 && std::fabs(q.second - c.second) < 1e-7;
            });
            if (it == g.end()) g.push_back(c);
            else *it = c;
        }
    }
    return true;
}

SweepCoef make_coef(const Predictor &p, double c0, double c1) {
    SweepCoef c{};
    c.c0 = c0;
    c.c1 = c1;
    c.w = 0.5 - (c0 + c1);
    if (p.kind == 0) {
        c.lo = 0.25 - c0;
        c.hi = 0.25 + c0;
    } else if (p.kind == 1) {
        c.hi = 0.25 + c0;
        c.lo = 0.25 - c0;
    }
    return c;
}

// get_H1 (c_codes/get_H.hpp): the symbols enter the map in order of first occurrence, which
// gives the reference's iteration order; p = freq * (1 / size); H1 -= p log2 p fused.
double h1_of(const u64 *hist, const u64 *first, u64 range, int64_t lo, u64 size) {
    std::vector<std::pair<u64, int64_t>> seen;
    for (u64 i = 0; i < range; i++)
        if (hist[i]) seen.push_back({first[i], lo + (int64_t)i});
    std::sort(seen.begin(), seen.end());
    std::unordered_map<int64_t, u64> m;
    for (const auto &s : seen) m.emplace(s.second, hist[(u64)(s.second - lo)]);
    const double inv = 1.0 / (double)size;
    double h1 = 0;
    for (const auto &kv : m) {
        const double pr = (double)kv.second * inv;
        h1 = std::fma(-pr, std::log2(pr), h1);
    }
    return h1;
}

void finish_row(asz_sweep_row &r, double range) {  // s2_many_prediction.cpp:423-430
    const double S = (double)r.samples;
    r.cr = (double)(r.samples * sizeof(float)) / (double)r.zstd_bytes;
    r.br = (8 * sizeof(float)) / r.cr;
    r.h1_cr = (8 * sizeof(float)) / r.h1;
    r.rmse = std::sqrt(r.rmse_sum / S);
    r.mae = r.mae_sum / S;
    r.psnr = 10 * std::log10((range * range / r.mse_sum) * S);
}

constexpr u64 kMaxSymbolRange = 1ull << 27;

}  // namespace

#define CK(call)                                                                                         \
    do {                                                                                                 \
        cudaError_t e_ = (call);                                                                         \
        if (e_ != cudaSuccess)                                                                           \
            return host::ctx_fail(ctx, ASZ_E_CUDA, std::string(#call) + ": " + cudaGetErrorString(e_)); \
    } while (0)

namespace asz::host {
void sweep_release(void *state) {
    SweepState *s = (SweepState *)state;
    if (!s) return;
    for (DevBuf *b : {&s->coef, &s->qb, &s->part, &s->sums, &s->mm, &s->hist, &s->first, &s->tab, &s->pay, &s->enc})
        b->release();
    s->small.release();
    s->counts.release();
    s->payload.release();
    for (auto &w : s->ws)
        if (w->cc) ZSTD_freeCCtx(w->cc);
    for (cudaEvent_t e : s->events) cudaEventDestroy(e);
    if (s->copies) cudaStreamDestroy(s->copies);
    delete s;
}
}  // namespace asz::host

extern "C" int asz_sweep_coefs(const char *predictor, const char *six_grid, double *c0, double *c1, uint64_t cap,
                               uint64_t *count) {
    Predictor p;
    std::string err;
    std::vector<std::pair<double, double>> g;
    if (!parse_predictor(predictor, p, err) || !coef_grid(p, six_grid ? six_grid : "legacy", g, err)) return ASZ_E_ARG;
    for (u64 i = 0; i < g.size() && i < cap; i++) {
        if (c0) c0[i] = g[i].first;
        if (c1) c1[i] = g[i].second;
    }
    if (count) *count = g.size();
    return ASZ_OK;
}

extern "C" int asz_sweep_targets(const uint64_t dims[3], const char *predictor, const char *targets, uint64_t *coords,
                                 uint64_t cap, uint64_t *count) {
    Predictor p;
    std::string err;
    const std::string tg = targets ? targets : "legacy";
    if (!dims || !count || !parse_predictor(predictor, p, err)) return ASZ_E_ARG;
    if (tg != "legacy" && tg != "shared1d" && tg != "common") return ASZ_E_ARG;
    SweepGeom g;
    sweep_geometry(p, dims, tg, g);
    *count = g.targets;
    if (!coords) return ASZ_OK;
    if (cap < g.targets) return ASZ_E_ARG;
    u64 visited = 0;
    for (u64 it = 0; it < g.lines * g.per_line; it++) {
        u64 i[3], j;
        if (!sweep_target(g, it, i, j)) continue;
        if (j >= g.targets) return ASZ_E_DEVICE;
        for (int a = 0; a < 3; a++) coords[3 * j + a] = i[a];
        visited++;
    }
    return visited == g.targets ? ASZ_OK : ASZ_E_DEVICE;
}

namespace {

// What the batches of one call share.
struct SweepCall {
    asz_ctx *ctx;
    SweepState &W;
    const SweepGeom &g;
    const float *d_in;
    double range, rel_eb, abs_eb, neg_2_eb;
    const std::vector<std::pair<double, double>> &grid;
    const Predictor &p;
    asz_sweep_row *rows;  // of this error bound
};
constexpr int kWide = INT_MAX;  // a QB does not fit Q

// Coefficients k0 .. k0 + kc - 1 of one error bound, with QBs of type Q.
template <class Q>
int sweep_batch(const SweepCall &S_, u64 k0, u64 kc) {
    asz_ctx *const ctx = S_.ctx;
    SweepState &W = S_.W;
    const u64 S = S_.g.targets;
    auto bad = [&](int code, const std::string &m) { return host::ctx_fail(ctx, code, m); };
    cudaStream_t st = host::ctx_stream(ctx);
    int dev = 0;
    CK(cudaGetDevice(&dev));
    const uint32_t nparts = sweep_predict_grid(S_.g);
    const size_t mm_at = kc * 3 * sizeof(double), ss_at = mm_at + kc * 2 * sizeof(long long);
    CK(W.coef.reserve(kc * sizeof(SweepCoef)));
    CK(W.qb.reserve(kc * S * sizeof(Q)));
    CK(W.part.reserve(kc * nparts * 3 * sizeof(double)));
    CK(W.sums.reserve(ss_at + kc * sizeof(SweepStream)));
    CK(W.small.reserve(kc * (sizeof(SweepCoef) + 3 * sizeof(double) + 2 * sizeof(long long) + sizeof(SweepStream))));
    SweepCoef *h_coef = (SweepCoef *)W.small.p;
    double *h_sums = (double *)(h_coef + kc);
    long long *h_mm = (long long *)(h_sums + 3 * kc);
    SweepStream *h_ss = (SweepStream *)(h_mm + 2 * kc);
    double *d_sums = W.sums.as<double>();
    long long *d_mm = (long long *)(W.sums.as<uint8_t>() + mm_at);
    SweepStream *d_ss = (SweepStream *)(W.sums.as<uint8_t>() + ss_at);
    Q *d_qb = W.qb.as<Q>();
    for (u64 k = 0; k < kc; k++) {
        h_coef[k] = make_coef(S_.p, S_.grid[k0 + k].first, S_.grid[k0 + k].second);
        h_mm[2 * k] = LLONG_MAX;
        h_mm[2 * k + 1] = LLONG_MIN;
    }
    CK(cudaMemcpyAsync(W.coef.p, h_coef, kc * sizeof(SweepCoef), cudaMemcpyHostToDevice, st));
    CK(cudaMemcpyAsync(d_mm, h_mm, kc * 2 * sizeof(long long), cudaMemcpyHostToDevice, st));
    CK(launch_sweep_predict<Q>(S_.d_in, S_.g, W.coef.as<SweepCoef>(), (uint32_t)kc, S_.abs_eb, S_.neg_2_eb, d_qb, S,
                               W.part.as<double>(), d_mm, st));
    CK(launch_sweep_sums(W.part.as<double>(), nparts, (uint32_t)kc, d_sums, st));
    CK(cudaMemcpyAsync(h_sums, d_sums, ss_at, cudaMemcpyDeviceToHost, st));  // the sums and the extremes
    CK(cudaStreamSynchronize(st));
    if (sizeof(Q) == 4)
        for (u64 k = 0; k < kc; k++)
            if (h_mm[2 * k] == LLONG_MIN) return kWide;
    const auto t_enc = clk::now();
    // Histograms and first positions of every stream of the batch.
    std::vector<u64> hoff(kc + 1, 0);
    for (u64 k = 0; k < kc; k++) {
        const u64 r = (u64)(h_mm[2 * k + 1] - h_mm[2 * k]) + 1;
        if (h_mm[2 * k] > h_mm[2 * k + 1] || r > kMaxSymbolRange)
            return bad(ASZ_E_UNSUPPORTED, "QB symbol range exceeds 2^27 values");
        h_ss[k] = SweepStream{h_mm[2 * k], r, hoff[k]};
        hoff[k + 1] = hoff[k] + r;
    }
    const u64 htot = hoff[kc];
    CK(W.hist.reserve(htot * 8));
    CK(W.first.reserve(htot * 8));
    CK(W.counts.reserve(htot * 16));
    CK(cudaMemsetAsync(W.hist.p, 0, htot * 8, st));
    CK(cudaMemsetAsync(W.first.p, 0xff, htot * 8, st));
    CK(cudaMemcpyAsync(d_ss, h_ss, kc * sizeof(SweepStream), cudaMemcpyHostToDevice, st));
    CK(launch_sweep_stats<Q>(d_qb, S, (uint32_t)kc, d_ss, W.hist.as<unsigned long long>(), W.first.as<unsigned long long>(), st));
    u64 *h_hist = (u64 *)W.counts.p, *h_first = h_hist + htot;
    CK(cudaMemcpyAsync(h_hist, W.hist.p, htot * 8, cudaMemcpyDeviceToHost, st));
    CK(cudaMemcpyAsync(h_first, W.first.p, htot * 8, cudaMemcpyDeviceToHost, st));
    CK(cudaStreamSynchronize(st));
    // Codes on the host threads.
    std::vector<HuffCode> code(kc);
    std::vector<double> h1(kc);
    std::vector<std::string> cerr(kc);
    std::vector<char> ok(kc, 1);
    host::ctx_parallel(ctx, kc, [&](u64 k) {
        std::vector<u64> hv(h_hist + hoff[k], h_hist + hoff[k + 1]);
        ok[k] = build_code(hv, h_mm[2 * k], h_mm[2 * k + 1], S, true, code[k], cerr[k]);
    });
    for (u64 k = 0; k < kc; k++)
        if (!ok[k]) return bad(ASZ_E_UNSUPPORTED, cerr[k]);
    // Groups of streams that are encoded in one launch and copied out behind it. A stream's frame in
    // the pinned buffer is its tree and length word (front), then the payload; a stream alone in its
    // group is copied straight there, others together to where the group begins, and from there by
    // the worker.
    struct Group {
        u64 k0, k1, es0, toff0, state0, tiles;
        u64 at;  // in the pinned buffer, of groups of several streams
    };
    std::vector<Group> groups;
    std::vector<EncStream> es;
    std::vector<u64> toff, tab_off(kc, 0), word_off(kc + 1, 0), frame(kc), front(kc), pay(kc), group_of(kc);
    u64 tab_tot = 0, states = 0, host_end = 0;
    for (u64 k = 0; k < kc; k++) {
        tab_off[k] = tab_tot;
        tab_tot += code[k].table.size();
        pay[k] = code[k].maxval == 1 ? 0 : (code[k].bits + 7) / 8;
        word_off[k + 1] = word_off[k] + (pay[k] + 3) / 4;
        front[k] = code[k].save_size() + 8;
        frame[k] = (host_end + front[k] + 63) / 64 * 64 - front[k];  // the payload on a line of its own
        host_end = frame[k] + front[k] + word_off[k + 1] * 4 - word_off[k] * 4;
    }
    CK(W.tab.reserve(std::max<u64>(tab_tot, 1) * sizeof(CodeEntry)));
    CK(W.pay.reserve(std::max<u64>(word_off[kc], 1) * 4));
    for (u64 k = 0; k < kc;) {
        Group G{k, k, es.size(), toff.size(), states, 0, host_end};
        toff.push_back(0);
        do {
            group_of[k] = groups.size();
            if (pay[k]) {
                es.push_back(EncStream{d_qb + k * S, S, h_mm[2 * k], W.tab.as<CodeEntry>() + tab_off[k],
                                       W.pay.as<uint32_t>() + word_off[k]});
                G.tiles += (S + enc_tile<Q>() - 1) / enc_tile<Q>();
                toff.push_back(G.tiles);
            }
            k++;
        } while (k < kc && (k - G.k0) * S < kGroupSymbols);
        G.k1 = k;
        if (G.k1 - G.k0 > 1) host_end += (word_off[G.k1] - word_off[G.k0]) * 4;
        states += G.tiles + 1;
        groups.push_back(G);
    }
    const u64 tab_at = (host_end + 15) / 16 * 16;
    CK(W.payload.reserve(tab_at + tab_tot * sizeof(CodeEntry)));
    CK(W.reserve_events(2 * groups.size()));
    CodeEntry *h_tab = (CodeEntry *)(W.payload.p + tab_at);
    for (u64 k = 0; k < kc; k++) std::memcpy(h_tab + tab_off[k], code[k].table.data(), code[k].table.size() * sizeof(CodeEntry));
    const u64 o_toff = (es.size() * sizeof(EncStream) + 15) / 16 * 16, o_err = o_toff + (toff.size() * 8 + 15) / 16 * 16,
              o_state = o_err + 16, end = o_state + states * 8;
    CK(W.enc.reserve(end));
    uint8_t *eb = W.enc.as<uint8_t>();
    CopiesEnd copies_end{W.copies};
    if (!es.empty()) {
        CK(cudaMemcpyAsync(W.tab.p, h_tab, tab_tot * sizeof(CodeEntry), cudaMemcpyHostToDevice, st));
        CK(cudaMemsetAsync(W.pay.p, 0, word_off[kc] * 4, st));
        CK(cudaMemcpyAsync(eb, es.data(), es.size() * sizeof(EncStream), cudaMemcpyHostToDevice, st));
        CK(cudaMemcpyAsync(eb + o_toff, toff.data(), toff.size() * 8, cudaMemcpyHostToDevice, st));
        CK(cudaMemsetAsync(eb + o_err, 0, end - o_err, st));
    }
    for (u64 i = 0; i < groups.size(); i++) {
        const Group &G = groups[i];
        const u64 es1 = i + 1 < groups.size() ? groups[i + 1].es0 : es.size();
        if (es1 == G.es0) continue;
        CK(launch_encode_tiles<Q>((const EncStream *)eb + G.es0, (uint32_t)(es1 - G.es0), (const u64 *)(eb + o_toff) + G.toff0,
                                  G.tiles, (u64 *)(eb + o_state) + G.state0, (u64 *)(eb + o_err), st));
        CK(cudaEventRecord(W.events[2 * i], st));
        CK(cudaStreamWaitEvent(W.copies, W.events[2 * i], 0));
        uint8_t *to = W.payload.p + (G.k1 - G.k0 > 1 ? G.at : frame[G.k0] + front[G.k0]);
        CK(cudaMemcpyAsync(to, W.pay.as<uint32_t>() + word_off[G.k0], (word_off[G.k1] - word_off[G.k0]) * 4,
                           cudaMemcpyDeviceToHost, W.copies));
        CK(cudaEventRecord(W.events[2 * i + 1], W.copies));
    }
    // Frame each stream (save + encode, huffman.hpp) and compress it with zstd level 3.
    std::vector<u64> zb(kc);
    std::vector<char> zok(kc, 1), there(kc, 1);
    std::mutex idle_mu;
    std::vector<WorkerScratch *> idle;
    for (auto &w : W.ws) idle.push_back(w.get());
    host::ctx_parallel(ctx, kc, [&](u64 k) {
        const HuffCode &c = code[k];
        WorkerScratch *mine;
        {
            std::lock_guard<std::mutex> g(idle_mu);
            if (idle.empty()) {
                W.ws.push_back(std::make_unique<WorkerScratch>());
                idle.push_back(W.ws.back().get());
            }
            mine = idle.back();
            idle.pop_back();
        }
        WorkerScratch &sc = *mine;
        uint8_t *const buf = W.payload.p + frame[k];
        const u64 len = front[k] + pay[k];
        write_tree(c, buf);
        write_len_word(c, buf + front[k] - 8);
        h1[k] = h1_of(h_hist + hoff[k], h_first + hoff[k], hoff[k + 1] - hoff[k], h_mm[2 * k], S);
        if (pay[k]) {
            const Group &G = groups[group_of[k]];
            there[k] = cudaSetDevice(dev) == cudaSuccess && cudaEventSynchronize(W.events[2 * group_of[k] + 1]) == cudaSuccess;
            if (G.k1 - G.k0 > 1) std::memcpy(buf + front[k], W.payload.p + G.at + (word_off[k] - word_off[G.k0]) * 4, pay[k]);
        }
        if (sc.z.size() < ZSTD_compressBound(len)) sc.z.resize(ZSTD_compressBound(len));
        if (!sc.cc) sc.cc = ZSTD_createCCtx();
        const size_t n = sc.cc ? ZSTD_compressCCtx(sc.cc, sc.z.data(), sc.z.size(), buf, len, 3)
                               : ZSTD_compress(sc.z.data(), sc.z.size(), buf, len, 3);
        zok[k] = !ZSTD_isError(n);
        zb[k] = n;
        std::lock_guard<std::mutex> g(idle_mu);
        idle.push_back(mine);
    });
    if (!es.empty()) {
        u64 enc_err = 0;
        CK(cudaMemcpyAsync(&enc_err, eb + o_err, sizeof(u64), cudaMemcpyDeviceToHost, st));
        CK(cudaStreamSynchronize(st));
        CK(cudaStreamSynchronize(W.copies));
        if (enc_err) return bad(ASZ_E_DEVICE, "Huffman encoder: a tile's wait for the tiles before it timed out");
    }
    const double enc_s = std::chrono::duration<double>(clk::now() - t_enc).count();
    for (u64 k = 0; k < kc; k++) {
        if (!there[k]) return bad(ASZ_E_CUDA, "waiting for a stream's payload failed");
        if (!zok[k]) return bad(ASZ_E_DATA, "zstd compression failed");
        asz_sweep_row &r = S_.rows[k0 + k];
        std::memset(&r, 0, sizeof r);
        r.rel_eb = S_.rel_eb;
        r.c0 = S_.grid[k0 + k].first;
        r.c1 = S_.grid[k0 + k].second;
        r.samples = S;
        r.huffman_bytes = front[k] + pay[k];
        r.zstd_bytes = zb[k];
        r.mse_sum = h_sums[3 * k];
        r.rmse_sum = h_sums[3 * k + 1];
        r.mae_sum = h_sums[3 * k + 2];
        r.h1 = h1[k];
        r.encode_seconds = enc_s / (double)kc;
        finish_row(r, S_.range);
    }
    return ASZ_OK;
}

}  // namespace

extern "C" int asz_sweep(asz_ctx *ctx, const float *data, int on_device, const uint64_t dims[3], const char *predictor,
                         const char *targets, const char *six_grid, const double *rel_eb, uint64_t n_eb, asz_sweep_row *rows,
                         uint64_t cap, uint64_t *n_rows, float *min_max) {
    if (!ctx) return ASZ_E_ARG;
    auto bad = [&](int code, const std::string &m) { return host::ctx_fail(ctx, code, m); };
    if (!data || !dims || !rel_eb || !n_rows) return bad(ASZ_E_ARG, "null argument");
    Predictor p;
    std::string err;
    if (!parse_predictor(predictor, p, err)) return bad(ASZ_E_ARG, err);
    const std::string tg = targets ? targets : "legacy", six = six_grid ? six_grid : "legacy";
    if (tg != "legacy" && tg != "shared1d" && tg != "common") return bad(ASZ_E_ARG, "target mode must be legacy, shared1d or common");
    std::vector<std::pair<double, double>> grid;
    if (!coef_grid(p, six, grid, err)) return bad(ASZ_E_ARG, err);
    if (n_eb == 0) return bad(ASZ_E_ARG, "error-bound grid is empty");
    for (u64 i = 0; i < n_eb; i++)
        if (!std::isfinite(rel_eb[i]) || rel_eb[i] <= 0) return bad(ASZ_E_ARG, "error bounds must be positive and finite");
    u64 N = 1;
    for (int a = 0; a < 3; a++) {  // s2_many_prediction.cpp:509-515
        if (dims[a] < 12 || N > ULLONG_MAX / dims[a]) return bad(ASZ_E_ARG, "invalid dimensions; each dimension must be at least 12");
        N *= dims[a];
    }
    SweepGeom g;
    sweep_geometry(p, dims, tg, g);
    const u64 K = grid.size(), S = g.targets;
    *n_rows = n_eb * K;
    if (cap < n_eb * K) return bad(ASZ_E_ARG, "row buffer too small");
    if (S == 0) return bad(ASZ_E_DATA, "no prediction targets");
    void *&sp = host::ctx_sweep_state(ctx);
    if (!sp) sp = new SweepState();
    SweepState &W = *(SweepState *)sp;

    const float *d_in = data;
    int rc;
    if (!on_device && (rc = host::ctx_upload(ctx, data, N, &d_in))) return rc;
    float mn, mx;  // s2_many_prediction.cpp:521-527
    if ((rc = host::ctx_range(ctx, d_in, N, true, mn, mx))) {
        if (rc == ASZ_E_DATA) return bad(ASZ_E_DATA, "input contains nonfinite values");
        return rc;
    }
    if (min_max) {
        min_max[0] = mn;
        min_max[1] = mx;
    }
    if (!(mx > mn)) return bad(ASZ_E_DATA, "constant input");
    const double range = (double)mx - (double)mn;

    // Coefficients per batch: their QB streams share the device with the field. The device's free
    // memory is asked for only where the buffer that is there does not hold them all (the question
    // takes 0.1 to 0.3 ms).
    u64 budget = 0;
    auto most = [&](u64 size, u64 &kb) -> int {
        kb = K;
        if (W.qb.cap >= K * S * size) return ASZ_OK;
        if (!budget) {
            size_t free_b = 0, total_b = 0;
            CK(cudaMemGetInfo(&free_b, &total_b));
            budget = std::max<u64>(S * 8, std::min<u64>(free_b / 3, 24ull << 30));
        }
        kb = std::max<u64>(1, std::min<u64>(K, budget / (S * size)));
        return ASZ_OK;
    };
    u64 KB = 0, KB8 = 0;
    if ((rc = most(4, KB))) return rc;
    for (u64 e = 0; e < n_eb; e++) {
        const double abs_eb = rel_eb[e] * range;  // :195-196
        const SweepCall call{ctx, W, g, d_in, range, rel_eb[e], abs_eb, 1 / (2 * abs_eb), grid, p, rows + e * K};
        for (u64 k0 = 0; k0 < K; k0 += KB) {
            const u64 kc = std::min<u64>(KB, K - k0);
            rc = sweep_batch<int32_t>(call, k0, kc);
            if (rc == kWide) {
                if (!KB8 && (rc = most(8, KB8))) return rc;
                rc = ASZ_OK;
                for (u64 k = k0; k < k0 + kc && !rc; k += KB8) rc = sweep_batch<int64_t>(call, k, std::min<u64>(KB8, k0 + kc - k));
            }
            if (rc) return rc;
        }
    }
    return ASZ_OK;
}
