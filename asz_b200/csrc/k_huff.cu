// Huffman stage on the GPU: symbol histograms, encoding into the reference's LSB-first bit
// layout (c_codes/asz_core/huffman.hpp:340-381, 610-632), and decoding of that layout.
//
// The reference decodes serially (huffman.hpp:383-526). Here the payload is cut into chunks
// of a fixed number of bits, and one thread decodes each chunk from a guessed codeword boundary.
// Huffman codes resynchronise after a few codewords, so a chunk decoded from the true start of
// its predecessor's last codeword ends at the same place as the guess. A warp settles a run of
// chunks and a check compares the runs' ends and starts (passes repeat while one moves). A final
// pass writes the symbols at offsets from a scan of per-chunk counts.
// Every loop is bounded by the chunk length plus the longest code.
#include <cuda_runtime.h>

#include <algorithm>


#include "dev_common.cuh"
#include "launch.h"

namespace asz {

// ---------------------------------------------------------------------------------------------
// Histogram of symbols in [offset, offset+range). Counts are 64-bit; of a range up to kHistShared a CTA
// counts in shared memory first. A thread takes runs of kHistRun consecutive symbols, from run r0 on in
// steps of dr, and adds equal neighbours together: most symbols of a stream are a few values, often
// repeated, so this saves most atomics.
constexpr uint32_t kHistRun = 8, kHistShared = 8192;
template <class T>
__device__ __forceinline__ void histogram_of(const T *__restrict__ s, uint64_t n, int64_t offset, uint64_t range,
                                             unsigned long long *__restrict__ hist, uint64_t r0, uint64_t r1, uint64_t dr) {
    extern __shared__ unsigned int sh[];
    const bool use_sh = range <= kHistShared;
    if (use_sh) {
        for (uint64_t i = threadIdx.x; i < range; i += blockDim.x) sh[i] = 0;
        __syncthreads();
    }
    auto add = [&](uint64_t v, uint32_t c) {
        if (use_sh) atomicAdd(&sh[v], c);
        else atomicAdd(&hist[v], (unsigned long long)c);
    };
    for (uint64_t r = r0; r < r1; r += dr) {
        const uint64_t i0 = r * kHistRun, i1 = min(i0 + kHistRun, n);
        uint64_t cur = (uint64_t)((int64_t)s[i0] - offset);
        uint32_t c = 1;
        for (uint64_t i = i0 + 1; i < i1; i++) {
            const uint64_t v = (uint64_t)((int64_t)s[i] - offset);
            if (v == cur) {
                c++;
            } else {
                add(cur, c);
                cur = v;
                c = 1;
            }
        }
        add(cur, c);
    }
    if (use_sh) {
        __syncthreads();
        for (uint64_t i = threadIdx.x; i < range; i += blockDim.x)
            if (sh[i]) atomicAdd(&hist[i], (unsigned long long)sh[i]);
    }
}

template <class T>
__global__ void histogram_kernel(const T *__restrict__ s, uint64_t n, int64_t offset, uint64_t range,
                                 unsigned long long *__restrict__ hist) {
    histogram_of(s, n, offset, range, hist, blockIdx.x * (uint64_t)blockDim.x + threadIdx.x, (n + kHistRun - 1) / kHistRun,
                 (uint64_t)gridDim.x * blockDim.x);
}

// The streams of a set, a CTA per tile of a stream. A launch per stream was bound by the launches and
// by CTAs too few to fill the chip: the 80 streams of eight fields (33M values) 0.56 -> 0.10 ms.
__global__ void histogram_set_kernel(const __grid_constant__ HistSet set) {
    uint32_t lo = 0, hi = set.n;  // the last stream that starts at or before this tile
    while (hi - lo > 1) {
        const uint32_t mid = (lo + hi) / 2;
        if (set.s[mid].tile <= blockIdx.x) lo = mid;
        else hi = mid;
    }
    const HistStream &h = set.s[lo];
    const uint64_t runs = (h.n + kHistRun - 1) / kHistRun, r = (uint64_t)(blockIdx.x - h.tile) * set.tile_runs;
    const uint64_t r0 = r + threadIdx.x, r1 = min(r + set.tile_runs, runs);
    if (h.wide) histogram_of((const int64_t *)h.sym, h.n, h.lo, h.range, h.hist, r0, r1, blockDim.x);
    else histogram_of((const int32_t *)h.sym, h.n, h.lo, h.range, h.hist, r0, r1, blockDim.x);
}

// ---------------------------------------------------------------------------------------------
// Tiled encoding of several streams in one launch: tiles of enc_tile<T>() symbols, a stream's
// tiles consecutive. A CTA takes tiles in order from a ticket counter and copies the next tile's
// symbols into shared memory (asynchronous copies) while it encodes the current one. Per tile it
// counts the tile's bits, publishes the count, and finds the tile's bit offset in its stream by
// looking back over the tiles before it (decoupled look-back: each tile's state word holds its
// count, then its inclusive prefix); it then builds the tile's bits in shared memory and writes
// them as whole words, with atomicOr only on its first and last word, which it may share with the
// neighbouring tiles. Tiles are handed out in order, so every tile a CTA waits for is held by a
// CTA that is running; every wait is bounded and a wait that runs out sets the error word.

__device__ __forceinline__ uint32_t stream_of(const uint64_t *toff, uint32_t ns, uint64_t t) {
    uint32_t lo = 0, hi = ns;  // toff[lo] <= t < toff[hi]
    while (hi - lo > 1) {
        const uint32_t mid = (lo + hi) >> 1;
        if (toff[mid] <= t) lo = mid;
        else hi = mid;
    }
    return lo;
}

// Tile state words: status in the top two bits, bits (count or inclusive prefix) below.
constexpr unsigned long long kTileCount = 1ull << 62, kTilePrefix = 2ull << 62, kTileValue = (1ull << 62) - 1;
constexpr uint32_t kLookbackPolls = 1u << 22;

template <class T>
__device__ __forceinline__ void cp_async_sym(T *dst, const T *src) {
    const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
    if constexpr (sizeof(T) == 4) asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(d), "l"(src) : "memory");
    else asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit_group() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_older() { asm volatile("cp.async.wait_group 1;\n" ::: "memory"); }

template <class T>
__global__ void __launch_bounds__(kEncThreads, 4)
    encode_tiles_kernel(const EncStream *__restrict__ S, uint32_t ns, const uint64_t *__restrict__ toff, uint64_t ntiles,
                        unsigned long long *state, unsigned long long *err) {
    constexpr uint32_t kTile = enc_tile<T>(), kPer = kTile / kEncThreads;
    // Symbol i of a tile sits at i + i / kPer: each thread reads its own kPer consecutive symbols,
    // and the one-slot gap between runs spreads a warp's reads over all banks.
    // Dynamic shared memory: two stages of symbols, then the tile's words (codes are at most 32
    // bits, plus the leading shift).
    extern __shared__ __align__(16) unsigned char enc_smem[];
    T(*sym_sh)[kTile + kEncThreads] = reinterpret_cast<T(*)[kTile + kEncThreads]>(enc_smem);
    uint32_t *buf = reinterpret_cast<uint32_t *>(enc_smem + 2 * (kTile + kEncThreads) * sizeof(T));
    __shared__ uint32_t wsum[kEncThreads / 32];
    __shared__ unsigned long long s_next, s_excl;
    unsigned long long *const ticket = state + ntiles;
    const uint32_t tid = threadIdx.x, lane = tid & 31;
    // Copies of tile t's symbols into stage b (this thread's share), committed as one group.
    auto issue = [&](uint64_t t, uint32_t b) {
        if (t < ntiles) {
            const uint32_t si = stream_of(toff, ns, t);
            const EncStream &E = S[si];
            const T *sym = reinterpret_cast<const T *>(E.s);
            const uint64_t i0 = (t - toff[si]) * kTile;
            const uint32_t cnt = (uint32_t)min((uint64_t)kTile, E.n - i0);
            for (uint32_t i = tid; i < cnt; i += kEncThreads) cp_async_sym(&sym_sh[b][i + i / kPer], sym + i0 + i);
        }
        cp_async_commit_group();
    };
    if (tid == 0) s_next = atomicAdd(ticket, 1ull);
    __syncthreads();
    uint64_t t = s_next;
    issue(t, 0);
    uint32_t b = 0;
    while (t < ntiles) {
        // Every thread has read s_next and is done with stage b ^ 1 (the tile before this one).
        __syncthreads();
        if (tid == 0) s_next = atomicAdd(ticket, 1ull);
        for (uint32_t i = tid; i < kTile + 2; i += kEncThreads) buf[i] = 0u;
        __syncthreads();
        const uint64_t tn = s_next;
        issue(tn, b ^ 1);
        cp_async_wait_older();
        __syncthreads();  // this tile's symbols, copied by every thread, are in place
        const uint32_t si = stream_of(toff, ns, t);
        const EncStream &E = S[si];
        const uint64_t t0 = toff[si];
        const uint64_t i0 = (t - t0) * kTile;
        const uint32_t cnt = (uint32_t)min((uint64_t)kTile, E.n - i0);
        // This thread's symbols: kPer consecutive ones, so its bits are one consecutive run.
        const uint32_t j0 = tid * kPer;
        uint32_t code[kPer], len[kPer];
        uint32_t mine = 0;
#pragma unroll
        for (uint32_t k = 0; k < kPer; k++) {
            CodeEntry e{0u, 0u};
            if (j0 + k < cnt) e = E.tab[(uint64_t)((int64_t)sym_sh[b][j0 + k + tid] - E.offset)];
            code[k] = e.code;
            len[k] = e.len;
            mine += e.len;
        }
        // Exclusive scan of the threads' bit counts (warp shuffles, then the warps' sums).
        uint32_t incl = mine;
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t v = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= (uint32_t)o) incl += v;
        }
        if (lane == 31) wsum[tid >> 5] = incl;
        __syncthreads();
        uint32_t before = 0, total = 0;
        for (uint32_t w = 0; w < kEncThreads / 32; w++) {
            if (w < (tid >> 5)) before += wsum[w];
            total += wsum[w];
        }
        // Pack the run at bit 0 of the tile's words (the tile's offset in its stream is applied when
        // the words are written, so the packing need not wait for it): the run's first and last
        // words may be shared with the neighbouring runs and are or-ed in; the words between belong
        // to this thread alone.
        const uint32_t pos = before + incl - mine;
        if (mine) {
            uint32_t w = pos >> 5, nacc = pos & 31;
            uint64_t acc = 0;
            bool first = true;
#pragma unroll
            for (uint32_t k = 0; k < kPer; k++) {
                acc |= (uint64_t)code[k] << nacc;
                nacc += len[k];
                if (nacc >= 32) {
                    if (first) atomicOr(&buf[w], (uint32_t)acc);
                    else buf[w] = (uint32_t)acc;
                    first = false;
                    w++;
                    acc >>= 32;
                    nacc -= 32;
                }
            }
            if (nacc) atomicOr(&buf[w], (uint32_t)acc);
        }
        // The tile's bit offset in its stream: publish the count, then add up the counts back to
        // the nearest published prefix (or the stream's first tile).
        if (tid < 32) {
            unsigned long long excl = 0;
            if (t == t0) {
                if (lane == 0) atomicExch(&state[t], kTilePrefix | total);
            } else {
                if (lane == 0) atomicExch(&state[t], kTileCount | total);
                for (int64_t j = (int64_t)t - 1;; j -= 32) {
                    const int64_t pidx = j - (int64_t)lane;
                    unsigned long long v = kTilePrefix;  // before the stream's first tile: prefix 0
                    if (pidx >= (int64_t)t0) {
                        const volatile unsigned long long *w = state + pidx;
                        v = *w;
                        for (uint32_t polls = 0; !(v >> 62) && polls < kLookbackPolls; polls++) {
                            __nanosleep(64);
                            v = *w;
                        }
                        if (!(v >> 62)) {
                            atomicOr(err, 1ull);
                            v = kTilePrefix;
                        }
                    }
                    const uint32_t pref = __ballot_sync(0xffffffffu, (v >> 62) == 2);
                    const uint32_t upto = pref ? (uint32_t)(__ffs(pref) - 1) : 31u;
                    unsigned long long x = lane <= upto ? (v & kTileValue) : 0ull;
                    for (int o = 16; o; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
                    excl += x;
                    if (pref) break;
                }
                if (lane == 0) atomicExch(&state[t], kTilePrefix | (excl + total));
            }
            if (lane == 0) s_excl = excl;
        }
        __syncthreads();
        // Words out, shifted to the tile's offset: word i takes the high bits of packed word i - 1.
        const uint64_t bit0 = s_excl + E.bit0;
        const uint32_t shift = (uint32_t)(bit0 & 31);
        const uint32_t nw = (shift + total + 31) >> 5;
        uint32_t *out = E.out + (bit0 >> 5);
        for (uint32_t i = tid; i < nw; i += kEncThreads) {
            const uint32_t v = shift ? (buf[i] << shift) | (i ? buf[i - 1] >> (32 - shift) : 0u) : buf[i];
            if (i == 0 || i == nw - 1) {
                if (v) atomicOr(&out[i], v);
            } else {
                out[i] = v;
            }
        }
        t = tn;
        b ^= 1;
    }
    cp_async_wait_older();  // the last committed group (past the end) holds no copies
}

// ---------------------------------------------------------------------------------------------
// Decoding. The host builds two tables per stream (huffman_host.h): one indexed by the next lut_bits
// payload bits (LSB-first), staged in shared memory, and, for longer codes, one by up to ten bits
// more, read through L1. Entries carry the code's length in the top 5 bits and its symbol; length 0
// leads on to the second table, and from there to the tree: child[2*node+bit] (a value >= 0x80000000
// marks a leaf whose symbol index is the low bits).
//
// A symbol is a dependent chain of a few shared-memory reads, so a kernel decodes as fast as its
// warps issue. A tile's payload is therefore staged in shared memory too, where the next 32 bits of
// any position are two words and a funnel shift; a queue of words in each thread's registers, refilled
// by 16-byte loads, had the threads of a warp refill at different symbols, so that every symbol of
// the warp ran all the refill's branches (512^3 at 1e-3, 6.6 bits a symbol: 0.75 ms to synchronise and
// 0.82 to write, now 0.47 and 0.49).

// A stream's tables, the first in shared memory.
struct DecodeTables {
    const uint32_t *lut, *lut2, *child;
    uint32_t lut_bits;
};

// A chunk's words: W of its own after a lead of up to 31 bits, and two more that its last codeword
// may reach. The odd stride keeps a warp's reads, at about the same place of its chunks, on
// different banks.
ASZ_HD constexpr uint32_t slot_words(uint32_t W) { return W + 3; }
constexpr uint32_t kDecodeSlotBytes = ((decode_tile(32) + decode_halo(32)) * slot_words(32) * 4 + 15) / 16 * 16;  // the most

// The 32 payload bits from bit `pos` of a slot on.
__device__ __forceinline__ uint32_t peek(const uint32_t *slot, uint32_t pos) {
    const uint32_t i = pos >> 5;
    return __funnelshift_r(slot[i], slot[i + 1], pos & 31);
}

// Decode the codeword at `pos`; returns the symbol index and advances pos by the code length. A path
// that leaves the tree moves pos past every limit (kBadPath).
constexpr uint32_t kBadPath = 1u << 30;

__device__ __forceinline__ uint32_t decode_sym(const uint32_t *slot, uint32_t &pos, const DecodeTables &T) {
    const uint32_t v = peek(slot, pos);
    uint32_t e = T.lut[v & ((1u << T.lut_bits) - 1)], len = e >> 27;
    e &= 0x7ffffffu;
    if (len == 0) {
        const uint32_t sub = e & 15u;
        const uint32_t e2 = __ldg(T.lut2 + (e >> 4) + ((v >> T.lut_bits) & ((1u << sub) - 1)));
        len = e2 >> 27;
        e = e2 & 0x7ffffffu;
        if (len == 0) {  // codes are at most 32 bits
            uint32_t node = e, used = T.lut_bits + sub;
            while (true) {
                const uint32_t c = __ldg(T.child + 2 * (uint64_t)node + ((v >> used) & 1));
                used++;
                if (c & 0x80000000u) {
                    e = c & 0x7fffffffu;
                    break;
                }
                node = c;
                if (used >= 32) {  // impossible for a validated tree; stop instead of running on
                    used = kBadPath;
                    break;
                }
            }
            len = used;
        }
    }
    pos += len;
    return e;
}

// ---------------------------------------------------------------------------------------------
// Batched decoding of every stream of a .asz in one launch per pass. A stream's chunks have
// DecStream::words words, 8 or 32, and are numbered globally (stream after stream); a tile of them
// (decode_tile: 192 or 240) never crosses a stream, so a CTA stages one stream's lookup table for a tile.
// When synchronising, a warp has the next decode_run chunks (24 or 30) and decodes the decode_halo
// before them as well. Bit positions are absolute from the 16-byte aligned stream buffer `base`.

__device__ __forceinline__ void stage_lut(uint4 *lut_sh, const uint32_t *__restrict__ lut, uint32_t lut_bits) {
    const uint4 *v = reinterpret_cast<const uint4 *>(lut);
    for (uint32_t i = threadIdx.x; i < ((1u << lut_bits) + 3) / 4; i += blockDim.x) lut_sh[i] = __ldg(v + i);
}

// The words of kSlots chunks from chunk `first` of the stream on (negative: none there) into their
// slots. Words outside the payload read as zero.
template <uint32_t W, uint32_t kSlots>
__device__ __forceinline__ void stage_payload(uint32_t *slots, const uint8_t *__restrict__ base, const DecStream &d, int64_t first) {
    const uint32_t *words = reinterpret_cast<const uint32_t *>(base);
    const int64_t lo = (int64_t)(d.bit_begin >> 5), hi = (int64_t)(d.bit_end >> 5) + 1;  // kDecodePad lies behind
    const int64_t w0 = lo + first * W;
    constexpr uint32_t kWords = kSlots * W + 2, kUnroll = 8;
    for (uint32_t i0 = threadIdx.x; i0 < kWords; i0 += kUnroll * kDecodeThreads) {
        uint32_t v[kUnroll];
#pragma unroll
        for (uint32_t u = 0; u < kUnroll; u++) {
            const int64_t g = w0 + i0 + u * kDecodeThreads;
            v[u] = g >= lo && g <= hi && i0 + u * kDecodeThreads < kWords ? __ldg(words + g) : 0u;
        }
#pragma unroll
        for (uint32_t u = 0; u < kUnroll; u++) {
            const uint32_t i = i0 + u * kDecodeThreads, slot = i / W, j = i % W;
            if (slot < kSlots) slots[slot * slot_words(W) + j] = v[u];
            if (j < 2 && slot && slot <= kSlots) slots[(slot - 1) * slot_words(W) + W + j] = v[u];
        }
    }
}

// One chunk's decoding, in bits from its slot's start: where it stopped and how many values it met.
// marks[j * kDecodeThreads] keeps a codeword's start about j + 1 eighths of the chunk after `lead`, with
// the values before it in the upper half. A chunk that has to start elsewhere is read until it meets
// one of them (codewords fall in step after a geometrically distributed number of bits, about 30 at 4
// bits a symbol and 130 at 10; from there on it is decoded already).
constexpr uint32_t kMarks = 7;

template <uint32_t W>
struct ChunkRun {
    static constexpr uint32_t kMarkBits = 4 * W;
    uint32_t end = 0, count = 0;

    __device__ __forceinline__ void decode(const uint32_t *slot, uint32_t lead, uint32_t pos, uint32_t lim, const DecodeTables &T,
                                           uint32_t *marks, uint32_t *err_word) {
        uint32_t c = 0, mark = lead + kMarkBits, j = 0;
        while (pos < lim) {
            decode_sym(slot, pos, T);
            c++;
            if (pos >= mark) {
                if (j >= kMarks || pos >= kBadPath) continue;
                const uint32_t old = marks[j * kDecodeThreads];
                marks[j * kDecodeThreads] = c << 16 | pos;
                if ((old & 0xffffu) == pos) {
                    const uint32_t more = c - (old >> 16);  // modulo 2^16, as the marks
                    for (uint32_t i = j + 1; i < kMarks; i++) marks[i * kDecodeThreads] += more << 16;
                    count += (uint32_t)(int32_t)(int16_t)more;
                    return;  // the same end
                }
                j++;
                mark += kMarkBits;
            }
        }
        if (pos >= kBadPath) atomicOr(err_word, 8u);
        end = pos;
        count = c;
        for (; j < kMarks; j++) marks[j * kDecodeThreads] = 0;  // not reached: no position
    }
};

// Synchronisation. Chunk k decodes from its start until it reaches the next chunk's first bit,
// recording where it stopped (end[k]) and how many values it produced (count[k]). First pass: every
// chunk starts at its first bit, and then, within its warp, where its predecessor ended, until no
// start moves. A warp's first chunk has its predecessor in another warp, so a warp's first
// lanes decode the chunks before its own as well: a wrong guess nearly always meets the
// true codewords within those bits (a 161x257x349 quintic stream at 1e-4 needed five passes
// over all chunks, with the host waiting for each; now it is this one). What it nearly always is,
// decode_check_kernel checks; a warp whose first chunk did start elsewhere is settled by the later
// passes, which start at start[] and decode only from a moved first chunk on (moved[k] != 0).
template <uint32_t W>
__device__ __forceinline__ bool sync_tile(const uint8_t *__restrict__ base, const DecStream &d, uint64_t tile, bool fresh,
                                          const uint32_t *__restrict__ luts, const uint32_t *__restrict__ lut2s,
                                          const uint32_t *__restrict__ childs, int first_pass, uint64_t *__restrict__ start,
                                          uint64_t *__restrict__ end, uint64_t *__restrict__ count,
                                          const uint32_t *__restrict__ moved, uint32_t *slots, uint4 *lut_sh, uint32_t *marks,
                                          uint32_t *err_word) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int64_t kl0 = (int64_t)((tile - d.tile0) * decode_tile(W)) - (int)decode_halo(W);
    if (!first_pass) {
        const uint64_t mine = (uint64_t)(tile - d.tile0) * decode_tile(W) + threadIdx.x;
        if (!__syncthreads_or(threadIdx.x < decode_tile(W) && mine < d.nchunks && moved[d.chunk0 + mine])) return false;
    }
    __syncthreads();  // the tile before is done with the shared memory
    if (fresh) stage_lut(lut_sh, luts + d.lut_off, d.lut_bits);
    stage_payload<W, decode_tile(W) + decode_halo(W)>(slots, base, d, kl0);
    for (uint32_t j = 0; j < kMarks; j++) marks[j * kDecodeThreads] = 0;
    __syncthreads();
    const DecodeTables T{reinterpret_cast<const uint32_t *>(lut_sh), lut2s + d.lut2_off, childs + d.child_off, d.lut_bits};
    const int at_slot = warp * (int)decode_run(W) + lane;
    const int64_t kl = kl0 + at_slot;
    const uint32_t *slot = slots + at_slot * slot_words(W);
    const bool own = lane >= (int)decode_halo(W) && kl < (int64_t)d.nchunks;
    const bool in = first_pass ? kl >= 0 && kl < (int64_t)d.nchunks : own;
    const bool after = in && lane > (first_pass ? 0 : (int)decode_halo(W)) && kl > 0;  // has a predecessor here
    const uint64_t k = d.chunk0 + (uint64_t)kl;
    // Positions relative to the chunk's slot.
    const uint32_t lead = (uint32_t)(d.bit_begin & 31), span = 32 * W;
    const uint64_t first = d.bit_begin + (uint64_t)kl * span, origin = first - lead;
    const uint32_t lim = in ? lead + (uint32_t)min((uint64_t)span, d.bit_end - first) : 0;
    uint32_t s = lead;
    ChunkRun<W> run;
    bool need = in;
    if (in && !first_pass) {
        s = (uint32_t)(start[k] - origin);
        run.end = (uint32_t)(end[k] - origin);
        run.count = (uint32_t)count[k];
        need = moved[k] != 0;
    }
    // Each turn makes at least one more chunk of the warp final.
    for (uint32_t turn = 0; turn <= 32; turn++) {
        if (need) run.decode(slot, lead, s, lim, T, marks, err_word);
        __syncwarp();
        const uint32_t before = __shfl_up_sync(0xffffffffu, run.end, 1);
        const uint32_t at = after ? before - span : s;
        need = at != s;
        s = at;
        if (!__any_sync(0xffffffffu, need)) break;
    }
    if (own) {
        start[k] = origin + s;
        end[k] = origin + run.end;
        count[k] = run.count;
    }
    return true;
}

__global__ void __launch_bounds__(kDecodeThreads, 4)
    decode_sync_kernel(const uint8_t *__restrict__ base, const DecStream *__restrict__ streams,
                       const uint32_t *__restrict__ tile_stream, uint64_t ntiles, const uint32_t *__restrict__ luts,
                       const uint32_t *__restrict__ lut2s, const uint32_t *__restrict__ childs, int first_pass,
                       uint64_t *__restrict__ start, uint64_t *__restrict__ end, uint64_t *__restrict__ count,
                       const uint32_t *__restrict__ moved, uint32_t *err_word) {
    extern __shared__ uint4 dec_smem[];
    __shared__ uint32_t marks_sh[kMarks * kDecodeThreads];
    uint32_t *const slots = reinterpret_cast<uint32_t *>(dec_smem);
    uint4 *const lut_sh = dec_smem + kDecodeSlotBytes / 16;
    uint32_t *const marks = marks_sh + threadIdx.x;
    uint32_t staged = 0xffffffffu;
    for (uint64_t tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
        const uint32_t si = tile_stream[tile];
        const DecStream &d = streams[si];
        const bool done = d.words == 8 ? sync_tile<8>(base, d, tile, si != staged, luts, lut2s, childs, first_pass, start, end, count,
                                                      moved, slots, lut_sh, marks, err_word)
                                       : sync_tile<32>(base, d, tile, si != staged, luts, lut2s, childs, first_pass, start, end, count,
                                                       moved, slots, lut_sh, marks, err_word);
        if (done) staged = si;  // its table is in shared memory
    }
}

__device__ __forceinline__ uint32_t stream_of_chunk(const DecStream *__restrict__ streams, uint32_t nstreams, uint64_t k) {
    uint32_t lo = 0, hi = nstreams;  // last stream with chunk0 <= k
    while (hi - lo > 1) {
        const uint32_t mid = (lo + hi) / 2;
        if (streams[mid].chunk0 <= k) lo = mid;
        else hi = mid;
    }
    return lo;
}

// After a pass: the start of chunk k (not the first of its stream) becomes end[k-1]. Marks the
// chunks whose start moved (moved[k]) and flags whether any did.
__global__ void decode_restart_kernel(const DecStream *__restrict__ streams, uint32_t nstreams, uint64_t nchunks,
                                      const uint64_t *__restrict__ end, uint64_t *__restrict__ start, uint32_t *__restrict__ moved,
                                      uint32_t *changed) {
    for (uint64_t k = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; k < nchunks; k += (uint64_t)gridDim.x * blockDim.x) {
        uint32_t m = 0;
        if (streams[stream_of_chunk(streams, nstreams, k)].chunk0 != k) {
            const uint64_t s = end[k - 1];
            if (s != start[k]) {
                start[k] = s;
                m = 1;
                *changed = 1u;
            }
        }
        moved[k] = m;
    }
}

// Per warp of a tile: whether its first chunk started where the one before it ended (`changed` if
// not). Per stream, once the starts are stable: the values decoded must equal the stream's count and the last
// chunk must end exactly at the payload's last bit. off[] is the exclusive scan of count[] over all
// chunks (nchunks + 1 entries).
__global__ void decode_check_kernel(const DecStream *__restrict__ streams, uint32_t nstreams,
                                    const uint32_t *__restrict__ tile_stream, uint64_t ntiles, const uint64_t *__restrict__ off,
                                    const uint64_t *__restrict__ start, const uint64_t *__restrict__ end, uint32_t *err_word,
                                    uint32_t *changed) {
    const uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
    constexpr uint32_t kRuns = kDecodeThreads / 32;
    if (i < ntiles * kRuns) {
        const uint64_t tile = i / kRuns;
        const DecStream &d = streams[tile_stream[tile]];
        const uint64_t kl = (tile - d.tile0) * decode_tile(d.words) + i % kRuns * decode_run(d.words), k = d.chunk0 + kl;
        if (kl && kl < d.nchunks && start[k] != end[k - 1]) *changed = 1u;
    }
    if (i >= nstreams) return;
    const DecStream d = streams[i];
    const uint64_t got = off[d.chunk0 + d.nchunks] - off[d.chunk0];
    if (got < d.count) atomicOr(err_word, 32u);
    if (got > d.count) atomicOr(err_word, 64u);
    if (end[d.chunk0 + d.nchunks - 1] != d.bit_end) atomicOr(err_word, 128u);
}

// Pass B over all tiles: write the values (symbol index + offset) of chunk k at its offset in its
// stream's output (int64 for the t stream, int32 for QB streams).
template <uint32_t W>
__device__ __forceinline__ void write_tile(const uint8_t *__restrict__ base, const DecStream &d, uint64_t tile, bool fresh,
                                           const uint32_t *__restrict__ luts, const uint32_t *__restrict__ lut2s,
                                           const uint32_t *__restrict__ childs, const uint64_t *__restrict__ start,
                                           const uint64_t *__restrict__ off, uint32_t *slots, uint4 *lut_sh, uint32_t *err_word) {
    const uint64_t kl0 = (tile - d.tile0) * decode_tile(W), kl = kl0 + threadIdx.x;
    __syncthreads();
    if (fresh) stage_lut(lut_sh, luts + d.lut_off, d.lut_bits);
    stage_payload<W, decode_tile(W)>(slots, base, d, (int64_t)kl0);
    __syncthreads();
    if (threadIdx.x >= decode_tile(W) || kl >= d.nchunks) return;
    const DecodeTables T{reinterpret_cast<const uint32_t *>(lut_sh), lut2s + d.lut2_off, childs + d.child_off, d.lut_bits};
    const uint32_t *slot = slots + threadIdx.x * slot_words(W);
    const uint64_t k = d.chunk0 + kl;
    const uint32_t lead = (uint32_t)(d.bit_begin & 31);
    const uint64_t first = d.bit_begin + kl * (32 * W);
    uint32_t pos = (uint32_t)(start[k] - (first - lead));
    const uint32_t lim = lead + (uint32_t)min((uint64_t)(32 * W), d.bit_end - first);
    if (pos >= lim) return;
    const uint64_t o0 = off[k] - off[d.chunk0], count = d.count;
    if (o0 >= count) {
        atomicOr(err_word, 16u);
        return;
    }
    const uint32_t room = (uint32_t)min(count - o0, (uint64_t)0xffffffffu);  // values left of the stream
    uint32_t o = 0;
    if (d.wide) {
        int64_t *out = static_cast<int64_t *>(d.out) + o0;
        const int64_t offset = d.offset;
        while (pos < lim && o < room) out[o++] = (int64_t)decode_sym(slot, pos, T) + offset;
    } else {
        // int32 values go out four at a time as one 16-byte store once the position is aligned:
        // whole sectors leave the thread instead of one value per store.
        int32_t *out = static_cast<int32_t *>(d.out) + o0;
        const uint32_t offset = (uint32_t)(int32_t)d.offset;
        const uint32_t head = min(room, (uint32_t)(-(intptr_t)((uintptr_t)out >> 2) & 3));  // up to the alignment
        while (pos < lim && o < head) out[o++] = (int32_t)(decode_sym(slot, pos, T) + offset);
        while (pos < lim && o + 4 <= room) {
            int4 v;
            v.x = (int32_t)(decode_sym(slot, pos, T) + offset);
            if (pos >= lim) {
                out[o++] = v.x;
                break;
            }
            v.y = (int32_t)(decode_sym(slot, pos, T) + offset);
            if (pos >= lim) {
                out[o] = v.x, out[o + 1] = v.y;
                o += 2;
                break;
            }
            v.z = (int32_t)(decode_sym(slot, pos, T) + offset);
            if (pos >= lim) {
                out[o] = v.x, out[o + 1] = v.y, out[o + 2] = v.z;
                o += 3;
                break;
            }
            v.w = (int32_t)(decode_sym(slot, pos, T) + offset);
            *reinterpret_cast<int4 *>(out + o) = v;
            o += 4;
        }
        while (pos < lim && o < room) out[o++] = (int32_t)(decode_sym(slot, pos, T) + offset);
    }
    if (pos < lim || pos >= kBadPath) atomicOr(err_word, 16u);
}

__global__ void __launch_bounds__(kDecodeThreads, 4)
    decode_write_kernel(const uint8_t *__restrict__ base, const DecStream *__restrict__ streams,
                        const uint32_t *__restrict__ tile_stream, uint64_t ntiles, const uint32_t *__restrict__ luts,
                        const uint32_t *__restrict__ lut2s, const uint32_t *__restrict__ childs,
                        const uint64_t *__restrict__ start, const uint64_t *__restrict__ off, uint32_t *err_word) {
    extern __shared__ uint4 dec_smem[];
    uint32_t *const slots = reinterpret_cast<uint32_t *>(dec_smem);
    uint4 *const lut_sh = dec_smem + kDecodeSlotBytes / 16;
    uint32_t staged = 0xffffffffu;
    for (uint64_t tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
        const uint32_t si = tile_stream[tile];
        const DecStream &d = streams[si];
        if (d.words == 8) write_tile<8>(base, d, tile, si != staged, luts, lut2s, childs, start, off, slots, lut_sh, err_word);
        else write_tile<32>(base, d, tile, si != staged, luts, lut2s, childs, start, off, slots, lut_sh, err_word);
        staged = si;
    }
}

template <class T>
__global__ void fill_kernel(T *__restrict__ out, uint64_t n, T v) {
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) out[i] = v;
}

// ---------------------------------------------------------------------------------------------
// Host-callable launchers (declared in launch.h).

cudaError_t launch_histogram_set(const HistStream *streams, uint32_t n, cudaStream_t st) {
    // Tiles of up to 16384 symbols, smaller where the chip would not be full of them.
    uint64_t runs = 0;
    for (uint32_t i = 0; i < n; i++) runs += (streams[i].n + kHistRun - 1) / kHistRun;
    const uint64_t tile = std::min<uint64_t>(std::max<uint64_t>((runs / (148 * 8) + 255) / 256 * 256, 256), 2048);
    for (uint32_t at = 0; at < n;) {
        HistSet set{};
        set.tile_runs = (uint32_t)tile;
        uint64_t tiles = 0, range = 0;
        for (; at < n && set.n < HistSet::kMost; at++) {
            const uint64_t t = ((streams[at].n + kHistRun - 1) / kHistRun + tile - 1) / tile;
            if (t == 0) continue;
            if (tiles + t > INT32_MAX) break;
            HistStream &h = set.s[set.n++] = streams[at];
            h.tile = (uint32_t)tiles;
            tiles += t;
            if (h.range <= kHistShared) range = std::max(range, h.range);
        }
        if (set.n == 0) {
            if (at < n) return cudaErrorInvalidValue;
            break;
        }
        histogram_set_kernel<<<(unsigned)tiles, 256, range * sizeof(unsigned int), st>>>(set);
        count_launch();
    }
    return cudaGetLastError();
}

template <class T>
cudaError_t launch_histogram(const T *s, uint64_t n, int64_t offset, uint64_t range, unsigned long long *hist,
                             cudaStream_t st) {
    if (n == 0) return cudaSuccess;
    size_t sh = range <= 8192 ? range * sizeof(unsigned int) : 0;
    uint64_t blocks = std::min<uint64_t>((n + 8 * 256 - 1) / (8 * 256), 148 * 8);
    histogram_kernel<T><<<(unsigned)blocks, 256, sh, st>>>(s, n, offset, range, hist);
    count_launch();
    return cudaGetLastError();
}

// ---------------------------------------------------------------------------------------------
// Exclusive prefix sums of n 64-bit values (in == out allowed): tiles of kScanTile values, a CTA
// each, scanned in registers and shared memory; the tiles' totals are scanned the same way (in
// tmp, a level per kScanTile-fold reduction), then added back to their tiles.
constexpr uint32_t kScanThreads = 1024, kScanPer = 4, kScanTile = kScanThreads * kScanPer;

__global__ void __launch_bounds__(kScanThreads)
    scan_tiles_kernel(const uint64_t *in, uint64_t *out, uint64_t n, uint64_t *tile_sums) {
    __shared__ uint64_t wsum[kScanThreads / 32];
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint64_t first = (uint64_t)blockIdx.x * kScanTile + (uint64_t)tid * kScanPer;
    uint64_t v[kScanPer], mine = 0;
#pragma unroll
    for (uint32_t k = 0; k < kScanPer; k++) {
        v[k] = first + k < n ? in[first + k] : 0;
        mine += v[k];
    }
    uint64_t incl = mine;
    for (int o = 1; o < 32; o <<= 1) {
        const uint64_t t = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= (uint32_t)o) incl += t;
    }
    if (lane == 31) wsum[warp] = incl;
    __syncthreads();
    if (warp == 0) {
        const uint64_t w = wsum[lane];
        uint64_t wi = w;
        for (int o = 1; o < 32; o <<= 1) {
            const uint64_t t = __shfl_up_sync(0xffffffffu, wi, o);
            if (lane >= (uint32_t)o) wi += t;
        }
        wsum[lane] = wi - w;
    }
    __syncthreads();
    uint64_t run = wsum[warp] + incl - mine;
#pragma unroll
    for (uint32_t k = 0; k < kScanPer; k++) {
        if (first + k < n) out[first + k] = run;
        run += v[k];
    }
    if (tile_sums && tid == kScanThreads - 1) tile_sums[blockIdx.x] = run;  // the tile's total
}

__global__ void scan_add_kernel(uint64_t *out, uint64_t n, const uint64_t *__restrict__ tile_offsets) {
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x)
        out[i] += tile_offsets[i / kScanTile];
}

static uint64_t scan_tmp_words(uint64_t n) {
    uint64_t w = 0;
    while (n > kScanTile) {
        n = (n + kScanTile - 1) / kScanTile;
        w += n;
    }
    return w;
}

static cudaError_t scan_u64_levels(const uint64_t *in, uint64_t *out, uint64_t n, uint64_t *tmp, cudaStream_t st) {
    if (n == 0) return cudaSuccess;
    const uint64_t tiles = (n + kScanTile - 1) / kScanTile;
    uint64_t *sums = tiles > 1 ? tmp : nullptr;
    scan_tiles_kernel<<<(unsigned)tiles, kScanThreads, 0, st>>>(in, out, n, sums);
    count_launch();
    if (tiles > 1) {
        cudaError_t e = scan_u64_levels(sums, sums, tiles, tmp + tiles, st);
        if (e != cudaSuccess) return e;
        scan_add_kernel<<<(unsigned)std::min<uint64_t>((n + 255) / 256, 148 * 16), 256, 0, st>>>(out, n, sums);
        count_launch();
    }
    return cudaGetLastError();
}

cudaError_t launch_scan_u64(const uint64_t *in, uint64_t *out, uint64_t n, void *tmp, size_t &tmp_bytes, cudaStream_t st) {
    if (tmp == nullptr) {
        tmp_bytes = std::max<size_t>(scan_tmp_words(n) * sizeof(uint64_t), 16);
        return cudaSuccess;
    }
    if (tmp_bytes < scan_tmp_words(n) * sizeof(uint64_t)) return cudaErrorInvalidValue;
    return scan_u64_levels(in, out, n, reinterpret_cast<uint64_t *>(tmp), st);
}

template <class T>
cudaError_t launch_encode_tiles(const EncStream *streams, uint32_t ns, const uint64_t *toff, uint64_t ntiles, uint64_t *tile_state,
                                uint64_t *err, cudaStream_t st) {
    if (ntiles == 0) return cudaSuccess;
    cudaError_t e;
    constexpr uint32_t kTile = enc_tile<T>();
    const int smem = (int)(2 * (kTile + kEncThreads) * sizeof(T) + (kTile + 2) * sizeof(uint32_t));
    e = cudaFuncSetAttribute(encode_tiles_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return e;
    const unsigned grid = (unsigned)std::min<uint64_t>(ntiles, 148 * 4);
    encode_tiles_kernel<T><<<grid, kEncThreads, smem, st>>>(streams, ns, toff, ntiles, (unsigned long long *)tile_state,
                                                            (unsigned long long *)err);
    count_launch();
    return cudaGetLastError();
}

template cudaError_t launch_encode_tiles<int32_t>(const EncStream *, uint32_t, const uint64_t *, uint64_t, uint64_t *, uint64_t *,
                                                  cudaStream_t);
template cudaError_t launch_encode_tiles<int64_t>(const EncStream *, uint32_t, const uint64_t *, uint64_t, uint64_t *, uint64_t *,
                                                  cudaStream_t);

// Persistent decode grid: 4 CTAs of 256 threads per SM, each with a tile's payload and a table of up to
// 16 KB. With a table of 12 bits the synchronising kernel, which has its marks beside them, takes 58,464
// bytes a CTA, and three of them an SM: the last 148 CTAs follow the others.
static unsigned decode_grid(uint64_t ntiles) { return (unsigned)(ntiles < 148 * 4 ? (ntiles ? ntiles : 1) : 148 * 4); }
static size_t decode_smem(uint32_t max_lut_bits) {
    return kDecodeSlotBytes + std::max<size_t>(((size_t)1 << max_lut_bits) * 4, 16);
}
constexpr uint32_t kDecodeLutBits = 12;  // a table's most; the kernels' limit is one for all threads and streams

cudaError_t launch_decode_sync(const uint8_t *base, const DecStream *streams, const uint32_t *tile_stream,
                               uint64_t ntiles, uint32_t max_lut_bits, const uint32_t *luts, const uint32_t *lut2s,
                               const uint32_t *childs,
                               int first_pass, uint64_t *start, uint64_t *end, uint64_t *count, const uint32_t *moved,
                               uint32_t *err, cudaStream_t st) {
    if (max_lut_bits > kDecodeLutBits) return cudaErrorInvalidValue;
    const size_t sh = decode_smem(max_lut_bits);
    const cudaError_t e =
        cudaFuncSetAttribute(decode_sync_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)decode_smem(kDecodeLutBits));
    if (e != cudaSuccess) return e;
    decode_sync_kernel<<<decode_grid(ntiles), kDecodeThreads, sh, st>>>(base, streams, tile_stream, ntiles, luts, lut2s,
                                                                      childs, first_pass, start, end, count, moved, err);
    count_launch();
    return cudaGetLastError();
}

cudaError_t launch_decode_restart(const DecStream *streams, uint32_t nstreams, uint64_t nchunks, const uint64_t *end,
                                  uint64_t *start, uint32_t *moved, uint32_t *changed, cudaStream_t st) {
    const uint64_t b = (nchunks + 255) / 256;
    decode_restart_kernel<<<(unsigned)(b < 148 * 8 ? (b ? b : 1) : 148 * 8), 256, 0, st>>>(streams, nstreams, nchunks, end, start,
                                                                                         moved, changed);
    count_launch();
    return cudaGetLastError();
}

cudaError_t launch_decode_check(const DecStream *streams, uint32_t nstreams, const uint32_t *tile_stream, uint64_t ntiles,
                                const uint64_t *off, const uint64_t *start, const uint64_t *end, uint32_t *err,
                                uint32_t *changed, cudaStream_t st) {
    const uint64_t n = std::max<uint64_t>(ntiles * (kDecodeThreads / 32), nstreams);
    decode_check_kernel<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(streams, nstreams, tile_stream, ntiles, off, start, end, err,
                                                                      changed);
    count_launch();
    return cudaGetLastError();
}

cudaError_t launch_decode_write(const uint8_t *base, const DecStream *streams, const uint32_t *tile_stream,
                                uint64_t ntiles, uint32_t max_lut_bits, const uint32_t *luts, const uint32_t *lut2s,
                               const uint32_t *childs,
                                const uint64_t *start, const uint64_t *off, uint32_t *err, cudaStream_t st) {
    if (max_lut_bits > kDecodeLutBits) return cudaErrorInvalidValue;
    const size_t sh = decode_smem(max_lut_bits);
    const cudaError_t e =
        cudaFuncSetAttribute(decode_write_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)decode_smem(kDecodeLutBits));
    if (e != cudaSuccess) return e;
    decode_write_kernel<<<decode_grid(ntiles), kDecodeThreads, sh, st>>>(base, streams, tile_stream, ntiles, luts, lut2s, childs,
                                                                       start, off, err);
    count_launch();
    return cudaGetLastError();
}

template <class T>
cudaError_t launch_fill(T *out, uint64_t n, T v, cudaStream_t st) {
    if (n == 0) return cudaSuccess;
    uint64_t blocks = std::min<uint64_t>((n + 255) / 256, 148 * 16);
    fill_kernel<T><<<(unsigned)blocks, 256, 0, st>>>(out, n, v);
    count_launch();
    return cudaGetLastError();
}

template cudaError_t launch_histogram<int32_t>(const int32_t *, uint64_t, int64_t, uint64_t, unsigned long long *, cudaStream_t);
template cudaError_t launch_histogram<int64_t>(const int64_t *, uint64_t, int64_t, uint64_t, unsigned long long *, cudaStream_t);
template cudaError_t launch_fill<int32_t>(int32_t *, uint64_t, int32_t, cudaStream_t);
template cudaError_t launch_fill<int64_t>(int64_t *, uint64_t, int64_t, cudaStream_t);

}  // namespace asz
