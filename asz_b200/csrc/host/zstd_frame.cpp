#include "zstd_frame.h"

#include <algorithm>
#include <cstring>
#include <vector>

#include "stream_copy.h"

// A Huffman payload does not compress any further, so most of a stream's blocks are stored. libzstd
// copies them one after the other on one thread (109 MB of a 512^3 field at 1e-3: 11.7 ms); their places
// are known from the headers alone, so they are collected and copied in parallel. The others go through
// libzstd's block functions, in order and when all before them is in place, since their matches reach
// back into it; ZSTD_insertBlock tells it about the blocks it has not seen.
namespace asz::host {

namespace {

constexpr size_t kMaxBlock = 128 << 10;
constexpr size_t kPiece = 512 << 10;  // a thread's share of a parallel copy, about
constexpr size_t kReady = 8 << 20;    // stored bytes that are copied at a time

struct Copy {
    uint8_t *to;
    const uint8_t *from;  // nullptr: `n` times `fill`
    size_t n;
    uint8_t fill;
};

uint64_t le(const uint8_t *p, unsigned n) {
    uint64_t v = 0;
    for (unsigned i = 0; i < n; i++) v |= (uint64_t)p[i] << (8 * i);
    return v;
}

}  // namespace

bool unframe(ZSTD_DCtx *z, const uint8_t *in, size_t len, uint8_t *dst, size_t raw, const ParallelRun &run,
             const std::function<bool(size_t)> &ready) {
    if (!z || len < 6 || le(in, 4) != 0xFD2FB528u) return false;
    const uint8_t fhd = in[4];
    const bool single = fhd & 0x20;
    if (fhd & 0x0f) return false;  // reserved bit, checksum, dictionary
    size_t at = 5;
    uint64_t window = 0;
    if (!single) {
        const unsigned log = 10 + (in[at] >> 3);
        if (log > 31) return false;
        window = (1ull << log) + ((1ull << log) >> 3) * (in[at] & 7);
        at++;
    }
    const unsigned fcs = (fhd >> 6) ? 1u << (fhd >> 6) : single ? 1u : 0u;
    if (fcs == 0 || len - at < fcs) return false;
    const uint64_t content = le(in + at, fcs) + (fcs == 2 ? 256 : 0);
    at += fcs;
    if (content != raw) return false;
    if (single) window = content;
    const size_t most = (size_t)std::min<uint64_t>(window, kMaxBlock);
    if (ZSTD_isError(ZSTD_decompressBegin(z))) return false;

    std::vector<Copy> todo;
    size_t pos = 0, stored = 0;  // written or collected so far; bytes of todo
    auto flush = [&] {
        if (todo.empty()) return true;
        // Shares of whole entries, of about kPiece bytes.
        std::vector<size_t> first{0};
        for (size_t i = 0, n = 0; i < todo.size(); i++) {
            n += todo[i].n;
            if (n >= kPiece || i + 1 == todo.size()) {
                first.push_back(i + 1);
                n = 0;
            }
        }
        run(first.size() - 1, [&](uint64_t k) {
            for (size_t i = first[k]; i < first[k + 1]; i++) {
                const Copy &c = todo[i];
                if (c.from) stream_copy(c.to, c.from, c.n);
                else std::memset(c.to, c.fill, c.n);
            }
        });
        todo.clear();
        stored = 0;
        return ready(pos);
    };
    for (bool last = false; !last;) {
        if (len - at < 3) return false;
        const uint32_t h = (uint32_t)le(in + at, 3);
        at += 3;
        last = h & 1;
        const unsigned type = (h >> 1) & 3;
        const size_t n = h >> 3;
        if (n > most || type == 3) return false;
        if (type == 2) {
            if (len - at < n || !flush()) return false;
            const size_t got = ZSTD_decompressBlock(z, dst + pos, raw - pos, in + at, n);
            if (ZSTD_isError(got) || got > most) return false;
            at += n;
            pos += got;
            continue;
        }
        const size_t take = type == 1 ? 1 : n;
        if (len - at < take || raw - pos < n) return false;
        if (n) {
            todo.push_back(Copy{dst + pos, type == 1 ? nullptr : in + at, n, take ? in[at] : (uint8_t)0});
            ZSTD_insertBlock(z, dst + pos, n);
            stored += n;
        }
        at += take;
        pos += n;
        if (stored >= kReady && !flush()) return false;
    }
    if (at != len || pos != raw || !flush()) return false;
    return ready(raw);
}

}  // namespace asz::host
