// Host side of the Huffman stage (see huffman_host.h).
#include "huffman_host.h"

#include <algorithm>
#include <cstring>

#include <queue>
#include <utility>

namespace asz {

uint64_t HuffCode::save_size() const {
    uint64_t s = 1 + 8 + 8 + 8;
    if (n > 1) s += (n * (uint64_t)(mbft + 2) - 1 + 7) >> 3;
    return s;
}

uint64_t HuffCode::encode_size() const { return 8 + (maxval == 1 ? 0 : (bits + 7) >> 3); }

bool build_code(const std::vector<uint64_t> &hist, int64_t min_sym, int64_t max_sym, uint64_t count, bool wide,
                HuffCode &c, std::string &err) {
    c = HuffCode();
    c.count = count;
    c.offset = min_sym;
    // huffman.hpp:275-281: maxval = max-min+1 in the symbol type; the usemp flag only changes the
    // first header byte (the map and vector forms build the same tree).
    if (wide) {
        int64_t mv = (int64_t)((uint64_t)max_sym - (uint64_t)min_sym + 1);
        c.maxval = (uint64_t)mv;
        c.usemp = (mv >= (1 << 12) && count < 2ull * (uint64_t)max_sym) || mv >= (1 << 28);
    } else {
        int32_t mv = (int32_t)((uint32_t)(int32_t)max_sym - (uint32_t)(int32_t)min_sym + 1u);
        c.maxval = (uint64_t)(int64_t)mv;
        c.usemp = (mv >= (1 << 12) && count < 2ull * (uint64_t)(int64_t)(int32_t)max_sym) || mv >= (1 << 28);
    }
    std::vector<uint64_t> freq;
    for (uint64_t i = 0; i < hist.size(); i++)
        if (hist[i]) {
            c.leaf_sym.push_back(i);
            freq.push_back(hist[i]);
        }
    c.n = c.leaf_sym.size();
    if (c.n == 0) {
        err = "empty Huffman stream";
        return false;
    }
    c.table.assign(hist.size(), CodeEntry{0, 0});
    if (c.n == 1 || c.maxval == 1) {  // huffman.hpp:193-210
        c.mbft = 1;
        c.maxval = 1;
        c.offset = min_sym + (int64_t)c.leaf_sym[0];
        c.table[c.leaf_sym[0]] = CodeEntry{0, 1};
        c.max_len = 1;
        c.bits = 0;
        return true;
    }
    c.mbft = 1;
    while ((1ull << c.mbft) < c.maxval) ++c.mbft;
    const uint64_t n = c.n;
    c.left.assign(n, -1);
    c.right.assign(n, -1);
    // The reference pops a min-heap on (frequency, node index) (huffman.hpp:222-240). Merged
    // weights come out nondecreasing and internal nodes are numbered after all leaves, so the
    // leaves sorted by (frequency, index) and a FIFO of internal nodes in creation order give
    // the same pops: at each step take the smaller front, the leaf on a frequency tie.
    // Leaves in (frequency, index) order: a stable radix sort on the frequency, one byte per
    // pass over the bytes that are not zero in every frequency, from leaves in index order.
    std::vector<uint32_t> order(n), tmp(n);
    uint64_t maxf = 0;
    for (uint64_t i = 0; i < n; i++) {
        order[i] = (uint32_t)i;
        maxf = std::max(maxf, freq[i]);
    }
    for (unsigned shift = 0; shift < 64 && (maxf >> shift) != 0; shift += 8) {
        uint64_t cnt[257] = {0};
        for (uint64_t i = 0; i < n; i++) cnt[((freq[order[i]] >> shift) & 255u) + 1]++;
        for (int b = 0; b < 256; b++) cnt[b + 1] += cnt[b];
        for (uint64_t i = 0; i < n; i++) tmp[cnt[(freq[order[i]] >> shift) & 255u]++] = order[i];
        order.swap(tmp);
    }
    std::vector<uint64_t> ifreq;
    ifreq.reserve(n);
    uint64_t ia = 0, ib = 0;
    auto pop = [&](uint64_t &node, uint64_t &f) {
        if (ia < n && (ib == ifreq.size() || freq[order[ia]] <= ifreq[ib])) {
            node = order[ia];
            f = freq[order[ia]];
            ia++;
        } else {
            node = n + ib;
            f = ifreq[ib];
            ib++;
        }
    };
    for (uint64_t k = 0; k + 1 < n; k++) {
        uint64_t u, fu, v, fv;
        pop(u, fu);
        pop(v, fv);
        c.left.push_back((int32_t)u);
        c.right.push_back((int32_t)v);
        ifreq.push_back(fu + fv);
    }
    c.root = c.left.size() - 1;
    // dfs_vec (huffman.hpp:80-95): bit k of the code is the branch taken at depth k+1. A node's
    // children come before it, so one pass from the root down meets every parent first.
    struct Path {
        uint64_t code;
        uint32_t len;
    };
    std::vector<Path> path(n - 1);  // of the internal nodes
    path[c.root - n] = Path{0, 0};
    for (uint64_t k = c.root; k >= n; k--) {
        const Path p = path[k - n];
        if (p.len >= 32) {
            err = "Huffman code longer than 32 bits";
            return false;
        }
        const uint64_t child[2] = {(uint64_t)c.left[k], (uint64_t)c.right[k]};
        for (int i = 0; i < 2; i++) {
            const uint64_t code = p.code | (uint64_t)i << p.len;
            const uint32_t len = p.len + 1;
            if (child[i] >= n) {
                path[child[i] - n] = Path{code, len};
                continue;
            }
            c.table[c.leaf_sym[child[i]]] = CodeEntry{(uint32_t)code, len};
            c.max_len = std::max(c.max_len, len);
            c.bits += freq[child[i]] * len;
        }
    }
    return true;
}

static void put_be64(uint8_t *b, uint64_t v) {
    for (int i = 0; i < 8; i++) b[i] = (uint8_t)(v >> (56 - 8 * i));
}
static uint64_t get_be64(const uint8_t *b) {
    uint64_t v = 0;
    for (int i = 0; i < 8; i++) v = (v << 8) | b[i];
    return v;
}

void write_tree(const HuffCode &c, uint8_t *dst) {
    uint8_t *p = dst;
    *p++ = (uint8_t)((c.usemp ? 0x80 : 0) | (c.n == 1 ? 0x40 : 0) | c.mbft);
    uint64_t ob = (uint64_t)c.offset;
    for (int i = 0; i < 8; i++) *p++ = (uint8_t)(ob >> (8 * i));
    put_be64(p, c.n);
    p += 8;
    put_be64(p, c.maxval);
    p += 8;
    if (c.n <= 1) return;
    // Preorder: internal node -> 0, leaf -> 1 followed by mbft bits of its symbol, LSB-first; written
    // by 64-bit words.
    uint64_t word = 0;
    unsigned have = 0;
    auto put = [&](uint64_t v, unsigned n) {  // n <= 63
        word |= v << have;
        if (have + n < 64) {
            have += n;
            return;
        }
        std::memcpy(p, &word, 8);
        p += 8;
        word = have ? v >> (64 - have) : 0;
        have = have + n - 64;
    };
    std::vector<uint32_t> st{(uint32_t)c.root};
    while (!st.empty()) {
        uint32_t u = st.back();
        st.pop_back();
        unsigned inner = 0;
        for (; u >= c.n; inner++) {
            st.push_back((uint32_t)c.right[u]);
            u = (uint32_t)c.left[u];
        }
        for (; inner > 32; inner -= 32) put(0, 32);
        put(0, inner);
        put(1, 1);
        put(c.leaf_sym[u], c.mbft);
    }
    for (unsigned i = 0; i < have; i += 8) *p++ = (uint8_t)(word >> i);
}

void write_len_word(const HuffCode &c, uint8_t *dst) {
    put_be64(dst, (c.maxval == 1 ? c.count : c.bits) ^ 0x1234abcdull);
}

namespace {

// Bits of buf[0, len) by position, LSB-first.
struct TreeBits {
    const uint8_t *buf;
    uint64_t len, avail;
    uint64_t pos = 0;
    // The next n bits (n <= 63; false past the end).
    bool read(unsigned n, uint64_t &v) {
        if (pos + n > avail) return false;
        const uint64_t byte = pos >> 3;
        const unsigned sh = (unsigned)(pos & 7);
        if (byte + 9 <= len) {
            uint64_t w;
            std::memcpy(&w, buf + byte, 8);
            w >>= sh;
            if (sh) w |= (uint64_t)buf[byte + 8] << (64 - sh);
            v = w & ((1ull << n) - 1);
        } else {
            v = 0;
            for (unsigned j = 0; j < n; j++) v |= (uint64_t)((buf[(pos + j) >> 3] >> ((pos + j) & 7)) & 1) << j;
        }
        pos += n;
        return true;
    }
    // The number of zero bits before the next one, at most `most` + 1 of them, all consumed but the one.
    bool zeros(unsigned most, unsigned &count) {
        count = 0;
        uint64_t v;
        while (count <= most) {
            const unsigned n = (unsigned)std::min<uint64_t>(32, avail - pos);
            if (n == 0 || !read(n, v)) return false;
            const unsigned z = v ? (unsigned)__builtin_ctzll(v) : n;
            count += z;
            if (v) {
                pos -= n - z;
                return true;
            }
        }
        return true;
    }
};

constexpr uint32_t kLutBits = 12, kLut2Bits = 10, kLutValueBits = 27, kLut2Most = 1u << 20;

struct LongLeaf {
    uint32_t code, len, sym;
};

constexpr uint32_t lut_entry(uint32_t len, uint32_t v) { return len << kLutValueBits | v; }

// The second table, for the codes longer than the first one (in preorder, so those of one prefix lie
// together), and the first one's entries that lead there.
bool fill_lut2(const std::vector<LongLeaf> &leaves, uint32_t sub_bits, HuffParsed &o) {
    o.lut2.clear();
    for (size_t i = 0; i < leaves.size();) {
        const uint32_t prefix = leaves[i].code & ((1u << kLutBits) - 1);
        size_t j = i;
        uint32_t most = 0;
        for (; j < leaves.size() && (leaves[j].code & ((1u << kLutBits) - 1)) == prefix; j++) most = std::max(most, leaves[j].len);
        const uint32_t bits = std::min(most - kLutBits, sub_bits), off = (uint32_t)o.lut2.size();
        if (off + (1u << bits) > kLut2Most) return false;
        o.lut2.resize(off + (1u << bits));
        uint32_t *t = o.lut2.data() + off;
        for (; i < j; i++) {
            const LongLeaf &l = leaves[i];
            const uint32_t rest = l.code >> kLutBits, len = l.len - kLutBits;
            if (len <= bits) {
                for (uint32_t k = rest; k < (1u << bits); k += 1u << len) t[k] = lut_entry(l.len, l.sym);
            } else {  // the tree node after the table's bits
                uint32_t node = 0;
                for (uint32_t k = 0; k < kLutBits + bits; k++) node = o.child[2 * (size_t)node + ((l.code >> k) & 1)];
                t[rest & ((1u << bits) - 1)] = lut_entry(0, node);
            }
        }
        o.lut[prefix] = lut_entry(0, off << 4 | bits);
    }
    return true;
}

}  // namespace

bool parse_stream(const uint8_t *buf, uint64_t len, uint64_t &pos, HuffParsed &o, std::string &err) {
    o = HuffParsed();
    if (len - pos < 25 || pos > len) {
        err = "truncated Huffman header";
        return false;
    }
    const uint8_t *b = buf + pos;
    o.mbft = b[0] & 0x3f;
    uint64_t ob = 0;
    for (int i = 0; i < 8; i++) ob |= (uint64_t)b[1 + i] << (8 * i);
    o.offset = (int64_t)ob;
    o.n = get_be64(b + 9);
    o.maxval = get_be64(b + 17);
    pos += 25;
    if (o.n == 0) {
        err = "Huffman stream with no symbols";
        return false;
    }
    if (o.n > 1) {
        if (o.mbft == 0 || o.mbft > 63 || o.n > (1ull << 31)) {
            err = "corrupt Huffman tree header";
            return false;
        }
        // The tree from its preorder bits, starting after the root's bit: internal nodes in their
        // order, a leaf in its parent's branch. The open nodes are the path to the next one; `turn`
        // has its branches (bit d: the branch taken at depth d).
        TreeBits in{buf + pos, len - pos, (len - pos) * 8, 1};
        o.child.reserve(2 * std::min<uint64_t>(o.n, len));
        o.child.assign(2, 0);
        o.lut.assign(1u << kLutBits, 0);
        std::vector<LongLeaf> longer;
        std::vector<uint32_t> open{0};
        uint64_t turn = 0, leaves = 0, nodes = 1;
        uint32_t min_len = 64, max_len = 0;
        bool in_range = true, fits = true;
        while (!open.empty()) {
            unsigned inner;
            if (!in.zeros(48, inner)) {
                err = "truncated Huffman tree";
                return false;
            }
            for (unsigned k = 0; k < inner; k++) {  // each the first branch of the one before
                const uint32_t id = (uint32_t)(o.child.size() / 2), d = (uint32_t)open.size() - 1;
                if (++nodes > 2 * o.n + 1 || open.size() > 40) {
                    err = "corrupt Huffman tree";
                    return false;
                }
                o.child[2 * (size_t)open.back() + ((turn >> d) & 1)] = id;
                o.child.resize(o.child.size() + 2);
                open.push_back(id);
            }
            uint64_t one, sym;
            if (!in.read(1, one) || !in.read(o.mbft, sym)) {
                err = "truncated Huffman tree";
                return false;
            }
            const uint32_t d = (uint32_t)open.size() - 1, l = d + 1;
            if (++nodes > 2 * o.n + 1 || l > 40) {
                err = "corrupt Huffman tree";
                return false;
            }
            o.child[2 * (size_t)open.back() + ((turn >> d) & 1)] = 0x80000000u | (uint32_t)sym;
            leaves++;
            min_len = std::min(min_len, l);
            max_len = std::max(max_len, l);
            in_range = in_range && (sym < std::max<uint64_t>(o.maxval, 1) || o.maxval >= (1ull << 31));
            fits = fits && sym < (1ull << kLutValueBits);
            if (l <= kLutBits) {
                const uint32_t e = lut_entry(l, (uint32_t)sym & ((1u << kLutValueBits) - 1));
                for (uint32_t i = (uint32_t)turn; i < o.lut.size(); i += 1u << l) o.lut[i] = e;
            } else if (l <= 32) {
                longer.push_back({(uint32_t)turn, l, (uint32_t)sym});
            }
            // On to the second branch of the deepest node that has not had it.
            while (!open.empty() && (turn >> (open.size() - 1)) & 1) {
                turn &= ~(1ull << (open.size() - 1));
                open.pop_back();
            }
            if (!open.empty()) turn |= 1ull << (open.size() - 1);
        }
        if (leaves != o.n) {
            err = "Huffman tree does not match its symbol count";
            return false;
        }
        pos += (in.pos + 7) >> 3;
        if (max_len > 32) {
            err = "Huffman code longer than 32 bits";
            return false;
        }
        if (!in_range) {
            err = "Huffman symbol outside its range";
            return false;
        }
        o.min_len = min_len;
        o.max_len = max_len;
        o.lut_bits = std::min(max_len, kLutBits);
        o.lut.resize(1ull << o.lut_bits);  // a shorter table's entries are the first ones
        uint32_t sub = kLut2Bits;
        fits = fits && o.child.size() / 2 < (1ull << kLutValueBits);
        while (fits && !fill_lut2(longer, sub, o)) fits = sub-- > 0;
        if (!fits) {  // every code is walked from the root
            o.lut_bits = 0;
            o.lut.assign(1, lut_entry(0, 0));
            o.lut2.assign(1, lut_entry(0, 0));
        }
        if (o.lut2.empty()) o.lut2.assign(1, 0);
    } else {
        o.single = true;
    }
    if (len - pos < 8) {
        err = "truncated Huffman payload";
        return false;
    }
    uint64_t w = get_be64(buf + pos) ^ 0x1234abcdull;
    pos += 8;
    if (o.single || o.maxval == 1) {
        o.single = true;
        o.single_count = w;
        o.payload_off = pos;
        return true;
    }
    // Compare in bits first: a corrupt length near 2^64 must not wrap when rounded up to bytes.
    if (w > (len - pos) * 8) {
        err = "truncated Huffman payload";
        return false;
    }
    o.payload_bits = w;
    o.payload_off = pos;
    uint64_t bytes = (w + 7) >> 3;
    if (bytes > len - pos) {
        err = "truncated Huffman payload";
        return false;
    }
    pos += bytes;
    return true;
}

}  // namespace asz
