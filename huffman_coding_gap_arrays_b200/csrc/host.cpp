// host.cpp -- host-side half of the path: codebook construction, the
// encoder/decoder tables the kernels take as launch parameters, and the
// container format.  Pure C++ (no CUDA calls).
#include <cstring>

#include "hgap_internal.h"

namespace {

// The present bytes by ascending count, ties in byte order: key = count << 8 |
// byte.  Radix sort by the counts' bytes (stable, and a histogram's keys come in
// byte order); returns their number.
uint32_t sorted_keys(const uint32_t hist[256], uint64_t key[256]) {
    uint64_t tmp[256];
    uint32_t n = 0, all = 0;
    for (uint32_t b = 0; b < 256; ++b) {
        key[n] = ((uint64_t)hist[b] << 8) | b;
        n += hist[b] != 0;
        all |= hist[b];
    }
    for (int shift = 8; shift < 40 && (all >> (shift - 8)) != 0; shift += 8) {
        uint32_t at[256] = {};
        for (uint32_t i = 0; i < n; ++i) ++at[(key[i] >> shift) & 0xff];
        uint32_t sum = 0;
        for (uint32_t d = 0; d < 256; ++d) {
            const uint32_t c = at[d];
            at[d] = sum;
            sum += c;
        }
        for (uint32_t i = 0; i < n; ++i) tmp[at[(key[i] >> shift) & 0xff]++] = key[i];
        std::memcpy(key, tmp, n * sizeof(uint64_t));
    }
    return n;
}

// Length-limited (16-bit) code lengths by package-merge, with the
// reference's tie rule: a package precedes a leaf of equal weight
// (encoder/src/package_merge.cpp:37,52,136).  `leaf` holds n >= 2 weights,
// ascending.  Level 1 is the leaf list; level l merges the leaves with the
// pairwise packages of level l-1 and keeps 2n-2 items.  Walking down from the
// top, the leaves inside each level's active prefix gain one bit, and the
// packages in it make the next level's active prefix twice as long; the leaves
// in a prefix are counted by what the merge noted, how many leaves precede each
// item.
// A merge is a chain of dependent steps (compare, advance, load), so each level
// is cut into kCuts pieces whose starts a binary search finds, and the pieces
// are merged side by side: 256 leaves in 9 us where one chain over pushed-back
// vectors took 40.
void package_merge(const uint64_t* leaf, int n, uint8_t* len) {
    constexpr int kCuts = 4, kMaxItems = 512;
    constexpr uint64_t kNone = ~0ull;
    const int keep = 2 * n - 2;
    uint64_t leaves[256 + 1], w[kMaxItems + 2], pk[kMaxItems / 2 + 1];
    uint16_t before[hgap::kMaxLen + 1][kMaxItems + 1];  // [level][k]: leaves among the level's first k items
    int size[hgap::kMaxLen + 1];
    std::memcpy(leaves, leaf, n * sizeof(uint64_t));
    leaves[n] = kNone;
    std::memcpy(w, leaf, n * sizeof(uint64_t));
    for (int k = 0; k <= n; ++k) before[1][k] = (uint16_t)k;
    size[1] = n;
    for (int l = 2; l <= hgap::kMaxLen; ++l) {
        const int np = size[l - 1] / 2;
        for (int j = 0; j < np; ++j) pk[j] = w[2 * j] + w[2 * j + 1];
        pk[np] = kNone;
        const int m = keep < n + np ? keep : n + np;
        const int step = (m + kCuts - 1) / kCuts;
        // leaves among the first d items: leaf i precedes package j iff its weight is smaller
        int li[kCuts], pi[kCuts];
        for (int c = 0; c < kCuts; ++c) {
            const int d = c * step < m ? c * step : m;
            int lo = d > np ? d - np : 0, hi = d < n ? d : n;
            while (lo < hi) {
                const int mid = (lo + hi) >> 1;
                if (leaves[mid] < pk[d - mid - 1]) lo = mid + 1;
                else hi = mid;
            }
            li[c] = lo;
            pi[c] = d - lo;
        }
        uint16_t* const bf = before[l];
        auto one = [&](int c, int k) {
            const uint64_t a = pk[pi[c]], b = leaves[li[c]];
            bf[k] = (uint16_t)li[c];
            const int take = a <= b;  // (whichever list has run out is kNone there: the other goes on)
            w[k] = take ? a : b;
            pi[c] += take;
            li[c] += 1 - take;
        };
        const int full = m - (kCuts - 1) * step;  // the last piece's items
        int k = 0;
        for (; k < full; ++k)
#pragma GCC unroll 4
            for (int c = 0; c < kCuts; ++c) one(c, c * step + k);
        for (; k < step; ++k)
            for (int c = 0; c < kCuts; ++c)
                if (c * step + k < m) one(c, c * step + k);
        int leaves_in = 0;
        for (int c = 0; c < kCuts; ++c)
            if (c * step < m) leaves_in = li[c];
        bf[m] = (uint16_t)leaves_in;
        size[l] = m;
    }
    std::memset(len, 0, n);
    int active = keep;
    for (int l = hgap::kMaxLen; l >= 1 && active > 0; --l) {
        if (active > size[l]) active = size[l];
        const int nleaf = before[l][active];
        for (int i = 0; i < nleaf; ++i) len[i]++;
        active = 2 * (active - nleaf);
    }
}

// Canonical codes from a container-order list (encoder/src/package_merge.cpp:168-181).
hgap_status assign_codes(hgap_codebook* cb) {
    std::memset(cb->table, 0, sizeof(cb->table));
    uint64_t kraft = 0;  // in units of 2^-16
    uint32_t code = 0;
    bool seen[256] = {};
    for (uint32_t i = 0; i < cb->symbol_count; ++i) {
        const uint32_t l = cb->symbols[i].length;
        const uint8_t s = cb->symbols[i].symbol;
        if (l < 1 || l > (uint32_t)hgap::kMaxLen || seen[s]) return HGAP_ERR_CORRUPT;
        seen[s] = true;
        const uint32_t nl = i + 1 < cb->symbol_count ? cb->symbols[i + 1].length : l;
        if (nl < l) return HGAP_ERR_CORRUPT;
        kraft += 1ull << (hgap::kMaxLen - l);
        cb->table[s].code = code;
        cb->table[s].length = l;
        code = (code + 1) << (nl - l);
    }
    if (kraft > (1ull << hgap::kMaxLen)) return HGAP_ERR_CORRUPT;
    return HGAP_OK;
}

}  // namespace

namespace hgap {

void make_enc_table(const hgap_codebook& cb, EncTable* t) {
    for (int b = 0; b < 256; ++b) {
        const uint32_t l = cb.table[b].length;
        t->e[b] = l ? ((cb.table[b].code & 0xffffu) | (l << 16)) : kEncAbsent;
    }
}

// Level-1 / level-2 tables of the decoder (layout in hgap_internal.h).  The
// level-1 boundary is the first prefix of a long code taken from the code
// itself -- the value the reference's get_twolevel_table computes
// (decoder/src/get_table.cpp:93-95) -- not the next symbol's code that its
// get_table_info uses (get_table.cpp:20).  A complete book (Kraft sum 1, what
// package-merge builds) needs at most 2368 level-2 entries: a prefix whose
// longest code has w extra bits is split by at least w+1 codes, so 256 codes
// give at most 36 prefixes of 2^6 entries and a remainder.
hgap_status make_dec_table(const hgap_codebook& cb, DecTable* t) {
    constexpr int P = kDecPrefix;
    for (int i = 0; i < (1 << P); ++i) t->t1[i] = kDecInvalid;
    for (int i = 0; i < kDecT2Cap; ++i) t->t2[i] = kDecInvalid;
    const uint32_t n = cb.symbol_count;
    uint32_t i = 0, t2off = 0;
    while (i < n) {
        const uint8_t sym = cb.symbols[i].symbol;
        const uint32_t l = cb.symbols[i].length;
        const uint32_t code = cb.table[sym].code;
        if (l <= (uint32_t)P) {
            const uint16_t e = (uint16_t)(((l - 1) << 8) | sym);
            const uint32_t first = code << (P - l), cnt = 1u << (P - l);
            for (uint32_t k = 0; k < cnt; ++k) t->t1[first + k] = e;
            ++i;
            continue;
        }
        // run of longer codes sharing this prefix; lengths ascend, so the
        // last one sets the level-2 width
        const uint32_t prefix = code >> (l - P);
        uint32_t j = i, width = 0;
        while (j < n) {
            const uint32_t lj = cb.symbols[j].length;
            if ((cb.table[cb.symbols[j].symbol].code >> (lj - P)) != prefix) break;
            width = lj - P;
            ++j;
        }
        if (t2off + (1u << width) > (uint32_t)kDecT2Cap) return HGAP_ERR_UNSUPPORTED;
        t->t1[prefix] = (uint16_t)(0x8000u | (width << 12) | t2off);
        for (uint32_t k = i; k < j; ++k) {
            const uint8_t sk = cb.symbols[k].symbol;
            const uint32_t lk = cb.symbols[k].length;
            const uint32_t sfx = cb.table[sk].code & ((1u << (lk - P)) - 1u);
            const uint32_t first = sfx << (width - (lk - P)), cnt = 1u << (width - (lk - P));
            const uint16_t e = (uint16_t)(((lk - 1) << 8) | sk);
            for (uint32_t m = 0; m < cnt; ++m) t->t2[t2off + first + m] = e;
        }
        t2off += 1u << width;
        i = j;
    }
    return HGAP_OK;
}

// From the numbers of codes of each length: a window of a pair has a first code
// of l1 bits, a second of l2, and any 11 - l1 - l2 bits after them.
double dec_pair_fraction(const hgap_codebook& cb) {
    constexpr uint32_t P = kDecPrefix;
    uint32_t of[kMaxLen + 1] = {}, pairs = 0;
    for (uint32_t i = 0; i < cb.symbol_count; ++i) ++of[cb.symbols[i].length];
    for (uint32_t l1 = 1; l1 < P; ++l1)
        for (uint32_t l2 = 1; l1 + l2 <= P; ++l2) pairs += (of[l1] * of[l2]) << (P - l1 - l2);
    return pairs / double(1u << P);
}

DecIndex dec_index_of(const hgap_codebook& cb, bool complete, int rows) {
    uint32_t first_long = 0, max_len = 0;
    const uint32_t P = dec_prefix(rows);
    for (uint32_t i = 0; i < cb.symbol_count; ++i) {
        const uint32_t l = cb.symbols[i].length;
        if (l <= P) first_long += 1u << (P - l);
        if (l > max_len) max_len = l;
    }
    return dec_index(first_long, max_len, complete, rows);
}

}  // namespace hgap

extern "C" {

const char* hgap_status_string(hgap_status s) {
    switch (s) {
        case HGAP_OK: return "ok";
        case HGAP_ERR_INVALID_ARG: return "invalid argument";
        case HGAP_ERR_CUDA: return "CUDA runtime error";
        case HGAP_ERR_TIMEOUT: return "device wait timed out";
        case HGAP_ERR_CORRUPT: return "corrupt stream, gap array or codebook";
        case HGAP_ERR_SIZE: return "size mismatch";
        case HGAP_ERR_WORKSPACE: return "workspace too small";
        case HGAP_ERR_NO_CODE: return "input byte without a codeword";
        case HGAP_ERR_UNSUPPORTED: return "unsupported";
    }
    return "unknown status";
}

hgap_sizes hgap_sizes_from_bits(uint64_t bits) {
    hgap_sizes z;
    z.bits = bits;
    z.words = (bits + 31) / 32;
    z.segments = (bits + HGAP_SEGMENT_BITS - 1) / HGAP_SEGMENT_BITS;
    z.gap_words = (z.segments + HGAP_GAPS_PER_WORD - 1) / HGAP_GAPS_PER_WORD;
    return z;
}

uint64_t hgap_encoded_bits(const hgap_codebook* cb, const uint32_t hist[256]) {
    uint64_t bits = 0;
    for (int b = 0; b < 256; ++b) bits += (uint64_t)cb->table[b].length * hist[b];
    return bits;
}

// store_symbols (encoder/src/symbols.cpp:29-43) + qsort(compare)
// (encoder/src/huff.cpp:17-21, stable on glibc for this size, so ties stay in
// byte order) + boundary_PM (encoder/src/package_merge.cpp:107-182).
hgap_status hgap_codebook_build(const uint32_t hist[256], hgap_codebook* cb, hgap_sizes* sizes) {
    if (!hist || !cb) return HGAP_ERR_INVALID_ARG;
    std::memset(cb, 0, sizeof(*cb));
    uint64_t key[256], weight[256];
    const uint32_t n = sorted_keys(hist, key);
    for (uint32_t i = 0; i < n; ++i) weight[i] = key[i] >> 8;
    cb->symbol_count = n;
    uint8_t len[256];
    if (n == 1) {
        len[0] = 1;  // defined here; the reference is undefined (package_merge.cpp:113-132)
    } else if (n >= 2) {
        package_merge(weight, (int)n, len);
    }
    for (uint32_t i = 0; i < n; ++i) {  // container order: most frequent first (huff.cpp:114)
        cb->symbols[i].symbol = (uint8_t)key[n - 1 - i];
        cb->symbols[i].length = len[n - 1 - i];
    }
    const hgap_status st = assign_codes(cb);
    if (st != HGAP_OK) return st;
    if (sizes) *sizes = hgap_sizes_from_bits(hgap_encoded_bits(cb, hist));
    return HGAP_OK;
}

hgap_status hgap_codebook_from_symbols(const hgap_symlen* symbols, uint32_t count,
                                       hgap_codebook* cb) {
    if (!cb || count > 256 || (count && !symbols)) return HGAP_ERR_INVALID_ARG;
    std::memset(cb, 0, sizeof(*cb));
    cb->symbol_count = count;
    for (uint32_t i = 0; i < count; ++i) cb->symbols[i] = symbols[i];
    return assign_codes(cb);
}

hgap_status hgap_decode_table_build(const hgap_codebook* cb, uint16_t* t1, uint16_t* t2) {
    if (!cb || !t1 || !t2) return HGAP_ERR_INVALID_ARG;
    hgap_codebook book;
    if (cb->symbol_count > 256) return HGAP_ERR_CORRUPT;
    hgap_status st = hgap_codebook_from_symbols(cb->symbols, cb->symbol_count, &book);
    if (st != HGAP_OK) return st;
    if (book.symbol_count == 0) return HGAP_ERR_CORRUPT;
    hgap::DecTable t;
    st = hgap::make_dec_table(book, &t);
    if (st != HGAP_OK) return st;
    std::memcpy(t1, t.t1, sizeof(t.t1));
    std::memcpy(t2, t.t2, sizeof(t.t2));
    return HGAP_OK;
}

size_t hgap_container_bytes(uint32_t symbol_count, uint64_t words, uint64_t segments) {
    return 8 + 2 * (size_t)symbol_count + 12 + 4 * (size_t)((segments + 7) / 8) + 4 * (size_t)words;
}

hgap_status hgap_container_write(void* dst, size_t capacity, const hgap_codebook* cb, uint64_t n,
                                 uint64_t words, uint64_t segments, const uint32_t* gaps,
                                 const uint32_t* bits, size_t* written) {
    if (!dst || !cb) return HGAP_ERR_INVALID_ARG;
    if (n > 0xffffffffull || words > 0xffffffffull || segments > 0xffffffffull)
        return HGAP_ERR_UNSUPPORTED;  // the header fields are u32 (encoder/src/huff.cpp:121-123)
    const size_t need = hgap_container_bytes(cb->symbol_count, words, segments);
    if (capacity < need) return HGAP_ERR_SIZE;
    uint8_t* p = static_cast<uint8_t*>(dst);
    const uint64_t c64 = cb->symbol_count;
    std::memcpy(p, &c64, 8);
    p += 8;
    for (uint32_t i = 0; i < cb->symbol_count; ++i) {
        *p++ = cb->symbols[i].symbol;
        *p++ = cb->symbols[i].length;
    }
    const uint32_t hdr[3] = {(uint32_t)n, (uint32_t)words, (uint32_t)segments};
    std::memcpy(p, hdr, 12);
    p += 12;
    const size_t gw = (size_t)((segments + 7) / 8);
    if (gw) std::memcpy(p, gaps, 4 * gw);
    p += 4 * gw;
    if (words) std::memcpy(p, bits, 4 * (size_t)words);
    p += 4 * (size_t)words;
    if (written) *written = (size_t)(p - static_cast<uint8_t*>(dst));
    return HGAP_OK;
}

hgap_status hgap_container_parse(const void* src, size_t size, hgap_codebook* cb, uint64_t* n,
                                 uint64_t* words, uint64_t* segments, const void** gaps,
                                 const void** bits) {
    if (!src || !cb || !n || !words || !segments) return HGAP_ERR_INVALID_ARG;
    const uint8_t* p = static_cast<const uint8_t*>(src);
    if (size < 8) return HGAP_ERR_CORRUPT;
    uint64_t c64;
    std::memcpy(&c64, p, 8);
    if (c64 > 256) return HGAP_ERR_CORRUPT;
    size_t off = 8;
    if (size < off + 2 * c64 + 12) return HGAP_ERR_CORRUPT;
    hgap_symlen syms[256];
    for (uint64_t i = 0; i < c64; ++i) {
        syms[i].symbol = p[off + 2 * i];
        syms[i].length = p[off + 2 * i + 1];
    }
    off += 2 * c64;
    uint32_t hdr[3];
    std::memcpy(hdr, p + off, 12);
    off += 12;
    const uint64_t gw = ((uint64_t)hdr[2] + 7) / 8;
    if (size < off + 4 * gw + 4 * (uint64_t)hdr[1]) return HGAP_ERR_CORRUPT;
    if (hdr[2] != (hdr[1] + 3) / 4) return HGAP_ERR_CORRUPT;  // a segment is 4 words
    if ((hdr[0] == 0) != (hdr[1] == 0) || (hdr[0] && c64 == 0)) return HGAP_ERR_CORRUPT;
    const hgap_status st = hgap_codebook_from_symbols(syms, (uint32_t)c64, cb);
    if (st != HGAP_OK) return st;
    *n = hdr[0];
    *words = hdr[1];
    *segments = hdr[2];
    if (gaps) *gaps = p + off;
    if (bits) *bits = p + off + 4 * gw;
    return HGAP_OK;
}

}  // extern "C"
