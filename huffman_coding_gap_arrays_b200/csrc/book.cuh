// book.cuh -- codebook construction on the device, one warp per book.
//
// Replaces the host round trip of store_symbols + qsort + boundary_PM +
// canonical code assignment (encoder/src/symbols.cpp:29-55,
// encoder/src/huff.cpp:17-21, encoder/src/package_merge.cpp:107-182) and the
// decoder's table build (decoder/src/get_table.cpp:48-139), so that batched
// and serving callers build thousands of books without leaving the GPU.  The
// results are identical to the host builder's (host.cpp): the same stable
// order by count, the same package-merge tie rule, the same canonical codes
// and the same two-level decoder table.
//
//   * sort: bitonic sort of (count << 8 | byte) keys in registers, eight a
//     lane, so equal counts keep byte order (what the reference's qsort yields
//     on glibc);
//   * package-merge, L = 16: level l merges the sorted leaves with the pairwise
//     packages of level l-1 (a package first on equal weight), keeping 2n-2
//     items; each level is one merge-path step -- every lane finds where its
//     16 outputs start by a binary search on its diagonal, then merges them
//     with one load a step, of whichever list it advanced (a book is a serial
//     chain on one warp: 58 us while every step loaded the heads of both lists
//     and summed a package); a 16-bit mask per lane records which items are
//     packages;
//   * lengths: walking down from level 16, the packages in a level's active
//     prefix make the next level's active prefix twice as long; a leaf's
//     length is the number of levels whose active prefix holds it;
//   * canonical codes: in container order (most frequent first) the code of
//     symbol i is the Kraft prefix sum before it, in units of 2^-16, shifted
//     down to its length -- the closed form of code = (code + 1) << (l' - l)
//     (encoder/src/package_merge.cpp:168-181);
//   * decoder table: every level-1 prefix, and every level-2 suffix of a
//     prefix whose codes are longer than kDecPrefix bits, looks up the
//     symbol whose left-aligned code is the largest not above it (canonical
//     codes ascend in container order); the lane walks its 64 prefixes in
//     order, so the search is a forward scan.
#pragma once

#include "device_util.cuh"

namespace hgap {

// The package-merge lanes read items 16 apart (weights) and about 8 apart
// (leaves): unpadded, a whole warp's reads land in one or two banks (the
// capture of one-warp-per-book showed two thirds of its shared wavefronts were
// conflicts).  One pad slot per 16 weights and per 8 keys spreads them.
__device__ __forceinline__ uint32_t wpad(uint32_t i) { return i + (i >> 4); }
__device__ __forceinline__ uint32_t kpad(uint32_t i) { return i + (i >> 3); }

// A book's symbols in container order: what the decoder's side needs.
struct BookSyms {
    uint32_t la[256];             // code << (16 - length)
    uint8_t sym[256];             // bytes
    uint8_t clen[256];            // lengths
    uint32_t seen[8];             // bitmap of the bytes (warp_load_symbols)
};

// W: 32-bit weights where the counts' sum is below kBook32, 64-bit otherwise.  A
// package's weight is at most 15 times that sum, and a key is count << 8 | byte
// (the largest stands for an absent byte).
template <class W>
struct BookScratch {
    union {
        W w[512 + 32];            // weights of one package-merge level (at wpad)
        BookSyms syms;            // the result, once the weights are done with
    };
    W leaf[256 + 32 + 2];         // leaf weights, ascending (at kpad), then ~0
    W pack[256 + 32 + 2];         // the level's packages (at kpad), then ~0
    uint16_t pk[kMaxLen + 1][32]; // bit b of pk[l][q]: item 16q+b of level l is a package
    uint16_t size[kMaxLen + 1];   // items kept at each level
    uint8_t order[256];           // ascending-count order: bytes
    uint8_t len[256];             // ascending-count order: code lengths
    uint8_t blen[256];            // per byte: code length (0: absent)
};
constexpr uint64_t kBook32 = (1u << 24) - 1;

__device__ __forceinline__ uint32_t warp_excl_scan(uint32_t v, uint32_t lane, uint32_t* total) {
    const uint32_t incl = warp_incl_scan(v, lane);
    *total = __shfl_sync(kFull, incl, 31);
    return incl - v;
}

// Sorts 256 keys, eight a lane (element 8 * lane + r in k[r]), ascending.
template <class W>
__device__ __forceinline__ void warp_sort256(W (&k)[8], uint32_t lane) {
#pragma unroll
    for (uint32_t size = 2; size <= 256; size <<= 1) {
#pragma unroll
        for (uint32_t j = size >> 1; j > 0; j >>= 1) {
            if (j >= 8) {  // partners in another lane
#pragma unroll
                for (int r = 0; r < 8; ++r) {
                    const W o = __shfl_xor_sync(kFull, k[r], j >> 3);
                    const bool up = ((8 * lane) & size) == 0, low = ((8 * lane) & j) == 0;
                    k[r] = (up == low) == (o < k[r]) ? o : k[r];
                }
            } else {
#pragma unroll
                for (int r = 0; r < 8; ++r) {
                    if (r & j) continue;
                    const bool up = size >= 8 ? ((8 * lane) & size) == 0 : (r & size) == 0;
                    const W x = k[r], y = k[r + j];
                    const bool swap = (y < x) == up;
                    k[r] = swap ? y : x;
                    k[r + j] = swap ? x : y;
                }
            }
        }
    }
}

// Fills s.order and s.len for the present bytes of `hist` and returns their
// number n (leaf r: ascending count, ties by byte).
template <class W>
__device__ inline uint32_t warp_code_lengths(const uint32_t* hist, BookScratch<W>& s, uint32_t lane) {
    uint32_t n = 0;
    {
        W k[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const uint32_t b = lane + 32 * j;
            const uint32_t h = hist[b];
            k[j] = h ? (((W)h << 8) | b) : ~(W)0;  // absent bytes sink to the end
            n += __popc(__ballot_sync(kFull, h != 0));
        }
        warp_sort256(k, lane);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const uint32_t r = 8 * lane + j;
            s.order[r] = (uint8_t)k[j];
            s.leaf[kpad(r)] = r < n ? k[j] >> 8 : ~(W)0;
            if (r < n) s.w[wpad(r)] = k[j] >> 8;
        }
        if (lane == 0) s.leaf[kpad(256)] = ~(W)0;
    }
    __syncwarp();
    if (n == 1) {
        if (lane == 0) s.len[0] = 1;  // one symbol: a 1-bit code (the reference is undefined here)
        __syncwarp();
        return n;
    }
    if (n < 2) return n;

    const uint32_t keep = 2 * n - 2;
    s.pk[1][lane] = 0;
    if (lane == 0) s.size[1] = (uint16_t)n;
    uint32_t prev_size = n;
    for (int l = 2; l <= kMaxLen; ++l) {
        const uint32_t np = prev_size / 2;
        const uint32_t m = keep < n + np ? keep : n + np;
#pragma unroll
        for (uint32_t t = 0; t < 8; ++t) {
            const uint32_t j = lane + 32 * t;
            if (j < np) s.pack[kpad(j)] = s.w[wpad(2 * j)] + s.w[wpad(2 * j + 1)];
        }
        if (lane == 0) s.pack[kpad(np)] = ~(W)0;
        __syncwarp();  // the packages are made: w is free for this level's items
        const uint32_t d = 16 * lane;
        uint32_t mask = 0;
        if (d < m) {
            // leaves among the first d items: leaf i precedes package j iff w(leaf i) < w(package j)
            uint32_t lo = d > np ? d - np : 0, hi = d < n ? d : n;
            while (lo < hi) {
                const uint32_t mid = (lo + hi) >> 1;
                if (s.leaf[kpad(mid)] < s.pack[kpad(d - mid - 1)]) lo = mid + 1;
                else hi = mid;
            }
            uint32_t i = lo, j = d - lo;
            W lw = s.leaf[kpad(i)], pw = s.pack[kpad(j)];
            const uint32_t cnt = m - d < 16 ? m - d : 16u;
            W* const out = s.w + wpad(d);  // (16 items between two pad slots)
#pragma unroll
            for (uint32_t pos = 0; pos < 16; ++pos) {
                if (pos >= cnt) break;
                const bool take = pw <= lw;  // (the list that has run out is ~0)
                out[pos] = take ? pw : lw;
                mask |= (uint32_t)take << pos;
                i += !take;
                j += take;
                const W next = *(take ? s.pack + kpad(j) : s.leaf + kpad(i));
                lw = take ? lw : next;
                pw = take ? next : pw;
            }
        }
        s.pk[l][lane] = (uint16_t)mask;
        if (lane == 0) s.size[l] = (uint16_t)m;
        prev_size = m;
        __syncwarp();
    }
    // walk down: leaves in each level's active prefix gain one bit
    uint32_t nleaf[kMaxLen + 1];
    uint32_t active = keep;
#pragma unroll
    for (int l = kMaxLen; l >= 1; --l) {
        const uint32_t a = active < s.size[l] ? active : s.size[l];
        const uint32_t q = a >> 4, rb = a & 15;
        uint32_t c = 0;
        if (lane < q) c = __popc(s.pk[l][lane]);
        else if (lane == q && rb) c = __popc(s.pk[l][lane] & ((1u << rb) - 1u));
        c = __reduce_add_sync(kFull, c);
        nleaf[l] = a - c;
        active = 2 * c;
    }
    for (uint32_t r = lane; r < n; r += 32) {
        uint32_t L = 0;
#pragma unroll
        for (int l = 1; l <= kMaxLen; ++l) L += nleaf[l] > r;
        s.len[r] = (uint8_t)L;
    }
    __syncwarp();
    return n;
}

// Container order from ascending order (symbol i = leaf n-1-i) and the
// canonical codes, into s.syms, plus the per-byte lengths s.blen.  Returns the
// Kraft sum in units of 2^-16 (65536: a complete book).
template <class W>
__device__ inline uint32_t warp_assign_codes(BookScratch<W>& s, uint32_t n, uint32_t lane) {
    for (uint32_t b = lane; b < 256; b += 32) s.blen[b] = 0;
    __syncwarp();
    uint32_t kr[8], tot = 0;
#pragma unroll
    for (int t = 0; t < 8; ++t) {
        const uint32_t c = 8 * lane + t;
        kr[t] = 0;
        if (c < n) {
            const uint32_t r = n - 1 - c;
            const uint32_t L = s.len[r];
            const uint32_t sym = s.order[r];
            s.syms.sym[c] = (uint8_t)sym;
            s.syms.clen[c] = (uint8_t)L;
            s.blen[sym] = (uint8_t)L;
            kr[t] = 1u << (kMaxLen - L);
        }
        tot += kr[t];
    }
    uint32_t kraft = 0;
    uint32_t run = warp_excl_scan(tot, lane, &kraft);
#pragma unroll
    for (int t = 0; t < 8; ++t) {
        const uint32_t c = 8 * lane + t;
        if (c < n) s.syms.la[c] = run;
        run += kr[t];
    }
    __syncwarp();
    return kraft;
}

// The book in the public layout (symbols in container order, per-byte table).
__device__ inline void warp_write_book(const BookSyms& s, uint32_t n, hgap_codebook* cb, uint32_t lane) {
    for (uint32_t b = lane; b < 256; b += 32) {
        cb->table[b].code = 0;
        cb->table[b].length = 0;
    }
    __syncwarp();
    for (uint32_t c = lane; c < n; c += 32) {
        const uint32_t L = s.clen[c], sym = s.sym[c];
        cb->symbols[c].symbol = (uint8_t)sym;
        cb->symbols[c].length = (uint8_t)L;
        cb->table[sym].code = s.la[c] >> (kMaxLen - L);
        cb->table[sym].length = L;
    }
    if (lane == 0) cb->symbol_count = n;
    __syncwarp();
}

// The encoder's per-byte table (code | length << 16, kEncAbsent if absent).
__device__ inline void warp_write_enc_table(const BookSyms& s, uint32_t n, EncTable* t, uint32_t lane) {
    for (uint32_t b = lane; b < 256; b += 32) t->e[b] = kEncAbsent;
    __syncwarp();
    for (uint32_t c = lane; c < n; c += 32) {
        const uint32_t L = s.clen[c];
        t->e[s.sym[c]] = (s.la[c] >> (kMaxLen - L)) | (L << 16);
    }
    __syncwarp();
}

// The same container-order arrays from a given symbol list (decoder side).
// Returns the Kraft sum, or ~0u if the list is not a valid canonical book
// (a length outside 1..16, a repeated byte, lengths not ascending, Kraft > 1).
__device__ inline uint32_t warp_load_symbols(const hgap_symlen* syms, uint32_t n, BookSyms& s, uint32_t lane) {
    uint32_t kr[8], tot = 0;
    bool bad = n > 256;
    if (lane < 8) s.seen[lane] = 0;
    __syncwarp();
#pragma unroll
    for (int t = 0; t < 8; ++t) {
        const uint32_t c = 8 * lane + t;
        kr[t] = 0;
        if (c < n && c < 256) {
            const uint32_t L = syms[c].length, sym = syms[c].symbol;
            s.sym[c] = (uint8_t)sym;
            s.clen[c] = (uint8_t)L;
            if (L < 1 || L > (uint32_t)kMaxLen) bad = true;
            else kr[t] = 1u << (kMaxLen - L);
            const uint32_t bit = 1u << (sym & 31);
            if (atomicOr(&s.seen[sym >> 5], bit) & bit) bad = true;
        }
        tot += kr[t];
    }
    __syncwarp();
    for (uint32_t c = lane; c + 1 < n && c + 1 < 256; c += 32)
        if (s.clen[c + 1] < s.clen[c]) bad = true;
    uint32_t kraft = 0;
    uint32_t run = warp_excl_scan(tot, lane, &kraft);
#pragma unroll
    for (int t = 0; t < 8; ++t) {
        const uint32_t c = 8 * lane + t;
        if (c < n && c < 256) s.la[c] = run;
        run += kr[t];
    }
    if (kraft > (1u << kMaxLen)) bad = true;
    bad = __any_sync(kFull, bad);
    __syncwarp();
    return bad ? ~0u : kraft;
}

// Decoder table (layout in hgap_internal.h) from the container-order arrays
// s.la / s.sym / s.clen of n >= 1 symbols.  Returns false if the level-2 part
// would exceed kDecT2Cap (only possible for an incomplete book).
__device__ inline bool warp_dec_table(const BookSyms& s, uint32_t n, DecTable* t, uint32_t lane) {
    constexpr uint32_t P = kDecPrefix, X = kMaxLen - kDecPrefix;  // 11, 5
    // symbol index of the largest left-aligned code <= v, starting from i
    auto advance = [&](uint32_t i, uint32_t v) {
        while (i + 1 < n && s.la[i + 1] <= v) ++i;
        return i;
    };
    auto entry = [&](uint32_t i, uint32_t v) -> uint16_t {
        const uint32_t L = s.clen[i];
        if (v < s.la[i] || v - s.la[i] >= (1u << (kMaxLen - L))) return kDecInvalid;
        return (uint16_t)(((L - 1) << 8) | s.sym[i]);
    };
    const uint32_t x0 = 64 * lane;
    // first pass: widths of this lane's pointer prefixes, for the level-2 offsets
    uint32_t i_last = 0, span = 0;
    for (uint32_t k = 0; k < 64; ++k) {
        const uint32_t x = x0 + k;
        i_last = advance(i_last, (x << X) | ((1u << X) - 1));
        const uint32_t L = s.clen[i_last];
        if (L > P && (s.la[i_last] >> X) == x) span += 1u << (L - P);
    }
    uint32_t total = 0;
    uint32_t off = warp_excl_scan(span, lane, &total);
    if (total > (uint32_t)kDecT2Cap) return false;
    for (uint32_t k = lane; k < (uint32_t)kDecT2Cap; k += 32) t->t2[k] = kDecInvalid;
    __syncwarp();  // cleared before any lane fills its level-2 groups
    uint32_t i_first = 0;
    i_last = 0;
    for (uint32_t k = 0; k < 64; ++k) {
        const uint32_t x = x0 + k;
        const uint32_t v = x << X;
        i_first = advance(i_first, v);
        i_last = advance(i_last, v | ((1u << X) - 1));
        const uint32_t L = s.clen[i_last];
        if (L > P && (s.la[i_last] >> X) == x) {
            const uint32_t w = L - P;
            t->t1[x] = (uint16_t)(0x8000u | (w << 12) | off);
            uint32_t i = i_first;
            for (uint32_t y = 0; y < (1u << w); ++y) {
                const uint32_t vy = v | (y << (X - w));
                i = advance(i, vy);
                t->t2[off + y] = entry(i, vy);
            }
            off += 1u << w;
        } else {
            t->t1[x] = entry(i_first, v);
        }
    }
    __syncwarp();
    return true;
}

}  // namespace hgap
