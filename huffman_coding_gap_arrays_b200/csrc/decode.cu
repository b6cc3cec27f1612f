// decode.cu -- segment-parallel Huffman decoder driven by the gap array, sm_100a.
//
// Replaces gpu_dec_l1_l2 (decoder/src/decoder.cu:454-730).  Same unit of
// parallelism -- a 128-bit segment that starts at its gap offset -- but each
// segment is decoded ONCE (the reference decodes it twice: a counting pass,
// then a writing pass, decoder.cu:529-569,672-725).
//
// A persistent CTA of W decoding warps (8, 15 or 16) and one more warp takes tiles
// of 32 W S consecutive segments of one stream.  A decoding warp owns 32 S
// of them, S per lane, and everything that is large is its own (no other warp
// reads or writes it), so a tile costs the CTA one barrier:
//   1. decode: a lane has its segment's words in registers (loaded a tile
//      ahead: one 16-byte load, the next segment's first word from the
//      neighbouring lane) and runs four phases of 32 bits, so its loop tests
//      only the phase's end.  One table in shared memory serves all code
//      lengths without a branch (DecIndex).  Position and output address
//      advance in one addition: an entry holds the bits and the number of its
//      symbols where the state has the position and the address.  The symbols
//      go to the lane's row in shared memory, sized for the book's shortest code
//      (of books with 1-bit codes as whole words, the lanes' rows interleaved);
//   2. the warps publish their symbol counts at the barrier;
//   3. the warp writes the PREVIOUS tile's symbols out of its image, with
//      16-byte stores shifted to the output's alignment (bytes at both ends),
//      clipped at exactly n bytes (the reference writes past n,
//      decoder.cu:529), and joins the rows of this tile to its image: a lane
//      stores the words it completes and ORs its unfinished last word into the
//      next lane's first (a segment has at least 8 symbols, so no word sees
//      three lanes).
// Meanwhile the extra warp publishes the tile's symbol count, resolves the
// tile's output offset with a bounded decoupled look-back, claims a tile two
// ahead, fetches its job, and copies the next tile's table into shared memory
// if it is another buffer's: none of those round trips is on the decoding
// warps' path, which need their results one barrier later.
// Checks: every segment must end exactly where the next gap entry says the
// next segment starts, every codeword must exist, and the stream must yield at
// least n symbols; failures set kDevCorrupt / kDevSize, never trap.
//
// The kernel is bound by shared-memory wavefronts (one lookup of 32 random
// entries and one or two byte stores per step: 84 % of the pipe on Zipf(1.2))
// and by instruction issue (72 %), not by HBM: fewer wavefronts at three more
// instructions a step measured slower (Last, below).  Measured (B200, 256 MiB,
// call without the status read), against a kernel with four CTA barriers a tile, a
// branch to a second table level and byte-wise compaction: Zipf(1.2) 524 -> 383
// us, mixed 489 -> 403, BF16 mantissa 422 -> 370, BF16 exponents 324 -> 267,
// clamped Gaussians of sigma 1 / 3 431 -> 247 / 321 -> 264; 1024 buffers of
// 4 KiB - 4 MiB (593 MB) 1047 -> 792 us.  (The kernel alone: Zipf(1.2) 362 us,
// mixed 383, mantissa 348, exponents 247.)  The branch-free table gave Zipf(1.2)
// 439 -> 401 us and the batch 896 -> 858; that no warp leaves alone when its wait
// gives up costs 0 to 1.2 % of a call (mixed 1 GiB 1494 -> 1511 us, the others less).
#include <cuda_runtime.h>

#include <type_traits>

#include "dec_entry.cuh"
#include "device_util.cuh"
#include "launch_cache.h"

namespace hgap {

// In place of a warp's symbol count: one of its waits gave up.
constexpr uint32_t kGaveUp = ~0u;

// R: stage rows of 4 symbols per segment (at most 4R symbols per segment); W: decoding warps;
// S: segments per lane of a tile.
template <int R, int W, int S>
struct DecCfg {
    static constexpr int kMaxSym = 4 * R;
    static constexpr int kSegs = 32 * W * S;           // segments per tile
    static constexpr int kThreads = 32 * (W + 1);
    static constexpr uint32_t P = dec_prefix(R);       // window bits of a lookup
    static constexpr int kTab = (int)dec_table_cap(R); // u32 table entries
    // one segment's row: its symbols, a byte or two that a multi-symbol entry stores past the
    // count, and the word after the last whole one; an odd number of words, so that the 32 rows a
    // warp writes start in 32 different banks (11 rows: at most 43 symbols, so 11 words do)
    static constexpr int kRowWords = R == 11 ? 11 : (R + 1) | 1;
    static constexpr int kRowBytes = 4 * kRowWords;
    static constexpr int kRowsBytes = 32 * S * kRowBytes;
    static constexpr int kImgBytes = 32 * S * kMaxSym + 32;  // the write-out reads 16-byte groups past the end
    static constexpr int kWarpBytes = kRowsBytes + kImgBytes;
    static constexpr size_t kSmem = 256 + (size_t)kTab * 4 + (size_t)W * kWarpBytes;
    // CTAs per SM: by shared memory (227 KiB usable, ~1.5 KiB static and reserved per CTA) and by
    // registers (40 a thread, 56 for two segments: 12 or 9 warps in each quarter of the SM)
    static constexpr int kBySmem = (int)((227u * 1024u) / (kSmem + 1536u));
    static constexpr int kByRegs = (S == 1 ? 48 : 36) / (W + 1);
    static constexpr int kMinBlocks = kBySmem < 1 ? 1 : kBySmem < kByRegs ? kBySmem : kByRegs;
    static_assert(kImgBytes % 16 == 0, "16-byte aligned images");
    static_assert((256 + 4 * kTab) % 128 == 0 && kRowsBytes % (128 * S) == 0, "rows on a multiple of 128");
};

// The decoder's table for one tile (DecIndex).
struct Table {
    const uint32_t* t1;      // shared memory
    const uint8_t* symlen;   // shared memory
    const uint16_t* t2;      // wide books: level 2, global memory
    uint32_t shift;
    int32_t offset;
};

// The entry (dec_entry.cuh) of the 32-bit window x at a code's start.
template <uint32_t P, bool WIDE, bool MULTI>
__device__ __forceinline__ uint32_t lookup(const Table& t, uint32_t x) {
    const int32_t i1 = (int32_t)(x >> (32 - (WIDE ? (uint32_t)kDecPrefix : P)));
    if (!WIDE) return t.t1[max(i1, (int32_t)(x >> t.shift) + t.offset)];
    uint32_t e = t.t1[i1];
    if (e & kEntPointer) {
        const uint32_t wd = (e >> 16) & 7u;
        e = entry_single<MULTI>(t.t2[(e & 0xffffu) + ((x << kDecPrefix) >> (32 - wd))]);
    }
    return e;
}

// The words of one segment in registers: its own four and the next segment's
// first (a code that starts in the segment may end up to 15 bits into it).
struct SegWords {
    uint32_t w0, w1, w2, w3, w4;
};

__device__ __forceinline__ void st_shared_u8(uint32_t addr, uint32_t v) {
    asm volatile("st.shared.u8 [%0], %1;" ::"r"(addr), "r"(v) : "memory");
}

__device__ __forceinline__ void st_shared_u32(uint32_t addr, uint32_t v) {
    asm volatile("st.shared.u32 [%0], %1;" ::"r"(addr), "r"(v) : "memory");
}

// Where a lane's symbols go.  One or two a step: bytes to a row of its own (`row`:
// its shared address).  Up to three (MULTI): whole words, made in a register, word
// k of lane l at 128 k + 4 l of the warp's rows (`row`: their address, a multiple
// of 128), which meets no other lane's bank; a lane's unfinished last word stays
// in the register.  Three byte stores of 32 drifting rows took 6 wavefronts and the
// shifts between them, one word store takes one: 1024 buffers of 4 KiB - 4 MiB, the
// 32-row class 150 -> 142 us.  With pairs the word form saves a quarter of the
// kernel's wavefronts and still loses (Zipf(1.2) 256 MiB 363 -> 385 us): two byte
// stores cost three instructions less, and there the kernel is short of those.
struct Last {
    uint32_t count, word;  // the lane's symbols, and (MULTI) the count % 4 last of them
};
// The last four symbols are in acc, the newest at the top; `at8` = 8 * (their
// number) mod 32: the word that entry e's symbols go on with (what is past them: junk).
__device__ __forceinline__ uint32_t row_word(uint32_t acc, uint32_t e, uint32_t at8) {
    return __funnelshift_l(acc, e, at8);
}

// Decodes the codes that start in one 128-bit segment (not the stream's last
// one), from bit `pos` (its gap offset), as four phases of 32 bits: phase k
// decodes the codes starting in word k, from the window of words k and k+1,
// so the loop tests only bit 5 of the position -- no word refill, no end test.
// Codes of a pair / multi entry all start inside the segment in phases 0-2
// (they fit the window of P bits and phase 2 ends 32 bits before the segment
// does); in phase 3 that holds while pos <= 32 - P, and the last bits take only
// the codes that start before bit 32 of the phase.  The symbols go to the lane's
// row; their number is returned in `last`.  Returns the end bit of the last code
// relative to phase 3 (32 + the next gap entry for a valid stream), or a value no
// stream yields after an invalid code.
template <uint32_t P, bool WIDE, bool COMPLETE, bool PAIRS, bool MULTI>
__device__ __forceinline__ uint32_t decode_segment(const Table& t, const SegWords& w, uint32_t pos, uint32_t row,
                                                   uint32_t lane4, Last& last) {
    static_assert(!MULTI || COMPLETE, "multi entries: complete books");
    constexpr uint32_t kBad = 1u << 16;
    constexpr uint32_t kEarly = (WIDE ? (uint32_t)kDecPrefix : P) - 1;  // the last phase's fast loop ends this many bits early
    if (MULTI) {
        uint32_t out = row >> 5, acc = 0;  // (row / 32 is a multiple of 4: out's low bits count the word's bytes)
        auto put = [&](uint32_t e, uint32_t n) {
            st_shared_u32(((out << 5) & ~127u) | lane4, row_word(acc, e, out << 3));
            acc = __funnelshift_r(acc, e, 8 * n);
            out += n;
        };
        auto fast = [&](uint32_t cw, uint32_t nw) {
            while (!(pos & 32)) {
                const uint32_t e = lookup<P, WIDE, true>(t, __funnelshift_l(nw, cw, pos));
                put(e, 1 + (e >> 29));
                pos += (e >> 24) & 31u;
            }
        };
        fast(w.w0, w.w1);
        pos -= 32;
        fast(w.w1, w.w2);
        pos -= 32;
        fast(w.w2, w.w3);
        pos += kEarly - 32;
        fast(w.w3 >> kEarly, __funnelshift_r(w.w4, w.w3, kEarly));
        pos -= kEarly;
        while (!(pos & 32)) {
            const uint32_t e = lookup<P, WIDE, true>(t, __funnelshift_l(w.w4, w.w3, pos));
            const uint32_t tot = (e >> 24) & 31u, more = e >> 29;
            const bool all = pos + tot <= 32;  // every code of the entry ends, so starts, inside
            put(e, all ? 1 + more : 1);
            pos += all || !more ? tot : t.symlen[e & 0xffu];
        }
        last.count = out - (row >> 5);
        last.word = row_word(acc, 0, out << 3);
        return pos;
    }
    uint32_t s = (row << 8) | pos;
    auto fast = [&](uint32_t cw, uint32_t nw) -> bool {  // false: an invalid code
        while (!(s & 32)) {
            const uint32_t e = lookup<P, WIDE, false>(t, __funnelshift_l(nw, cw, s));
            if (!COMPLETE && (e & kEntInvalidBit)) return false;
            st_shared_u8(s >> 8, e);
            if (PAIRS) st_shared_u8((s >> 8) + 1, e >> 8);  // a single entry's second byte: overwritten or past the count
            s += e >> 16;
        }
        return true;
    };
    auto run = [&]() -> bool {
        if (!fast(w.w0, w.w1)) return false;
        s -= 32;
        if (!fast(w.w1, w.w2)) return false;
        s -= 32;
        if (!fast(w.w2, w.w3)) return false;
        s -= 32;
        if (!PAIRS) return fast(w.w3, w.w4);
        s += kEarly;
        if (!fast(w.w3 >> kEarly, __funnelshift_r(w.w4, w.w3, kEarly))) return false;
        s -= kEarly;
        while (!(s & 32)) {  // the last bits: only the codes that start before bit 32
            const uint32_t e = lookup<P, WIDE, false>(t, __funnelshift_l(w.w4, w.w3, s));
            if (!COMPLETE && (e & kEntInvalidBit)) return false;
            st_shared_u8(s >> 8, e);
            st_shared_u8((s >> 8) + 1, e >> 8);
            uint32_t by = e >> 16;
            if (by & 0x200u) {  // two symbols: the second one counts only if it starts inside
                const uint32_t l1 = t.symlen[e & 0xffu];
                if ((s & 31u) + l1 >= 32) by = 0x100u + l1;
            }
            s += by;
        }
        return true;
    };
    const bool valid = run();
    last.count = (s >> 8) - row;
    return COMPLETE || valid ? s & 0xffu : kBad;
}

// The stream's last segment: its codes end at bit `end` (<= 128) and zero
// padding follows, which may not decode.  One code per step (the first code of
// any pair or multi entry), the words picked by index.
template <uint32_t P, bool WIDE, bool COMPLETE, bool MULTI>
__device__ __forceinline__ Last decode_last_segment(const Table& t, const SegWords& w, uint32_t pos, uint32_t end,
                                                    uint32_t row, uint32_t lane4) {
    auto word = [&](uint32_t i) { return i == 0 ? w.w0 : i == 1 ? w.w1 : i == 2 ? w.w2 : i == 3 ? w.w3 : w.w4; };
    uint32_t cnt = 0, acc = 0;
    while (pos < end) {
        const uint32_t wi = pos >> 5;
        const uint32_t e = lookup<P, WIDE, MULTI>(t, __funnelshift_l(word(wi + 1), word(wi), pos));
        if (!COMPLETE && (e & kEntInvalidBit)) break;  // the padding after the final codeword
        const uint32_t more = MULTI ? e >> 29 : (e >> 24) - 1;
        const uint32_t len = MULTI ? (e >> 24) & 31u : (e >> 16) & 31u;
        if (MULTI) {
            st_shared_u32((row + 32 * (cnt & ~3u)) | lane4, row_word(acc, e, 8 * cnt));
            acc = __funnelshift_r(acc, e, 8);
        } else {
            st_shared_u8(row + cnt, e);
        }
        ++cnt;
        pos += more ? t.symlen[e & 0xffu] : len;
    }
    return {cnt, row_word(acc, 0, 8 * cnt)};
}

// A claimed tile, in shared memory: what the decoding warps need of it (clipped
// to the tile, 32-bit), then what the extra warp does.
struct DecSlot {
    const uint32_t* bits;  // the tile's first word
    const uint32_t* gaps;  // and gap word
    uint32_t nwords;       // words from there to the stream's end (at most one past the tile)
    uint32_t ngaps;        // gap words of the tile
    uint32_t nseg;         // segments (0: no tile)
    uint32_t last_bits;    // bits of the stream's last segment if it is in this tile, else 0
    uint32_t job_id;
    DecIndex index;        // of its job's table
    bool first, last;      // of its job's tiles
    uint64_t rec;          // look-back record
    uint8_t* out;          // the job's output
    uint64_t n;            // and its size
};

// COMPLETE: the book's Kraft sum is 1 (every package-merge book with two or
// more symbols), so no table entry is invalid and the decode loop skips that test.
// PAIRS: level-1 entries carry two symbols where both codes fit in the window
// (worth it for short-code books; for long codes the extra store only costs);
// with a complete book of the shortest codes, up to three (dec_multi).
template <int R, int W, int S, bool COMPLETE, bool PAIRS>
__global__ void __launch_bounds__(DecCfg<R, W, S>::kThreads, DecCfg<R, W, S>::kMinBlocks)
    decode_kernel(const __grid_constant__ DecArgs a, const __grid_constant__ DecTable tab) {
    using C = DecCfg<R, W, S>;
    extern __shared__ __align__(128) unsigned char smem[];
    uint8_t* const symlen = smem;                          // a symbol's code length, where it is at most kDecPrefix
    uint32_t* const t1 = reinterpret_cast<uint32_t*>(smem + 256);
    unsigned char* const areas = smem + 256 + 4 * C::kTab; // the warps' rows, then their images
    __shared__ DecSlot slot[4];                            // tile i in slot i % 4
    __shared__ uint32_t tot[2][W];                         // by tile parity: the warps' symbol counts,
    __shared__ uint8_t* dst[2];                            // the tile's place in the output,
    __shared__ uint32_t room[2];                           // and the bytes there until n
    // completed once for every second tile (by its parity): its counts are published; its slot is
    // filled; dst and room are set
    __shared__ uint64_t published[2], filled[2], placed[2];
    __shared__ uint64_t tbar;                              // a table copy landed
    __shared__ uint64_t s_nitems;

    constexpr bool MULTI = PAIRS && dec_multi(R, COMPLETE);
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;

    // the tile `item` into slot s (one thread)
    auto fill_slot = [&](int s, uint64_t item) {
        DecSlot& d = slot[s];
        d.nseg = 0;
        if (item >= s_nitems) return;
        const uint32_t j = a.jobs ? a.job_of[item] : 0u;
        const DecJob& J = a.jobs ? a.jobs[j] : a.single;
        const uint64_t local = a.jobs ? item - a.item0s[j] : item;
        const uint64_t s0 = local * C::kSegs, left = J.segments - s0;
        const uint64_t words = J.words - 4 * s0, gws = J.gap_words - s0 / 8;
        d.bits = J.bits + 4 * s0;
        d.gaps = J.gaps + s0 / 8;
        d.nwords = words < 4 * C::kSegs + 1 ? (uint32_t)words : 4 * C::kSegs + 1;
        d.ngaps = gws < C::kSegs / 8 ? (uint32_t)gws : C::kSegs / 8;
        d.nseg = left < (uint64_t)C::kSegs ? (uint32_t)left : (uint32_t)C::kSegs;
        // (every entry point checks segments == ceil(words / 4))
        d.last_bits = left <= (uint64_t)C::kSegs ? (uint32_t)(32 * words - 128 * (left - 1)) : 0u;
        d.job_id = j;
        d.index = a.jobs ? a.tables[j].index : a.index;
        d.first = local == 0;
        d.last = local + 1 == J.ntiles;
        d.rec = J.item0 + local;
        d.out = J.out_aligned + J.out_lo;
        d.n = J.n;
    };
    auto copy_table = [&](const DecSlot& d) {  // one thread
        fence_proxy_async_smem();              // after the reads of the table before it
        // (symlen and t1 lie together, here and in DecTableW)
        bulk_load(symlen, a.tables[d.job_id].symlen, 256 + 4 * d.index.used, &tbar);
    };

    if (!a.jobs) {
        // single path: the u16 tables to shared memory (the areas are still free), and the entries
        // made from there (the launch parameters' bank serves one address at a time)
        constexpr int kRaw = sizeof(DecTable) / 8, kT1 = 1 << kDecPrefix;
        static_assert(sizeof(DecTable) <= (size_t)W * C::kWarpBytes, "the raw table fits the areas");
        uint64_t* const raw = reinterpret_cast<uint64_t*>(areas);
        const uint64_t* const src = reinterpret_cast<const uint64_t*>(&tab);
        for (int i = tid; i < kRaw; i += C::kThreads) raw[i] = src[i];
        __syncthreads();
        const DecTable& r = *reinterpret_cast<const DecTable*>(areas);
        const bool wide = a.index.first_long == kDecWide;
        for (int i = tid; i < (int)a.index.used; i += C::kThreads) {
            uint32_t e = kEntInvalid;
            if (wide) {
                e = MULTI   ? entry_multi<kDecPrefix>(r.t1, i)
                    : PAIRS ? entry_pair<kDecPrefix>(r.t1, i)
                            : entry_single<false>(r.t1[i]);
            } else if ((uint32_t)i < a.index.first_long) {
                e = MULTI   ? entry_multi<C::P>(r.t1, i)
                    : PAIRS ? entry_pair<C::P>(r.t1, i)
                            : entry_single<false>(r.t1[i << (kDecPrefix - C::P)]);
            } else {
                // a longer code: v = its window's bits down to the longest length
                const uint32_t v = (uint32_t)(i - a.index.offset), len = 32 - a.index.shift;
                if (v < 1u << len) {
                    const uint32_t below = len - kDecPrefix;  // (len is 11 or more)
                    uint32_t e1 = r.t1[v >> below];
                    if (e1 & 0x8000u)
                        e1 = r.t2[(e1 & 0xfffu) + ((v & ((1u << below) - 1u)) >> (below - ((e1 >> 12) & 7u)))];
                    e = entry_single<MULTI>(e1);
                }
            }
            t1[i] = e;
        }
        for (int i = tid; i < kT1; i += C::kThreads) {
            const uint32_t e1 = r.t1[i];
            if (!(e1 & (0x8000u | kDecInvalid))) symlen[e1 & 0xffu] = (uint8_t)((e1 >> 8) + 1);
        }
    }
    if (tid == 32 * W) {
        for (int k = 0; k < 2; ++k) {
            mbar_init(&published[k], 1);
            mbar_init(&filled[k], 1);
            mbar_init(&placed[k], 1);
            room[k] = 0;
        }
        mbar_init(&tbar, 1);
        mbar_init_fence();
        s_nitems = a.nitems_dev ? *a.nitems_dev : a.nitems;
        fill_slot(0, atomicAdd(a.counter, 1u));
        mbar_arrive(&filled[0]);
        if (a.jobs && slot[0].nseg) copy_table(slot[0]);
    }
    __syncthreads();
    if (slot[0].nseg == 0) return;
    // Waits between the warps of the CTA: false for a lane that gave up (so did a look-back
    // somewhere, or this took longer than any look-back should).
    auto wait = [&](uint64_t* bar, uint32_t i) {
        return mbar_wait(&bar[i & 1], (i >> 1) & 1, a.status, true, kCtaWaitLimitNs);
    };

    if (warp == W) {
        // ---- the extra warp -------------------------------------------------------
        // (the second tile is claimed only now, when the other CTAs have their first: a CTA that
        // held two consecutive tiles would keep all later ones waiting for its second)
        uint32_t claim = 0, copies = a.jobs ? 1 : 0;  // table copies issued
        if (lane == 0) {
            fill_slot(1, atomicAdd(a.counter, 1u));
            mbar_arrive(&filled[1]);
        }
        __syncwarp();
        for (uint32_t i = 0; slot[i & 3].nseg != 0; ++i) {
            const DecSlot& T = slot[i & 3];
            const DecSlot& N = slot[(i + 1) & 3];
            if (!__all_sync(kFull, wait(published, i))) break;  // tile i is decoded: the table is free
            const uint32_t t = lane < (uint32_t)W ? tot[i & 1][lane] : 0u;
            if (__any_sync(kFull, t == kGaveUp)) break;
            const uint32_t Ct = __reduce_add_sync(kFull, t);
            if (lane == 0 && N.nseg) {
                claim = atomicAdd(a.counter, 1u);  // (its answer is needed only after the look-back)
                if (a.jobs && N.job_id != T.job_id) {
                    copy_table(N);
                    ++copies;
                }
            }
            const uint64_t O = lookback_resolve(a.lookback, T.rec, Ct, T.first, a.status, lane, wait_limit(a.hook),
                                                T.rec + 1 != a.hook.hold_plus1);
            if (lane == 0) {
                if (T.last && O + Ct < T.n) atomicOr(a.status, kDevSize);
                dst[i & 1] = T.out + O;
                room[i & 1] = O >= T.n ? 0u : T.n - O < 0x40000000ull ? (uint32_t)(T.n - O) : 0x40000000u;
                mbar_arrive(&placed[i & 1]);
                if (N.nseg) fill_slot((i + 2) & 3, claim);
                else slot[(i + 2) & 3].nseg = 0;
                mbar_arrive(&filled[i & 1]);
            }
            __syncwarp();
        }
        // never leave the CTA with a copy still in flight into its shared memory
        if (lane == 0 && copies) mbar_wait(&tbar, (copies - 1) & 1, a.status, false);
        return;
    }

    // ---- the decoding warps -------------------------------------------------------
    unsigned char* const rows = areas + warp * C::kRowsBytes;
    unsigned char* const img = areas + W * C::kRowsBytes + warp * C::kImgBytes;
    // the lane's first word of its first segment, and the words from one of its words to the next
    constexpr int kNext = MULTI ? 32 : 1;
    uint32_t* const row32 = reinterpret_cast<uint32_t*>(rows + lane * (MULTI ? 4 : C::kRowBytes));
    const uint32_t u0 = warp * 32 * S + lane;  // the lane's segments in the tile: u0 + 32 k

    // A tile's words and gap entries, loaded a tile ahead: a segment's four words (one 16-byte load
    // where the stream is 16-byte aligned), for lane 31 the first word of the next segment, the gap
    // word of the segment's entry, for lane 0 the one of the entry before.
    uint4 pre_q[S];
    uint32_t pre_w4[S], pre_gap[S], pre_gap0[S];
    auto prefetch = [&](const DecSlot& N) {
        const uint32_t words = N.nseg ? N.nwords : 0u, ngaps = N.nseg ? N.ngaps : 0u;
        const bool al16 = (reinterpret_cast<uintptr_t>(N.bits) & 15) == 0;
#pragma unroll
        for (int k = 0; k < S; ++k) {
            const uint32_t u = u0 + 32 * k, w = 4 * u;
            const uint32_t* const p = N.bits + w;
            if (al16 && w + 4 <= words) {
                pre_q[k] = ld_stream_v4(p);
            } else {
                pre_q[k].x = w < words ? ld_stream_u32(p) : 0u;
                pre_q[k].y = w + 1 < words ? ld_stream_u32(p + 1) : 0u;
                pre_q[k].z = w + 2 < words ? ld_stream_u32(p + 2) : 0u;
                pre_q[k].w = w + 3 < words ? ld_stream_u32(p + 3) : 0u;
            }
            pre_w4[k] = lane == 31 && w + 4 < words ? ld_stream_u32(p + 4) : 0u;
            pre_gap[k] = (u >> 3) < ngaps ? __ldg(N.gaps + (u >> 3)) : 0u;
            pre_gap0[k] = lane == 0 && w < words && (u || !N.first) ? __ldg(N.gaps + (u >> 3) - 1) : 0u;
        }
    };
    prefetch(slot[0]);
    uint32_t copies = 0;  // table copies waited for
    auto table_landed = [&] {
        return __all_sync(kFull, mbar_wait(&tbar, copies++ & 1, a.status, true, kCtaWaitLimitNs));
    };
    // A warp whose wait gave up may not go alone: the others' barrier of the next tile, number i,
    // counts all W.  It says so there, and all leave after that barrier, the extra warp with them.
    auto give_up = [&](uint32_t i) {
        if (lane == 0) tot[i & 1][warp] = kGaveUp;
        named_barrier(1, 32 * W);
        if (tid == 0) mbar_arrive(&published[i & 1]);
    };
    if (a.jobs && !table_landed()) return give_up(0);

    uint32_t prev_m = 0, prev_before = 0;  // the warp's symbols of the tile before, and those before them in it
    for (uint32_t i = 0;; ++i) {
        const DecSlot& T = slot[i & 3];
        const bool have = T.nseg != 0, prev = i != 0;

        // ---- 1. decode ---------------------------------------------------------------
        uint32_t n[S], part[S];
#pragma unroll
        for (int k = 0; k < S; ++k) {
            n[k] = part[k] = 0;
            if (!have) continue;  // uniform
            const Table t{t1, symlen, a.jobs ? a.tables[T.job_id].t2() : tab.t2, T.index.shift, T.index.offset};
            const uint32_t u = u0 + 32 * k;
            SegWords w;
            w.w0 = pre_q[k].x;
            w.w1 = pre_q[k].y;
            w.w2 = pre_q[k].z;
            w.w3 = pre_q[k].w;
            const uint32_t up = __shfl_down_sync(kFull, pre_q[k].x, 1);
            w.w4 = lane == 31 ? pre_w4[k] : up;
            const uint32_t gap = (pre_gap[k] >> (4 * (u & 7))) & 0xfu;  // where the next segment's first code starts
            const uint32_t before = __shfl_up_sync(kFull, gap, 1);
            const uint32_t pos = lane == 0 ? pre_gap0[k] >> 28 : before;
            const uint32_t row = smem_addr(row32 + 32 * k * C::kRowWords) - (MULTI ? 4 * lane : 0u);
            Last last = {0, 0};
            // (every wide book's tile takes the second branch: uniform over the CTA)
            auto segment = [&](auto wide) {
                constexpr bool WIDE = decltype(wide)::value;
                if (T.last_bits && u + 1 == T.nseg) {
                    last = decode_last_segment<C::P, WIDE, COMPLETE, MULTI>(t, w, pos, T.last_bits, row, 4 * lane);
                } else {
                    const uint32_t end = decode_segment<C::P, WIDE, COMPLETE, PAIRS, MULTI>(t, w, pos, row, 4 * lane, last);
                    if (end != 32 + gap) atomicOr(a.status, kDevCorrupt);
                }
            };
            if (u < T.nseg) {
                if (COMPLETE && T.index.first_long != kDecWide) segment(std::integral_constant<bool, false>());
                else segment(std::integral_constant<bool, true>());
            }
            n[k] = last.count;
            part[k] = last.word;
        }
        // both segments' counts in one scan (a warp's 32 have less than 2^13 symbols)
        uint32_t packed = n[0];
        if (S > 1) packed |= n[S - 1] << 16;
        const uint32_t incl = warp_incl_scan(packed, lane);
        const uint32_t sums = __shfl_sync(kFull, incl, 31);
        const uint32_t sum0 = S > 1 ? sums & 0xffffu : sums, m = S > 1 ? sum0 + (sums >> 16) : sums;  // the warp's symbols
        uint32_t before = 0;
        bool reload = false, together = true, ok = true;  // together: no warp gave up before this tile's barrier
        if (have) {
            if (lane == 0) tot[i & 1][warp] = m;
            named_barrier(1, 32 * W);  // the counts are in place, the table is free
            const uint32_t t = lane < (uint32_t)W ? tot[i & 1][lane] : 0u;
            together = t != kGaveUp;
            before = __reduce_add_sync(kFull, lane < warp ? t : 0u);
            if (warp == 0) {
                // the aggregate first: nothing that this CTA waits for may hold it back
                const uint32_t Ct = __reduce_add_sync(kFull, t);
                if (lane == 0) {
                    if (T.rec + 1 != a.hook.hold_plus1) lookback_publish(a.lookback, T.rec, Ct, T.first);
                    mbar_arrive(&published[i & 1]);
                }
            }
            const DecSlot& N = slot[(i + 1) & 3];
            ok = wait(filled, i + 1);
            if (ok) {
                reload = a.jobs && N.nseg && N.job_id != T.job_id;
                prefetch(N);
            }
        } else {
            named_barrier_arrive(1, 32 * W);  // for a warp that gave up and knows of no end
        }
        if (prev) ok = wait(placed, i - 1) && ok;
        if (!__all_sync(kFull, ok && together)) {
            if (have && __all_sync(kFull, together)) give_up(i + 1);
            break;
        }

        // ---- 2. write out the tile before -----------------------------------------------
        if (prev) {
            uint8_t* const out = dst[(i & 1) ^ 1] + prev_before;
            const uint32_t left = room[(i & 1) ^ 1];
            uint32_t m = left > prev_before ? left - prev_before : 0u;
            if (m > prev_m) m = prev_m;
            uint32_t h = (0u - (uint32_t)reinterpret_cast<uintptr_t>(out)) & 15u;  // bytes before the first 16-byte group
            if (h > m) h = m;
            const uint32_t nq = (m - h) >> 4;
            // the ragged ends: 16 lanes each
            const uint32_t b = lane < 16 ? lane : h + 16 * nq + lane - 16;
            if (b < (lane < 16 ? h : m)) out[b] = img[b];
            const uint4* const src = reinterpret_cast<const uint4*>(img);
            uint4* const out16 = reinterpret_cast<uint4*>(out + h);
            const uint32_t sh = 8 * (h & 3);
#pragma unroll 1
            for (uint32_t c = lane; c < nq; c += 32) {
                const uint4 p = src[c], g = src[c + 1];
                uint4 o;
                auto join = [sh](uint32_t lo, uint32_t hi) { return __funnelshift_r(lo, hi, sh); };
                switch (h >> 2) {  // uniform over the warp
                    case 0: o = make_uint4(join(p.x, p.y), join(p.y, p.z), join(p.z, p.w), join(p.w, g.x)); break;
                    case 1: o = make_uint4(join(p.y, p.z), join(p.z, p.w), join(p.w, g.x), join(g.x, g.y)); break;
                    case 2: o = make_uint4(join(p.z, p.w), join(p.w, g.x), join(g.x, g.y), join(g.y, g.z)); break;
                    default: o = make_uint4(join(p.w, g.x), join(g.x, g.y), join(g.y, g.z), join(g.z, g.w)); break;
                }
                out16[c] = o;
            }
        }

        if (!have) break;

        // ---- 3. this tile's rows to the image --------------------------------------------
        {
            prev_before = before;
            prev_m = m;
            uint32_t* to[S];
            uint32_t full[S], rest[S], shift[S];
            __syncwarp();  // the image is written out
#pragma unroll
            for (int k = 0; k < S; ++k) {
                uint32_t* const r = row32 + 32 * k * C::kRowWords;
                const uint32_t c = n[k];
                const uint32_t d = k == 0 ? (incl & (S > 1 ? 0xffffu : ~0u)) - c : sum0 + (incl >> 16) - c;  // first byte
                const uint32_t sh = 8 * (d & 3), whole = c >> 2;
                shift[k] = sh;
                full[k] = ((d & 3) + c) >> 2;
                to[k] = reinterpret_cast<uint32_t*>(img) + (d >> 2);
                // the row's word after the last whole one: what is past the count cleared
                const uint32_t xl = MULTI ? part[k] : r[whole] & ((1u << (8 * (c & 3))) - 1u);
                r[kNext * whole] = xl;
                // the lane's unfinished word
                const uint32_t xk = whole ? r[kNext * (whole - 1)] : 0u;
                rest[k] = full[k] > whole ? __funnelshift_l(xl, 0u, sh) : (xl << sh) | __funnelshift_l(xk, 0u, sh);
                // the words that no lane completes: the last lane's, and in the stream's last tile, whose
                // last segment may have fewer symbols, any lane's
                if (T.last_bits || (k == S - 1 && lane == 31)) to[k][full[k]] = 0;
            }
            if (T.last_bits) __syncwarp();
#pragma unroll
            for (int k = 0; k < S; ++k) {
                const uint32_t* const r = row32 + 32 * k * C::kRowWords;
                const uint32_t sh = shift[k];
                const uint32_t most = __reduce_max_sync(kFull, full[k]);
                uint32_t cur = 0;
#pragma unroll
                for (int j = 0; j <= R; ++j) {
                    if ((uint32_t)j >= most) break;  // uniform
                    const uint32_t x = r[kNext * j];
                    if ((uint32_t)j < full[k]) to[k][j] = cur | (x << sh);
                    cur = __funnelshift_l(x, 0u, sh);
                }
            }
            __syncwarp();
#pragma unroll
            for (int k = 0; k < S; ++k)
                if (n[k]) atomicOr(to[k] + full[k], rest[k]);
            __syncwarp();
        }
        if (reload && !table_landed()) return give_up(i + 1);
    }
}

uint64_t decode_tiles(uint64_t segments, uint32_t min_len, uint32_t tile_segs) {
    const uint64_t segs = dec_tile_segs_for(dec_stage_rows(min_len ? min_len : 1), tile_segs);
    return (segments + segs - 1) / segs;
}

template <int R, int W, int S, bool COMPLETE, bool PAIRS>
static int launch_decode_r(const DecArgs& a, const DecTable& t, int ctas_per_sm, cudaStream_t st) {
    using C = DecCfg<R, W, S>;
    auto kern = decode_kernel<R, W, S, COMPLETE, PAIRS>;
    static LaunchCache cache;  // one per kernel instantiation
    const LaunchFacts f = cache.get(reinterpret_cast<const void*>(kern), C::kThreads, C::kSmem);
    if (f.err != cudaSuccess) return f.err;
    const int sms = f.sms, per_sm = f.per_sm;
    const int k = (ctas_per_sm > 0 && ctas_per_sm < per_sm) ? ctas_per_sm : per_sm;
    const uint64_t cap = (uint64_t)sms * k;
    const unsigned grid = (unsigned)(a.nitems_dev ? cap : (a.nitems < cap ? (a.nitems ? a.nitems : 1) : cap));
    kern<<<grid, C::kThreads, C::kSmem, st>>>(a, t);
    return cudaGetLastError();
}

template <int R, bool COMPLETE, bool PAIRS>
static int launch_decode_s(const DecArgs& a, const DecTable& t, int k, uint32_t tile_segs, cudaStream_t st) {
    const int segs = dec_tile_segs_for(R, tile_segs);
    if (segs == 256) return launch_decode_r<R, 8, 1, COMPLETE, PAIRS>(a, t, k, st);
    if (segs == 480) {
        // a batch's complete books (it decodes the incomplete ones with 32 rows)
        if constexpr (R == 16 && COMPLETE && PAIRS) return launch_decode_r<16, 15, 1, true, true>(a, t, k, st);
        return cudaErrorInvalidValue;
    }
    constexpr int W = R == 16 ? 16 : 8, S = R >= 16 ? 1 : 2;
    static_assert(DecCfg<R, W, S>::kSegs == dec_tile_segs(R), "the tile's shape");
    return launch_decode_r<R, W, S, COMPLETE, PAIRS>(a, t, k, st);
}

template <bool COMPLETE, bool PAIRS>
static int launch_decode_c(const DecArgs& a, const DecTable& t, uint32_t min_len, int k, uint32_t tile_segs,
                           cudaStream_t st) {
    switch (dec_stage_rows(min_len)) {
        case 8: return launch_decode_s<8, COMPLETE, PAIRS>(a, t, k, tile_segs, st);
        case 11: return launch_decode_s<11, COMPLETE, PAIRS>(a, t, k, tile_segs, st);
        case 16: return launch_decode_s<16, COMPLETE, PAIRS>(a, t, k, tile_segs, st);
        default: return launch_decode_s<32, COMPLETE, PAIRS>(a, t, k, tile_segs, st);
    }
}

int launch_decode(const DecArgs& a, const DecTable& t, uint32_t min_len, bool complete, bool pairs,
                  int ctas_per_sm, uint32_t tile_segs, void* stream) {
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (min_len == 0) min_len = 1;
    if (pairs)
        return complete ? launch_decode_c<true, true>(a, t, min_len, ctas_per_sm, tile_segs, st)
                        : launch_decode_c<false, true>(a, t, min_len, ctas_per_sm, tile_segs, st);
    return complete ? launch_decode_c<true, false>(a, t, min_len, ctas_per_sm, tile_segs, st)
                    : launch_decode_c<false, false>(a, t, min_len, ctas_per_sm, tile_segs, st);
}

}  // namespace hgap
