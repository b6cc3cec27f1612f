// batch.cu -- the batched path (include/hgap.h, "batched path") and the
// device-side codebook entry points.  No counterpart in the reference.
//
// Compress, all on the stream, nothing back to the host:
//   1. benc_setup   each buffer's alignment, region size and region count; an
//                   exclusive scan numbers the regions globally;
//   2. hist_st      per-region histograms and per-buffer histograms;
//   3. book         one warp per buffer: length-limited canonical codebook,
//                   encoder table, sizes (book.cuh);
//   4. benc_place   scans of the stream sizes place every bitstream
//                   (16-byte aligned) and gap array in the two arenas;
//   5. enc_plan     one warp per region: bit count, first output bit, all that
//                   a CTA needs to start on it;
//   6. encode       the single-buffer encoder kernel over all regions, the
//                   CTA reloading its code table when the buffer changes.
// Decompress:
//   1. bdec_table   one CTA per buffer: checks the book, writes its decoder
//                   table in the form the decode kernel keeps in shared
//                   memory (DecTableW), puts the buffer in one of 8 classes
//                   (decoder stage size by the shortest code x complete book
//                   or not), and writes its decode job (stream, output, tile
//                   count);
//   2. bdec_setup   look-back record numbering over all tiles, and
//                   per class the numbering of the class's tiles;
//   3. bdec_map     tile -> buffer map of each class;
//   4. decode       one persistent launch per class of complete books and one
//                   for all incomplete ones (or those the caller names in
//                   dec_class_mask), the single-buffer decoder kernel over the
//                   class's tiles.
// Every launch has a fixed grid and reads its work counts from device memory,
// so the sequence can be captured once and replayed.
#include <cuda_runtime.h>

#include <cstring>

#include "book.cuh"
#include "dec_entry.cuh"
#include "launch_cache.h"

namespace hgap {
namespace {

// Books (warps) per CTA of the book kernels.  A book is one warp's serial chain,
// so its latency and the books in flight set the time: with 32-bit weights a
// book's scratch takes 6.3 KiB and 32 books share an SM.  1024 books 69 -> 31 us,
// 4096 books 158 -> 58 (64-bit weights throughout, 14 books an SM, both lists'
// heads loaded in every merge step).  A book of kBook32 bytes or more takes
// 64-bit weights and the whole CTA's scratch, after the CTA's other books.
constexpr int kBookWarps = 2;
using Book32 = BookScratch<uint32_t>;
using Book64 = BookScratch<uint64_t>;
constexpr size_t kBookSmem = kBookWarps * sizeof(Book32) > sizeof(Book64) ? kBookWarps * sizeof(Book32) : sizeof(Book64);
constexpr int kScanThreads = 1024;
constexpr uint32_t kClasses = 8;
constexpr uint32_t kNoClass = 0xffu;
constexpr uint32_t kIncomplete = 6;  // the class number all incomplete books are launched under (32 rows)

// ----------------------------------------------------------- block scans ---
// Exclusive scan of one u64 per thread over a 1024-thread CTA; returns the
// exclusive prefix and the block total.
__device__ __forceinline__ uint64_t block_excl_scan_u64(uint64_t v, uint64_t* total, uint64_t* s_warp) {
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint64_t x = v;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const uint64_t t = __shfl_up_sync(kFull, x, d);
        if (lane >= (uint32_t)d) x += t;
    }
    if (lane == 31) s_warp[warp] = x;
    __syncthreads();
    if (warp == 0) {
        uint64_t w = s_warp[lane];
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const uint64_t t = __shfl_up_sync(kFull, w, d);
            if (lane >= (uint32_t)d) w += t;
        }
        s_warp[lane] = w;  // inclusive over warps
    }
    __syncthreads();
    const uint64_t before = warp ? s_warp[warp - 1] : 0;
    *total = s_warp[31];
    __syncthreads();  // s_warp free for the next call
    return before + x - v;
}

// The same for two values per thread at once (one set of barriers).
__device__ __forceinline__ void block_excl_scan2_u64(uint64_t& a, uint64_t& b, uint64_t* total_a, uint64_t* total_b,
                                                     uint64_t (*s_warp)[32]) {
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint64_t x = a, y = b;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const uint64_t t = __shfl_up_sync(kFull, x, d);
        const uint64_t u = __shfl_up_sync(kFull, y, d);
        if (lane >= (uint32_t)d) {
            x += t;
            y += u;
        }
    }
    if (lane == 31) {
        s_warp[0][warp] = x;
        s_warp[1][warp] = y;
    }
    __syncthreads();
    if (warp < 2) {
        uint64_t w = s_warp[warp][lane];
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const uint64_t t = __shfl_up_sync(kFull, w, d);
            if (lane >= (uint32_t)d) w += t;
        }
        s_warp[warp][lane] = w;  // inclusive over warps
    }
    __syncthreads();
    a = (warp ? s_warp[0][warp - 1] : 0) + x - a;
    b = (warp ? s_warp[1][warp - 1] : 0) + y - b;
    *total_a = s_warp[0][31];
    *total_b = s_warp[1][31];
    __syncthreads();  // s_warp free for the next call
}

// --------------------------------------------------------------- compress ---

// The scans over the buffers run on several CTAs: each takes a run of buffers and
// sums what precedes its run itself -- independent loads, where one CTA went
// through the buffers 1024 at a time behind four barriers each (4096 buffers:
// benc_setup 21 -> 9 us, benc_place 26 -> 9, bdec_setup 14 -> 8).  256
// buffers a CTA, so that its 1024 threads share the regions of few buffers; at
// most kScanCtas, so that the repeated reads stay a small multiple of the
// buffers, and then up to 1024 buffers a step.
constexpr uint32_t kScanCtas = 64, kScanMin = 256;
__device__ __forceinline__ uint64_t scan_run(uint32_t count) {  // buffers per CTA
    const uint64_t per = ((uint64_t)count + gridDim.x - 1) / gridDim.x;
    const uint64_t unit = per > kScanThreads / 2 ? kScanThreads : kScanMin;
    return (per + unit - 1) / unit * unit;
}

// Sum of one u64 per thread over the CTA.
__device__ __forceinline__ uint64_t block_sum_u64(uint64_t v, uint64_t* s_warp) {
    const uint64_t w = warp_sum_u64(v);
    if ((threadIdx.x & 31) == 0) s_warp[threadIdx.x >> 5] = w;
    __syncthreads();
    const uint64_t t = warp_sum_u64(s_warp[threadIdx.x & 31]);  // 32 warps
    __syncthreads();  // s_warp free for the next call
    return t;
}

// The region size when the caller names none: 8 chunks, and larger ones where the
// batch still gives every encoder CTA (296) many of them, since each region costs
// its histogram fold, its plan and a last step that is partly empty.
// Compress in us at 8 / 16 / 32 chunks, by regions of 8 chunks: 4 KiB - 4 MiB
// buffers, 4725 regions 390 / 396 / 431, 9644: 717 / 693 / 723, 19678: 1383 /
// 1321 / 1329, 39879: 2734 / 2591 / 2558; buffers of 1 MiB, 4352: 358 / 344 /
// 351, 17408: 1209 / 1146 / 1130; of 256 KiB, 2560: 212 / 210 / 223, 10240: 653 /
// 619 / 618.  (12 and 24 chunks lie between or above.)  By the batch's own regions:
// the workspace may be one kept for larger batches.  Returns log2(chunks / 8).
__device__ __forceinline__ uint32_t default_shift(uint64_t regions) {
    return regions >= 80 * kEncCtas ? 2u : regions >= 20 * kEncCtas ? 1u : 0u;
}

// Numbers the regions, starts the encoder jobs and writes every region for the
// histogram pass (so that no CTA searches for a region's buffer there).
// base_chunks: the smallest region size, 0: default_shift.
__global__ void __launch_bounds__(kScanThreads) benc_setup_kernel(uint32_t count, const uint8_t* const* inputs,
                                                                  const uint64_t* sizes,
                                                                  const uint8_t* region_chunks,
                                                                  uint32_t base_chunks, EncJob* jobs,
                                                                  uint64_t* item0s, HistRegion* regions,
                                                                  uint64_t* nitems, uint64_t max_regions,
                                                                  uint32_t* status) {
    __shared__ uint64_t s_warp[32];
    __shared__ const uint8_t* s_in[kScanThreads];   // of 1024 buffers: aligned input, last byte, first region
    __shared__ uint64_t s_hi[kScanThreads];
    __shared__ uint32_t s_item0[kScanThreads + 1], s_st[kScanThreads];  // and region size, lo in its upper half
    struct Buf {
        const uint8_t* in;
        uint64_t n, nst;
        uint32_t lo, st;
    };
    uint32_t base = base_chunks;
    auto load = [&](uint64_t j) {
        Buf b = {nullptr, 0, 0, 0, 0};
        if (j < count) {
            b.n = sizes[j];
            b.in = inputs[j];
            uint32_t rc = region_chunks ? region_chunks[j] : base;
            if (rc < base) rc = base;
            if (rc > 32) rc = 32;
            b.lo = (uint32_t)(reinterpret_cast<uintptr_t>(b.in) & 15);
            b.st = rc * (uint32_t)kEncChunkBytes;
            b.nst = b.n ? (b.lo + b.n + b.st - 1) / b.st : 0;
        }
        return b;
    };
    const uint64_t run = scan_run(count), first = blockIdx.x * run;
    const uint64_t end = first + run < count ? first + run : count;
    uint64_t sum = 0;
    if (base) {
        for (uint64_t j = threadIdx.x; j < first && j < count; j += kScanThreads) sum += load(j).nst;
    } else {  // the regions of 8 chunks in all buffers, and of every size before this CTA's run
        uint64_t all = 0, before[3] = {};
        for (uint64_t j = threadIdx.x; j < count; j += kScanThreads) {
            const uint64_t n = sizes[j], end = n ? n + (reinterpret_cast<uintptr_t>(inputs[j]) & 15) : 0;
#pragma unroll
            for (uint32_t k = 0; k < 3; ++k) {
                const uint32_t st = (8u << k) * kEncChunkBytes;
                const uint64_t nst = (end + st - 1) / st;
                if (k == 0) all += nst;
                if (j < first) before[k] += nst;
            }
        }
        const uint32_t k = default_shift(block_sum_u64(all, s_warp));
        base = 8u << k;
        sum = k == 0 ? before[0] : k == 1 ? before[1] : before[2];
    }
    uint64_t carry = block_sum_u64(sum, s_warp);
    for (uint64_t base = first; base < end; base += kScanThreads) {
        const uint64_t j = base + threadIdx.x;
        const Buf b = load(j < end ? j : count);
        uint64_t total = 0;
        const uint64_t excl = block_excl_scan_u64(b.nst, &total, s_warp);
        if (j < end) {
            EncJob J;
            memset(&J, 0, sizeof(J));
            J.in_aligned = b.in - b.lo;
            J.lo = b.lo;
            J.hi = b.lo + b.n;
            J.item0 = carry + excl;
            J.nst = b.nst;
            J.st_bytes = b.st;
            jobs[j] = J;
            item0s[j] = carry + excl;
        }
        // the regions of these buffers, spread over the threads (their number per buffer varies widely)
        s_in[threadIdx.x] = b.in - b.lo;
        s_hi[threadIdx.x] = b.lo + b.n;
        s_st[threadIdx.x] = b.st | b.lo;  // (a multiple of 8 KiB, and less than 16)
        s_item0[threadIdx.x] = (uint32_t)excl;
        __syncthreads();
        const uint64_t fit = carry < max_regions ? max_regions - carry : 0, todo = total < fit ? total : fit;
        for (uint64_t r = threadIdx.x; r < todo; r += kScanThreads) {
            uint32_t lo = 0, hi = kScanThreads;  // the last buffer with item0 <= r
            while (hi - lo > 1) {
                const uint32_t mid = (lo + hi) >> 1;
                if (s_item0[mid] <= r) lo = mid;
                else hi = mid;
            }
            const uint32_t st = s_st[lo] & ~15u;
            const uint64_t k = r - s_item0[lo], v = k * st, left = s_hi[lo] - v;
            HistRegion R;
            R.in = s_in[lo] + v;
            R.lo = k == 0 ? s_st[lo] & 15u : 0u;
            R.hi = left < st ? (uint32_t)left : st;
            R.job = (uint32_t)(base + lo);
            R.pad[0] = R.pad[1] = R.pad[2] = 0;
            regions[carry + r] = R;
        }
        carry += total;
        __syncthreads();
    }
    if (threadIdx.x == 0 && first < count && first + run >= count) {  // the last CTA's run
        item0s[count] = carry;
        // a workspace smaller than the query asked for: nothing is encoded
        if (carry > max_regions) atomicOr(status, kDevSize);
        *nitems = carry > max_regions ? 0 : carry;
    }
}

// The codebook of histogram h, on one warp.  Optional outputs (book j's): the
// public codebook, sizes, encoder table, batch entry.
template <class W>
__device__ __forceinline__ void make_book(const uint32_t* h, BookScratch<W>& s, uint32_t lane, uint32_t j,
                                          hgap_codebook* books, hgap_sizes* sizes, EncTable* enc,
                                          hgap_batch_entry* entries, const uint64_t* in_sizes) {
    const uint32_t n = warp_code_lengths(h, s, lane);
    warp_assign_codes(s, n, lane);
    uint64_t part = 0;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        const uint32_t b = lane + 32 * k;
        part += (uint64_t)h[b] * s.blen[b];
    }
    const uint64_t bits = warp_sum_u64(part);
    const uint64_t words = (bits + 31) / 32, segs = (bits + 127) / 128;
    if (books) warp_write_book(s.syms, n, books + j, lane);
    if (enc) warp_write_enc_table(s.syms, n, enc + j, lane);
    if (sizes && lane == 0) {
        sizes[j].bits = bits;
        sizes[j].words = words;
        sizes[j].segments = segs;
        sizes[j].gap_words = (segs + 7) / 8;
    }
    if (entries) {
        hgap_batch_entry& e = entries[j];
        for (uint32_t c = lane; c < n; c += 32) {
            e.symbols[c].symbol = s.syms.sym[c];
            e.symbols[c].length = s.syms.clen[c];
        }
        if (lane == 0) {
            e.n = in_sizes ? in_sizes[j] : 0;
            e.bits = bits;
            e.words = words;
            e.segments = segs;
            e.gap_words = (segs + 7) / 8;
            e.symbol_count = n;
            e.status = 0;
        }
    }
    __syncwarp();
}

__global__ void __launch_bounds__(32 * kBookWarps, 16) book_kernel(uint32_t count, const uint32_t* hists,
                                                               hgap_codebook* books, hgap_sizes* sizes,
                                                               EncTable* enc, hgap_batch_entry* entries,
                                                               const uint64_t* in_sizes) {
    extern __shared__ __align__(16) unsigned char book_smem[];
    __shared__ uint32_t s_large[kBookWarps];
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (uint64_t j0 = (uint64_t)blockIdx.x * kBookWarps; j0 < count; j0 += (uint64_t)gridDim.x * kBookWarps) {
        const uint32_t j = (uint32_t)(j0 + warp);
        bool large = false;
        if (j0 + warp < count) {
            const uint32_t* h = hists + 256 * (uint64_t)j;
            uint64_t sum = 0;
#pragma unroll
            for (int k = 0; k < 8; ++k) sum += h[lane + 32 * k];
            large = warp_sum_u64(sum) >= kBook32;
            if (!large)
                make_book(h, reinterpret_cast<Book32*>(book_smem)[warp], lane, j, books, sizes, enc, entries, in_sizes);
        }
        if (lane == 0) s_large[warp] = large;
        __syncthreads();
        if (warp == 0) {
            for (uint32_t k = 0; k < (uint32_t)kBookWarps; ++k)
                if (s_large[k])
                    make_book(hists + 256 * (j0 + k), *reinterpret_cast<Book64*>(book_smem), lane, (uint32_t)j0 + k, books,
                              sizes, enc, entries, in_sizes);
        }
        __syncthreads();
    }
}

// Places every stream in the arenas (bitstreams 16-byte aligned) and
// completes the encoder jobs.
__global__ void __launch_bounds__(kScanThreads) benc_place_kernel(uint32_t count, hgap_batch_entry* entries,
                                                                  EncJob* jobs, uint32_t* bits,
                                                                  uint64_t bits_cap, uint32_t* gaps,
                                                                  uint64_t gaps_cap, uint32_t* status) {
    __shared__ uint64_t s_warp[2][32];
    const uint64_t run = scan_run(count), first = blockIdx.x * run;
    uint64_t cb = 0, cg = 0;
    for (uint64_t j = threadIdx.x; j < first && j < count; j += kScanThreads) {
        cb += (entries[j].words + 3) & ~3ull;
        cg += entries[j].gap_words;
    }
    cb = block_sum_u64(cb, s_warp[0]);
    cg = block_sum_u64(cg, s_warp[1]);
    const uint64_t end = first + run < count ? first + run : count;
    for (uint64_t base = first; base < end; base += kScanThreads) {
        const uint64_t j = base + threadIdx.x;
        uint64_t words = 0, gap_words = 0, segments = 0;
        if (j < end) {
            words = entries[j].words;
            gap_words = entries[j].gap_words;
            segments = entries[j].segments;
        }
        uint64_t ob = (words + 3) & ~3ull, og = gap_words, tb = 0, tg = 0;
        block_excl_scan2_u64(ob, og, &tb, &tg, s_warp);
        ob += cb;
        og += cg;
        if (j < end) {
            hgap_batch_entry& e = entries[j];
            EncJob& J = jobs[j];
            e.bits_offset = ob;
            e.gaps_offset = og;
            if (ob + words > bits_cap || og + gap_words > gaps_cap) {
                e.status = HGAP_ERR_SIZE;  // the arena is too small: this stream is not written
                atomicOr(status, kDevSize);
                J.bits = bits;
                J.words = 0;
                J.gaps = gaps;
                J.gap_words = 0;
            } else {
                J.bits = bits + ob;
                J.words = words;
                J.gaps = gaps + og;
                J.gap_words = gap_words;
            }
            J.segments = segments;
            J.bits_aligned16 = 1;
        }
        cb += tb;
        cg += tg;
    }
}

// ------------------------------------------------------------- decompress ---

// 8 classes: the decoder's stage size (from the shortest code) x complete book
__constant__ int kStageRows[4] = {8, 11, 16, 32};
__device__ __forceinline__ uint32_t class_of(uint32_t min_len, bool complete) {
    const uint32_t r = min_len >= 4 ? 0 : 4 - min_len;  // stage rows 8, 11, 16, 32
    return 2 * r + (complete ? 1 : 0);
}

// The entry (dec_entry.cuh) of a P-bit window x whose first code ends inside it,
// without a branch: s1 has the code at each 11-bit window, length << 8 | byte
// (kLongCode: one that ends outside).
constexpr uint16_t kLongCode = 31 << 8;
template <uint32_t P, bool MULTI>
__device__ __forceinline__ uint32_t window_entry(const uint16_t* s1, uint32_t x) {
    constexpr uint32_t kMask = (1u << kDecPrefix) - 1;
    x <<= kDecPrefix - P;
    const uint32_t e1 = s1[x], l1 = e1 >> 8;
    const uint32_t e2 = s1[x << l1 & kMask], l12 = l1 + (e2 >> 8);
    const uint32_t two = __byte_perm(e1, e2, 0x7740);  // (the upper bytes of an e are zero)
    if (!MULTI) return l12 <= P ? two + (l12 << 16) + 0x02000000u : (e1 & 0xffu) + (l1 << 16) + 0x01000000u;
    const uint32_t e3 = s1[x << (l12 & 31) & kMask], l123 = l12 + (e3 >> 8);
    return l123 <= P  ? __byte_perm(two, e3, 0x7410) + (l123 << 24) + (2u << 29)
           : l12 <= P ? two + (l12 << 24) + (1u << 29)
                      : (e1 & 0xffu) + (l1 << 24);
}

constexpr int kTableThreads = 256;

// One CTA per buffer: checks the entry, writes the buffer's decoder table
// (DecTableW), classifies the buffer and writes its decode job (all but its
// first look-back record, which bdec_setup numbers).  One symbol a thread: a
// block scan gives its left-aligned code, and it marks the 11-bit prefix where
// that code starts; every thread then fills its own 8 prefixes with the last
// code to start at or below each (a complete book has no holes), and the entries
// of up to three symbols (dec_entry.cuh) are made from those.  Of codes longer
// than a prefix every thread writes its symbol's entries.  A book whose one
// table would be too large (DecIndex) gets two levels, the same ones as
// warp_dec_table builds (book.cuh): a block scan places the level-2 groups in
// prefix order.  Bound by instructions and the chain of barriers between the
// steps; at 32 registers a thread (no spills) eight CTAs fit an SM.  Measured for
// 4096 buffers of 4-64 KiB: 44 us (58 while one warp read the symbols, every
// prefix walked the symbol list to its own and every longer code was searched).
__global__ void __launch_bounds__(kTableThreads, 8) bdec_table_kernel(uint32_t count, const hgap_batch_entry* entries,
                                                                   const uint32_t* bits, const uint32_t* gaps,
                                                                   uint8_t* const* outputs, uint32_t tile_segs,
                                                                   uint32_t class_mask, DecTableW* wtables, uint8_t* cls,
                                                                   DecJob* jobs, uint32_t* status) {
    constexpr uint32_t P = kDecPrefix, X = kMaxLen - kDecPrefix;  // 11, 5
    constexpr uint32_t kT1 = 1u << P, kPer = kT1 / kTableThreads;  // 8 prefixes a thread
    __shared__ BookSyms s;
    __shared__ __align__(16) uint16_t s1[kT1];
    __shared__ uint16_t s_end[kT1];  // level-2 offset after each prefix's group (0 for none)
    __shared__ uint32_t s_warp[kTableThreads / 32];
    __shared__ uint32_t s_long;
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    for (uint32_t j = blockIdx.x; j < count; j += gridDim.x) {
        const hgap_batch_entry& e = entries[j];
        const uint32_t n = e.symbol_count;
        bool bad = n > 256 || e.segments != (e.words + 3) / 4 || e.gap_words != (e.segments + 7) / 8 ||
                   (e.n != 0) != (e.words != 0) || (e.n != 0 && n == 0);
        // one symbol a thread: the book's checks (as warp_load_symbols), and its left-aligned code
        if (tid < 8) s.seen[tid] = 0;
        if (tid == 0) s_long = ~0u;
        reinterpret_cast<uint4*>(s1)[tid] = make_uint4(~0u, ~0u, ~0u, ~0u);  // no code starts here
        __syncthreads();
        const bool mine = !bad && tid < n;
        uint32_t L = 0, sym = 0, prev = 0;
        bool wrong = false;
        if (mine) {
            L = e.symbols[tid].length;
            sym = e.symbols[tid].symbol;
            prev = tid ? e.symbols[tid - 1].length : 0u;
            const uint32_t bit = 1u << (sym & 31);
            wrong = L < 1 || L > (uint32_t)kMaxLen || L < prev || (atomicOr(&s.seen[sym >> 5], bit) & bit);
        }
        const uint32_t span_c = mine && !wrong ? 1u << (kMaxLen - L) : 0u;
        const uint32_t run = warp_incl_scan(span_c, lane);
        if (lane == 31) s_warp[warp] = run;
        bad = __syncthreads_or(wrong) || bad;
        const uint32_t runs = warp_incl_scan(lane < kTableThreads / 32 ? s_warp[lane] : 0u, lane);
        const uint32_t kraft = __shfl_sync(kFull, runs, kTableThreads / 32 - 1);
        const uint32_t la = (warp ? __shfl_sync(kFull, runs, warp - 1) : 0u) + run - span_c;
        if (kraft > (1u << kMaxLen)) bad = true;
        uint32_t c = kNoClass;
        if (!bad && n) {  // uniform over the CTA
            // the largest symbol index i >= from with la[i] <= v (la[0] = 0, la ascends)
            auto advance = [&](uint32_t i, uint32_t v) {
                while (i + 1 < n && s.la[i + 1] <= v) ++i;
                return i;
            };
            auto search = [&](uint32_t v) {
                uint32_t lo = 0, hi = n;
                while (hi - lo > 1) {
                    const uint32_t mid = (lo + hi) >> 1;
                    if (s.la[mid] <= v) lo = mid;
                    else hi = mid;
                }
                return lo;
            };
            auto entry = [&](uint32_t i, uint32_t v) -> uint16_t {
                const uint32_t l = s.clen[i];
                if (v < s.la[i] || v - s.la[i] >= (1u << (kMaxLen - l))) return kDecInvalid;
                return (uint16_t)(((l - 1) << 8) | s.sym[i]);
            };
            // the class, and the shape of its table
            const bool complete = kraft == (1u << kMaxLen);
            const uint32_t cc = class_of(e.symbols[0].length, complete);
            const int rows = kStageRows[cc >> 1];
            const uint32_t Pr = dec_prefix(rows);
            if (mine) {
                s.la[tid] = la;
                s.sym[tid] = (uint8_t)sym;
                s.clen[tid] = (uint8_t)L;
                s1[la >> X] = L > P ? kLongCode : (uint16_t)((L << 8) | sym);  // (one code, or all long ones)
                if (L > Pr && prev <= Pr) s_long = la >> (kMaxLen - Pr);
            }
            __syncthreads();
            const uint32_t x0 = kPer * tid;
            if (complete) {  // every 11-bit prefix's code: the last one to start at or below it
                uint4* const own = reinterpret_cast<uint4*>(s1) + tid;
                uint4 q = *own;
                uint32_t* const h = &q.x;
                uint32_t cur = h[0] & 0xffffu;
                if (cur == 0xffffu) {
                    const uint32_t i = search(x0 << X);  // (shorter than P bits, or a code would start here)
                    cur = ((uint32_t)s.clen[i] << 8) | s.sym[i];
                }
#pragma unroll
                for (uint32_t k = 0; k < kPer / 2; ++k) {
                    const uint32_t lo = h[k] & 0xffffu, hi = h[k] >> 16;
                    const uint32_t e0 = lo == 0xffffu ? cur : lo;
                    cur = hi == 0xffffu ? e0 : hi;
                    h[k] = e0 | (cur << 16);
                }
                *own = q;
            }
            __syncthreads();
            const DecIndex ix = dec_index(s_long < 1u << Pr ? s_long : 1u << Pr, s.clen[n - 1], complete, rows);
            const bool multi = dec_multi(rows, complete);
            DecTableW& w = wtables[j];
            if (ix.first_long != kDecWide) {
                c = cc;
                if (multi)
                    for (uint32_t i = tid; i < ix.first_long; i += kTableThreads)
                        w.t1[i] = window_entry<dec_prefix(32), true>(s1, i);
                else
                    for (uint32_t i = tid; i < ix.first_long; i += kTableThreads)
                        w.t1[i] = window_entry<kDecPrefix, false>(s1, i);
                // the longer codes: each thread its symbol's entries, and the padding to whole 16 bytes
                const uint32_t len = 32 - ix.shift;  // the longest, or the prefix's if none is longer
                const uint32_t end = (1u << len) + ix.offset;
                if (mine && L > Pr) {
                    const uint32_t v = (((L - 1) << 8) | sym);
                    const uint32_t e1 = multi ? entry_single<true>(v) : entry_single<false>(v);
                    uint32_t* const at = w.t1 + (int32_t)(la >> (kMaxLen - len)) + ix.offset;
                    for (uint32_t k = 0; k < 1u << (len - L); ++k) at[k] = e1;
                }
                if (tid < ix.used - end) w.t1[end + tid] = kEntInvalid;
            } else {
                // two levels: the level-1 entries, and the widths of this thread's pointer prefixes
                uint32_t span = 0, pmask = 0;
                const uint32_t i_start = search(x0 << X);
                uint32_t i_first = i_start, i_last = i_first;
                for (uint32_t k = 0; k < kPer; ++k) {
                    const uint32_t x = x0 + k;
                    const uint32_t v = x << X;
                    i_first = advance(i_first, v);
                    i_last = advance(i_last > i_first ? i_last : i_first, v | ((1u << X) - 1));
                    const uint32_t l = s.clen[i_last];
                    if (l > P && (s.la[i_last] >> X) == x) {
                        span += 1u << (l - P);
                        pmask |= 1u << k;
                    } else {
                        s1[x] = entry(i_first, v);
                    }
                }
                // block scan of the spans: the level-2 offset of this thread's first group
                const uint32_t incl = warp_incl_scan(span, lane);
                if (lane == 31) s_warp[warp] = incl;
                __syncthreads();
                const uint32_t wt = warp_incl_scan(lane < kTableThreads / 32 ? s_warp[lane] : 0u, lane);
                const uint32_t total = __shfl_sync(kFull, wt, kTableThreads / 32 - 1);
                uint32_t off = (warp ? __shfl_sync(kFull, wt, warp - 1) : 0u) + incl - span;
                if (total <= (uint32_t)kDecT2Cap) {  // uniform; larger only for an incomplete book
                    // (one decoder launch serves the incomplete books of every shortest code: only
                    // hand-made ones and those of a single symbol are incomplete)
                    c = complete ? cc : kIncomplete;
                    // pass 2: the pointer prefixes, and every prefix's level-2 end offset
                    i_first = i_start;
                    for (uint32_t k = 0; k < kPer; ++k) {
                        const uint32_t x = x0 + k;
                        const uint32_t v = x << X;
                        i_first = advance(i_first, v);
                        if (pmask >> k & 1u) {
                            i_last = advance(i_first, v | ((1u << X) - 1));
                            const uint32_t wd = s.clen[i_last] - P;
                            s1[x] = (uint16_t)(0x8000u | (wd << 12) | off);
                            off += 1u << wd;
                        }
                        s_end[x] = (uint16_t)off;
                    }
                    __syncthreads();
                    // the level-2 entries, spread over all threads (the pointer prefixes sit
                    // together at the top of the code space, so per-prefix ownership would leave
                    // a few threads with hundreds of entries): entry k belongs to the first prefix
                    // whose end offset exceeds k
                    const uint32_t used = (total + 7) & ~7u;  // whole 16-byte groups, the tail invalid
                    for (uint32_t k = tid; k < used; k += kTableThreads) {
                        uint16_t e2 = kDecInvalid;
                        if (k < total) {
                            uint32_t lo = 0, hi = kT1 - 1;
                            while (lo < hi) {
                                const uint32_t mid = (lo + hi) >> 1;
                                if (s_end[mid] > k) hi = mid;
                                else lo = mid + 1;
                            }
                            const uint32_t e1 = s1[lo];  // a pointer entry: width and start of its group
                            const uint32_t wd = (e1 >> 12) & 7u;
                            const uint32_t vy = (lo << X) | ((k - (e1 & 0xfffu)) << (X - wd));
                            e2 = entry(search(vy), vy);
                        }
                        w.t2()[k] = e2;
                    }
                    for (uint32_t i = tid; i < kT1; i += kTableThreads)
                        w.t1[i] = multi ? entry_multi<kDecPrefix>(s1, i) : entry_pair<kDecPrefix>(s1, i);
                } else {
                    bad = true;
                }
            }
            if (!bad && e.segments && class_mask && !(class_mask >> cc & 1u)) {
                // a class the caller left out of the launch: the buffer stays undecoded
                if (tid == 0) atomicOr(status, kDevPlan);
                c = kNoClass;
            }
            if (c != kNoClass) {
                if (mine) w.symlen[sym] = (uint8_t)L;
                if (tid == 0) w.index = ix;
            }
        }
        if (tid == 0) {
            if (bad) {
                atomicOr(status, kDevCorrupt);
                c = kNoClass;
            }
            cls[j] = (uint8_t)c;
            // the buffer's decode job (its first look-back record comes from bdec_setup)
            uint64_t nt = 0;
            if (c != kNoClass) {  // tiles of the class's decoder
                const uint64_t segs = dec_tile_segs_for(dec_stage_rows(c / 2 == 0 ? 4 : 4 - c / 2), tile_segs);
                nt = (e.segments + segs - 1) / segs;
            }
            DecJob J;
            memset(&J, 0, sizeof(J));
            J.bits = bits + e.bits_offset;
            J.words = e.words;
            J.gaps = gaps + e.gaps_offset;
            J.gap_words = e.gap_words;
            J.segments = e.segments;
            uint8_t* out = outputs[j];
            J.out_lo = reinterpret_cast<uintptr_t>(out) & 15;
            J.out_aligned = out - J.out_lo;
            J.n = e.n;
            J.ntiles = nt;
            jobs[j] = J;
        }
        __syncthreads();  // s and s1 are reused for the next buffer
    }
}

// The look-back record numbering over all buffers' tiles, and per class the
// numbering of the class's tiles (the jobs come from bdec_table).  Per 1024
// buffers: nine warp scans of the tile counts (all tiles, and one per class with
// the other classes' buffers counting 0) need no barrier; nine warps then scan
// the 32 warp totals of one sum each, between two barriers, and every buffer
// writes its record and, for its own class only, its first class tile (the
// only entry the map and the decoder read).
__global__ void __launch_bounds__(kScanThreads) bdec_setup_kernel(uint32_t count, const uint8_t* cls, DecJob* jobs,
                                                                  uint64_t* item0s, uint64_t* class_nitems,
                                                                  uint64_t tiles_cap, uint32_t* status) {
    constexpr uint32_t kSums = kClasses + 1;  // the classes, then all tiles
    constexpr uint32_t kWarps = kScanThreads / 32;
    __shared__ uint64_t s_tot[2][kSums][kWarps];  // by chunk parity: warp totals, then warp offsets
    __shared__ uint64_t s_carry[kSums];           // the sums over the earlier chunks
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint64_t run = scan_run(count), first = blockIdx.x * run;
    if (first >= count) return;  // (uniform)
    {
        uint64_t sum[kSums] = {};
        for (uint64_t j = threadIdx.x; j < first; j += kScanThreads) {
            const uint32_t c = cls[j];
            const uint64_t nt = jobs[j].ntiles;  // 0 for a buffer in no class
#pragma unroll
            for (uint32_t k = 0; k < kSums; ++k) sum[k] += k == kClasses || c == k ? nt : 0;
        }
#pragma unroll
        for (uint32_t k = 0; k < kSums; ++k) {
            const uint64_t w = warp_sum_u64(sum[k]);
            if (lane == 0) s_tot[0][k][warp] = w;
        }
        __syncthreads();
        if (warp < kSums) {
            const uint64_t w = warp_sum_u64(s_tot[0][warp][lane]);
            if (lane == 0) s_carry[warp] = w;
        }
        __syncthreads();
    }
    uint32_t par = 0;
    const uint64_t end = first + run < count ? first + run : count;
    for (uint64_t base = first; base < end; base += kScanThreads, par ^= 1u) {
        const uint64_t j = base + threadIdx.x;
        uint32_t c = kNoClass;
        uint64_t nt = 0;
        if (j < end) {
            c = cls[j];
            nt = jobs[j].ntiles;
        }
        uint64_t x_all = nt, x_own = 0;
        for (uint32_t k = 0; k < kSums; ++k) {
            uint64_t x = k == kClasses ? nt : (c == k ? nt : 0);
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const uint64_t t = __shfl_up_sync(kFull, x, d);
                if (lane >= (uint32_t)d) x += t;
            }
            if (lane == 31) s_tot[par][k][warp] = x;
            if (k == kClasses) x_all = x;
            else if (c == k) x_own = x;
        }
        __syncthreads();
        if (warp < kSums) {
            const uint64_t v = s_tot[par][warp][lane];
            uint64_t x = v;
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const uint64_t t = __shfl_up_sync(kFull, x, d);
                if (lane >= (uint32_t)d) x += t;
            }
            const uint64_t carry = s_carry[warp];
            __syncwarp();
            s_tot[par][warp][lane] = carry + x - v;
            if (lane == 31) s_carry[warp] = carry + x;
        }
        __syncthreads();
        if (j < end) {
            jobs[j].item0 = s_tot[par][kClasses][warp] + x_all - nt;
            if (c < kClasses) item0s[(uint64_t)c * (count + 1) + j] = s_tot[par][c][warp] + x_own - nt;
        }
    }
    if (first + run < count) return;  // the last CTA's run completes the sums
    // (the last chunk's second barrier orders every s_carry update before these reads)
    const uint64_t all = s_carry[kClasses];
    // a workspace smaller than the query asked for: nothing is decoded
    const bool fits = all <= tiles_cap;
    if (threadIdx.x == 0 && !fits) atomicOr(status, kDevSize);
    if (threadIdx.x < kClasses) {
        const uint64_t tk = s_carry[threadIdx.x];
        item0s[(uint64_t)threadIdx.x * (count + 1) + count] = tk;
        class_nitems[threadIdx.x] = fits ? tk : 0;
    }
}

// tile -> job map of each class: job_of[k * cap + item] = job
__global__ void bdec_map_kernel(uint32_t count, const DecJob* jobs, const uint8_t* cls, const uint64_t* item0s,
                                uint32_t* job_of, uint64_t cap) {
    const uint32_t lane = threadIdx.x & 31;
    for (uint32_t j = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); j < count;
         j += gridDim.x * (blockDim.x >> 5)) {
        const uint32_t c = cls[j];
        if (c == kNoClass) continue;
        const uint64_t i0 = item0s[(uint64_t)c * (count + 1) + j];
        const uint64_t nt = jobs[j].ntiles;
        for (uint64_t t = lane; t < nt; t += 32)
            if (i0 + t < cap) job_of[(uint64_t)c * cap + i0 + t] = j;
    }
}

// One warp per book: the decoder table of a public codebook.
__global__ void __launch_bounds__(32 * kBookWarps) dec_table_kernel(uint32_t count, const hgap_codebook* books,
                                                                    uint16_t* tables, uint32_t* status) {
    __shared__ BookSyms scratch[kBookWarps];
    BookSyms& s = scratch[threadIdx.x >> 5];
    const uint32_t lane = threadIdx.x & 31;
    for (uint32_t j = blockIdx.x * kBookWarps + (threadIdx.x >> 5); j < count; j += gridDim.x * kBookWarps) {
        const uint32_t n = books[j].symbol_count;
        DecTable* t = reinterpret_cast<DecTable*>(tables + (uint64_t)j * (HGAP_DEC_T1_ENTRIES + HGAP_DEC_T2_ENTRIES));
        bool ok = n >= 1 && n <= 256;
        if (ok) {
            const uint32_t kraft = warp_load_symbols(books[j].symbols, n, s, lane);
            ok = kraft != ~0u && warp_dec_table(s, n, t, lane);
        }
        if (!ok && lane == 0 && status) atomicOr(status + j, 1u);
        __syncwarp();
    }
}

// --------------------------------------------------------- host helpers ---

template <class K>
cudaError_t set_book_smem(K kern) {
    return cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kBookSmem);
}

// One warp per book (or buffer), every CTA launched at once: the block
// scheduler starts each as a slot frees.
unsigned book_grid(uint32_t count) {
    const uint64_t want = (count + kBookWarps - 1) / kBookWarps;
    const uint64_t cap = 1u << 24;
    return (unsigned)(want < cap ? (want ? want : 1) : cap);
}

unsigned scan_grid(uint32_t count) {
    const uint32_t want = (uint32_t)(((uint64_t)count + kScanMin - 1) / kScanMin);
    return want < 1 ? 1 : want < kScanCtas ? want : kScanCtas;
}

// One CTA per buffer: the block scheduler hands a buffer to whichever SM frees
// a slot first, where a grid of a fixed multiple of the SMs that looped over
// the buffers started its last CTAs only after the first ones' loops ended.
unsigned table_grid(uint32_t count) {
    constexpr uint32_t kMax = 1u << 24;
    return count < kMax ? (count ? count : 1) : kMax;
}

size_t align256(size_t x) { return (x + 255) & ~(size_t)255; }

uint32_t base_chunks(const hgap_batch_config* cfg) {
    uint32_t rc = cfg && cfg->region_chunks ? cfg->region_chunks : 8;
    return rc > 32 ? 32 : rc;
}

// Compress workspace: [header 1024: status @0, counters @4 (three), nitems @64] [hists]
// [st_rec] (zero at the start of a call, together: one memset) [jobs] [item0s]
// [tables] [plan] [st_hist], the per-region arrays (st_rec, plan, st_hist) for
// as many regions as the workspace holds.
constexpr size_t kEncPerRegion = 8 + sizeof(EncRegion) + 1024;

struct EncLayout {
    size_t jobs, item0s, tables, hists, st_rec, plan, st_hist, fixed;
    uint64_t max_regions;
};

EncLayout enc_layout(uint32_t count, size_t workspace_bytes) {
    EncLayout L;
    const size_t jobs = align256(sizeof(EncJob) * (size_t)count), item0s = align256(8 * ((size_t)count + 1));
    const size_t tables = align256(sizeof(EncTable) * (size_t)count);
    L.hists = 1024;
    L.st_rec = L.hists + 1024 * (size_t)count;
    L.fixed = L.st_rec + jobs + item0s + tables;
    L.max_regions = workspace_bytes > L.fixed + 512 ? (workspace_bytes - L.fixed - 512) / kEncPerRegion : 0;
    L.jobs = align256(L.st_rec + 8 * (size_t)L.max_regions);
    L.item0s = L.jobs + jobs;
    L.tables = L.item0s + item0s;
    L.plan = L.tables + tables;
    L.st_hist = align256(L.plan + sizeof(EncRegion) * (size_t)L.max_regions);
    return L;
}

uint64_t worst_regions(uint32_t count, const uint64_t* sizes, const hgap_batch_config* cfg) {
    const uint64_t st = (uint64_t)base_chunks(cfg) * kEncChunkBytes;
    uint64_t r = 0;
    for (uint32_t j = 0; j < count; ++j) r += sizes[j] ? (sizes[j] + 15 + st - 1) / st : 0;
    return r;
}

// Decompress workspace: [header 1024: status @0, counters[8] @64, class nitems[8] @128]
// [records] (zero at the start of a call, together) [jobs] [widened tables] [classes]
// [item0s 8 x (count+1)] [job_of 8 x cap], the per-tile arrays (records, job_of) for as
// many tiles as the workspace holds.
constexpr size_t kDecPerTile = 8 + 4 * kClasses;

struct DecLayout {
    size_t jobs, wtables, cls, item0s, records, job_of, fixed;
    uint64_t tiles_cap;
};

DecLayout dec_layout(uint32_t count, size_t workspace_bytes) {
    DecLayout L;
    const size_t jobs = align256(sizeof(DecJob) * (size_t)count), wtables = align256(sizeof(DecTableW) * (size_t)count);
    const size_t cls = align256((size_t)count), item0s = align256(8 * (size_t)kClasses * ((size_t)count + 1));
    L.records = 1024;
    L.fixed = L.records + jobs + wtables + cls + item0s;
    L.tiles_cap = workspace_bytes > L.fixed + 256 ? (workspace_bytes - L.fixed - 256) / kDecPerTile : 0;
    L.jobs = align256(L.records + 8 * (size_t)L.tiles_cap);
    L.wtables = L.jobs + jobs;
    L.cls = L.wtables + wtables;
    L.item0s = L.cls + cls;
    L.job_of = L.item0s + item0s;
    return L;
}

uint64_t worst_tiles(uint32_t count, const uint64_t* sizes) {
    // a stream has at most ceil(n / 8) segments (16-bit codes): ceil(n / 2048) tiles of 256
    uint64_t cap = 0;
    for (uint32_t j = 0; j < count; ++j) cap += (sizes[j] + 2047) / 2048;
    return cap;
}

inline hgap_status cuda_status(int e) { return e == 0 ? HGAP_OK : HGAP_ERR_CUDA; }

}  // namespace
}  // namespace hgap

using namespace hgap;

extern "C" {

hgap_status hgap_codebook_build_device(uint32_t count, const uint32_t* d_hists, hgap_codebook* d_books,
                                       hgap_sizes* d_sizes, hgap_stream_t stream) {
    if (count == 0) return HGAP_OK;
    if (!d_hists || !d_books) return HGAP_ERR_INVALID_ARG;
    if (set_book_smem(book_kernel) != cudaSuccess) return HGAP_ERR_CUDA;
    book_kernel<<<book_grid(count), 32 * kBookWarps, kBookSmem, reinterpret_cast<cudaStream_t>(stream)>>>(
        count, d_hists, d_books, d_sizes, nullptr, nullptr, nullptr);
    return cuda_status(cudaGetLastError());
}

hgap_status hgap_decode_table_build_device(uint32_t count, const hgap_codebook* d_books, uint16_t* d_tables,
                                           uint32_t* d_status, hgap_stream_t stream) {
    if (count == 0) return HGAP_OK;
    if (!d_books || !d_tables) return HGAP_ERR_INVALID_ARG;
    dec_table_kernel<<<book_grid(count), 32 * kBookWarps, 0, reinterpret_cast<cudaStream_t>(stream)>>>(
        count, d_books, d_tables, d_status);
    return cuda_status(cudaGetLastError());
}

size_t hgap_batch_compress_workspace_bytes(uint32_t count, const uint64_t* sizes, const hgap_batch_config* cfg) {
    if (count && !sizes) return 0;
    const EncLayout L = enc_layout(count, 0);
    return L.fixed + 256 + kEncPerRegion * (size_t)worst_regions(count, sizes, cfg) + 256;
}

size_t hgap_batch_decompress_workspace_bytes(uint32_t count, const uint64_t* sizes) {
    if (count && !sizes) return 0;
    const DecLayout L = dec_layout(count, 0);
    return L.fixed + 256 + kDecPerTile * (size_t)worst_tiles(count, sizes) + 256;
}

uint64_t hgap_batch_bits_capacity(uint32_t count, const uint64_t* sizes) {
    uint64_t w = 0;  // at most 16 bits per byte, each stream rounded up to 4 words
    for (uint32_t j = 0; j < count; ++j) w += ((sizes[j] * 16 + 31) / 32 + 3) & ~3ull;
    return w;
}

uint64_t hgap_batch_gaps_capacity(uint32_t count, const uint64_t* sizes) {
    uint64_t g = 0;
    for (uint32_t j = 0; j < count; ++j) g += ((sizes[j] * 16 + 127) / 128 + 7) / 8;
    return g;
}

hgap_status hgap_batch_compress(uint32_t count, const uint8_t* const* d_inputs, const uint64_t* d_sizes,
                                const uint8_t* d_region_chunks, uint32_t* d_bits, uint64_t bits_capacity,
                                uint32_t* d_gaps, uint64_t gaps_capacity, hgap_batch_entry* d_entries,
                                void* d_workspace, size_t workspace_bytes, const hgap_batch_config* cfg,
                                hgap_stream_t stream) {
    if (count == 0) return HGAP_OK;
    if (!d_inputs || !d_sizes || !d_bits || !d_gaps || !d_entries || !d_workspace) return HGAP_ERR_INVALID_ARG;
    if ((reinterpret_cast<uintptr_t>(d_workspace) & 255) || (reinterpret_cast<uintptr_t>(d_bits) & 15) ||
        (reinterpret_cast<uintptr_t>(d_gaps) & 3))
        return HGAP_ERR_INVALID_ARG;
    const hgap_batch_config dflt = {0, 0, 0, 0, 0, 0};
    if (!cfg) cfg = &dflt;
    const EncLayout L = enc_layout(count, workspace_bytes);
    if (L.max_regions == 0) return HGAP_ERR_WORKSPACE;
    uint8_t* ws = static_cast<uint8_t*>(d_workspace);
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    uint32_t* status = reinterpret_cast<uint32_t*>(ws);
    uint64_t* nitems = reinterpret_cast<uint64_t*>(ws + 64);
    EncJob* jobs = reinterpret_cast<EncJob*>(ws + L.jobs);
    uint64_t* item0s = reinterpret_cast<uint64_t*>(ws + L.item0s);
    EncTable* tables = reinterpret_cast<EncTable*>(ws + L.tables);
    uint32_t* hists = reinterpret_cast<uint32_t*>(ws + L.hists);
    uint64_t* st_rec = reinterpret_cast<uint64_t*>(ws + L.st_rec);
    uint32_t* st_hist = reinterpret_cast<uint32_t*>(ws + L.st_hist);
    EncRegion* plan = reinterpret_cast<EncRegion*>(ws + L.plan);
    // (the histogram pass is done with its regions before the plan is made in their place)
    static_assert(sizeof(HistRegion) <= sizeof(EncRegion), "one array for both");
    HistRegion* hist_regions = reinterpret_cast<HistRegion*>(plan);

    // (per-buffer sizes are the caller's choice too)
    const uint32_t chunks = cfg->region_chunks || d_region_chunks ? base_chunks(cfg) : 0;
    if (cudaMemsetAsync(ws, 0, L.st_rec + 8 * (size_t)L.max_regions, st) != cudaSuccess) return HGAP_ERR_CUDA;
    benc_setup_kernel<<<scan_grid(count), kScanThreads, 0, st>>>(count, d_inputs, d_sizes, d_region_chunks, chunks, jobs,
                                                                 item0s, hist_regions, nitems, L.max_regions, status);
    if (cudaGetLastError() != cudaSuccess) return HGAP_ERR_CUDA;

    HistStArgs h;
    std::memset(&h, 0, sizeof(h));
    h.nitems_dev = nitems;
    h.hist = hists;
    h.st_hist = st_hist;
    h.regions = hist_regions;
    h.counter = status + 2;  // in the zeroed header, beside the encoder's region counter
    if (launch_hist_st(h, (int)cfg->hist_ctas_per_sm, stream) != 0) return HGAP_ERR_CUDA;

    if (set_book_smem(book_kernel) != cudaSuccess) return HGAP_ERR_CUDA;
    book_kernel<<<book_grid(count), 32 * kBookWarps, kBookSmem, st>>>(count, hists, nullptr, nullptr, tables,
                                                                      d_entries, d_sizes);
    if (cudaGetLastError() != cudaSuccess) return HGAP_ERR_CUDA;
    benc_place_kernel<<<scan_grid(count), kScanThreads, 0, st>>>(count, d_entries, jobs, d_bits, bits_capacity, d_gaps,
                                                  gaps_capacity, status);
    if (cudaGetLastError() != cudaSuccess) return HGAP_ERR_CUDA;

    EncArgs a;
    std::memset(&a, 0, sizeof(a));
    a.jobs = jobs;
    a.item0s = item0s;
    a.tables = tables;
    a.count = count;
    a.nitems = L.max_regions;
    a.nitems_dev = nitems;
    a.plan = plan;
    a.st_rec = st_rec;
    a.st_hist = st_hist;
    a.counter = status + 1;
    a.plan_counter = status + 3;
    a.status = status;
    EncTable unused;
    std::memset(&unused, 0, sizeof(unused));
    return cuda_status(launch_encode(a, unused, (int)cfg->enc_ctas_per_sm, stream));
}

hgap_status hgap_batch_decompress(uint32_t count, const hgap_batch_entry* d_entries, const uint32_t* d_bits,
                                  const uint32_t* d_gaps, uint8_t* const* d_outputs, void* d_workspace,
                                  size_t workspace_bytes, const hgap_batch_config* cfg, hgap_stream_t stream) {
    if (count == 0) return HGAP_OK;
    if (!d_entries || !d_bits || !d_gaps || !d_outputs || !d_workspace) return HGAP_ERR_INVALID_ARG;
    if (reinterpret_cast<uintptr_t>(d_workspace) & 255) return HGAP_ERR_INVALID_ARG;
    const hgap_batch_config dflt = {0, 0, 0, 0, 0, 0};
    if (!cfg) cfg = &dflt;
    const DecLayout L = dec_layout(count, workspace_bytes);
    if (L.tiles_cap == 0) return HGAP_ERR_WORKSPACE;
    uint8_t* ws = static_cast<uint8_t*>(d_workspace);
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    uint32_t* status = reinterpret_cast<uint32_t*>(ws);
    uint32_t* counters = reinterpret_cast<uint32_t*>(ws + 64);
    uint64_t* class_nitems = reinterpret_cast<uint64_t*>(ws + 128);
    DecJob* jobs = reinterpret_cast<DecJob*>(ws + L.jobs);
    DecTableW* wtables = reinterpret_cast<DecTableW*>(ws + L.wtables);
    uint8_t* cls = ws + L.cls;
    uint64_t* item0s = reinterpret_cast<uint64_t*>(ws + L.item0s);
    uint64_t* records = reinterpret_cast<uint64_t*>(ws + L.records);
    uint32_t* job_of = reinterpret_cast<uint32_t*>(ws + L.job_of);

    // (the workspace's room tells the buffers' average size: a tile for every 2048 bytes)
    const uint32_t tile_segs = cfg->dec_tile_segs ? cfg->dec_tile_segs
                               : L.tiles_cap < 32 * (uint64_t)count ? kDecTileSmall
                                                                    : kDecTileBatch;
    if (cudaMemsetAsync(ws, 0, L.records + 8 * (size_t)L.tiles_cap, st) != cudaSuccess) return HGAP_ERR_CUDA;
    bdec_table_kernel<<<table_grid(count), kTableThreads, 0, st>>>(count, d_entries, d_bits, d_gaps, d_outputs,
                                                                   tile_segs, cfg->dec_class_mask, wtables, cls, jobs,
                                                                   status);
    if (cudaGetLastError() != cudaSuccess) return HGAP_ERR_CUDA;
    bdec_setup_kernel<<<scan_grid(count), kScanThreads, 0, st>>>(count, cls, jobs, item0s, class_nitems, L.tiles_cap,
                                                  status);
    if (cudaGetLastError() != cudaSuccess) return HGAP_ERR_CUDA;
    bdec_map_kernel<<<book_grid(count), 32 * kBookWarps, 0, st>>>(count, jobs, cls, item0s, job_of, L.tiles_cap);
    if (cudaGetLastError() != cudaSuccess) return HGAP_ERR_CUDA;
    DecTable unused;
    std::memset(&unused, 0, sizeof(unused));
    static const uint32_t kMinLen[4] = {4, 3, 2, 1};  // a representative shortest code per stage size
    for (uint32_t c = 0; c < kClasses; ++c) {
        // complete books' classes, and one launch for all incomplete ones
        if (!(c & 1u) && c != kIncomplete) continue;
        const uint32_t named = c == kIncomplete ? 0x55u : 1u << c;
        if (cfg->dec_class_mask && !(cfg->dec_class_mask & named)) continue;
        DecArgs a;
        std::memset(&a, 0, sizeof(a));
        a.jobs = jobs;
        a.job_of = job_of + (uint64_t)c * L.tiles_cap;
        a.item0s = item0s + (uint64_t)c * (count + 1);
        a.tables = wtables;
        a.nitems_dev = class_nitems + c;
        a.lookback = records;
        a.counter = counters + c;
        a.status = status;
        // batched streams are compressible ones on the whole: always two symbols per lookup where they fit
        if (launch_decode(a, unused, kMinLen[c / 2], (c & 1) != 0, true, (int)cfg->dec_ctas_per_sm,
                          tile_segs, stream) != 0)
            return HGAP_ERR_CUDA;
    }
    return HGAP_OK;
}

uint32_t hgap_batch_decoder_class(const hgap_symlen* symbols, uint32_t count) {
    if (!symbols || count == 0) return kNoClass;
    uint32_t min_len = kMaxLen;
    uint64_t kraft = 0;
    for (uint32_t i = 0; i < count; ++i) {
        const uint32_t L = symbols[i].length;
        if (L >= 1 && L <= (uint32_t)kMaxLen) {
            min_len = L < min_len ? L : min_len;
            kraft += 1ull << (kMaxLen - L);
        }
    }
    const uint32_t r = min_len >= 4 ? 0 : 4 - min_len;
    return 2 * r + (kraft == (1ull << kMaxLen) ? 1u : 0u);
}

hgap_status hgap_batch_status(const void* d_workspace, hgap_stream_t stream) {
    return hgap_workspace_status(d_workspace, stream);
}

}  // extern "C"
