// encode.cu -- fused Huffman encoder with gap-array emission, sm_100a.
//
// Replaces cuencoder + cu_get_gaparray (encoder/src/encoder.cu:142-379) and
// produces the same bitstream and gap array bit for bit.
//
// Work unit: a region (super-tile) of st_bytes input bytes of one job, taken
// by global id by persistent CTAs of 16 warps; the single-buffer entry points
// run one job, the batched ones thousands, each with its own codebook (the
// CTA reloads its code table when the job changes).  A region's bit count is
// one dot product of its histogram (recorded by hist_st_kernel in the same
// pass that builds the global histogram) with the code lengths, so a small
// kernel before the encoder gives every region's first output bit G
// (enc_plan_kernel).  A CTA holds its next region's plan and claims the one
// after it while it encodes; nothing in the encoder waits for another CTA.
//
// Input: steps of 16 KiB are staged in a ring of shared-memory buffers by 1-D
// bulk copies (completion on an mbarrier), one step ahead of the one being
// encoded.  In a step every warp owns 1 KiB and every lane 32 consecutive
// bytes.
//
// The kernel is bound by instruction issue (8-bit symbols, integer work only),
// so the loop is built to spend few instructions per byte:
//   * one 8-byte lookup per byte, {left-aligned code, length}, from a table
//     replicated over 16 lanes ([byte][lane & 15]: a half-warp's 8-byte reads
//     each have their own bank pair);
//   * codes are joined without branches, two to a word and four to a 64-bit
//     piece, before their place in the output is known; the running lengths of
//     the piece's four codes ride in one register, a byte each (multiply-adds,
//     on the pipe that the shifts leave idle);
//   * one barrier per step: each warp publishes its bit count and its last 32
//     code bits, and then knows where its own bits start and what the word it
//     starts in holds already, so it packs, and writes, its words alone: no
//     word is shared between warps;
//   * in the warp, a lane stores the words it completes with plain shared
//     stores (32 bytes are at least 32 bits: no word sees three lanes) and
//     ORs its unfinished last word into the next lane's first;
//   * a piece that reaches a segment's end leaves its four running lengths,
//     minus the distance to that end, in a ring of records indexed by segment:
//     the first byte with its top bit set is the spill of the code that ends
//     or crosses there, which is the segment's gap entry
//     (encoder/src/encoder.cu:307-312).  One step later the records become gap
//     words, one thread to a word of eight entries.
// Bytes outside the job in a warp at one of its ends are encoded with the rest
// and masked off again, so there is one packing loop; a warp whose bits do not
// fit its image (over 10 bits a byte) packs its two halves one after the other.
// Nothing is pre-zeroed (the reference memsets its outputs, encoder.cu:412-414)
// and there are no global atomics: a region's first word is completed by
// re-encoding the bits before G, and its first gap byte likewise, so
// neighbouring regions never wait on each other.
//
// Measured (B200, kernel alone), against a loop that packed two codes at a time
// into one image of the CTA with two barriers per 8 KiB: 256 MiB of Zipf(1.2)
// 344 -> 239 us, of the mixed stream 409 -> 243, of BF16 sign|mantissa bytes
// 353 -> 254, of BF16 exponents 335 -> 237; 1024 buffers of 4 KiB - 4 MiB
// (593 MB) in 64 KiB regions 879 -> 525 us, in 256 KiB regions 791 -> 546.
// 0.74 warp instructions per byte (1.12 before) at 74 % of the issue slots.
#include <cuda_runtime.h>

#include "device_util.cuh"
#include "launch_cache.h"

namespace hgap {

constexpr int kEncThreads = 512;
constexpr int kEncWarps = kEncThreads / 32;
constexpr int kLaneBytes = 32;                        // input bytes per lane and step
constexpr int kPieces = kLaneBytes / 4;               // 64-bit pieces of four codes per lane
constexpr int kWarpBytes = 32 * kLaneBytes;
constexpr int kStepBytes = kEncWarps * kWarpBytes;    // 16 KiB
static_assert(kEncChunkBytes % kWarpBytes == 0, "a region ends on a warp's boundary");
constexpr int kRing = 2;                              // input steps staged
constexpr int kLutRep = 16;                           // table copies: one per lane of a half-warp
// Output words a warp packs at once (a multiple of 4): 10.4 bits per byte, and enough for half a
// warp's bytes at 16; 16 warps' images, the table, the ring and the records fit twice in an SM.
// The first words are slack: the up to 15 bytes before a job's first one (its 16-byte group) are
// encoded too, below its first bit, and never written out.
constexpr int kImgWords = 348;
constexpr uint32_t kSlackBits = 256;
static_assert(kSlackBits >= 15 * kMaxLen && kSlackBits % 128 == 0, "room for 15 codes, whole segments");
constexpr uint32_t kLaneMaxBits = kLaneBytes * kMaxLen;
static_assert(kImgWords % 4 == 0 && kImgWords * 32 > kSlackBits + 128 + 17 * kLaneMaxBits,
              "half a warp fits, with as much again as a lane's bytes after the job's last");
// gap records: a step closes at most 16 KiB * 16 bits / 128 = 2048 segments, and the records of
// two steps are live at once
constexpr uint32_t kRecs = 4096;
constexpr size_t kEncSmem = (size_t)256 * kLutRep * 8 + (size_t)kRing * kStepBytes +
                            (size_t)kEncWarps * kImgWords * 4 + (size_t)kRecs * 4;
constexpr uint32_t kLen4 = 0x01010101u;
constexpr uint32_t kPieceBias = 0x7f7f7f7fu;  // 0x7f + running length per byte

struct EncShared {
    uint64_t mbar[kRing];       // one per ring buffer: its bulk copy landed
    EncRegion reg[3];           // the CTA's k-th region in reg[k % 3]: the current one, the next, the one after
    EncTable next_codes;        // the next region's codes, if they are another job's
    uint32_t tot[2][kEncWarps]; // per step parity: the warps' bit counts
    // the last 32 code bits before warp w's first of step c, at [(16 c + w) % 64]: four steps, since
    // warp 0 still reads its entry when warp 15 is a step further
    uint32_t tail[4 * kEncWarps];
    uint32_t lut_job;           // job whose codes are in the table
    uint32_t p_issued;          // producer: copies issued so far (step sequence number)
    uint32_t p_step;            // producer: step index of the next copy within its region
    int p_which;                // producer: next copy from the current region (0) or the next one (1)
};

// Length and left-aligned code of an entry of a job's table.
__device__ __forceinline__ void code_of(uint32_t e, uint32_t& c, uint32_t& len) {
    len = (e >> 16) & 31u;
    c = len ? (e & 0xffffu) << (32 - len) : 0u;
}

// End of region st of job J (virtual input index, like J.lo / J.hi).
__device__ __forceinline__ uint64_t region_end(const EncJob& J, uint64_t st) {
    const uint64_t v1 = (st + 1) * (uint64_t)J.st_bytes;
    return v1 < J.hi ? v1 : J.hi;
}

constexpr int kPlanThreads = 256;
constexpr int kPlanWarps = kPlanThreads / 32;  // regions of a group

// One warp per region: its bit count (its histogram times the code lengths),
// its first output bit, and by re-encoding a few bytes backwards from there
// what precedes it in its first word and gap byte.  The counts are summed over a
// CTA's eight regions first, and the look-back runs over these groups (over
// single regions it took 13 us for the 1171 regions of 256 MiB, here 7): a
// group in which a job starts publishes the sum from there on as an inclusive
// prefix.  Groups are claimed in order, and the next one only when the current
// one's sum is published: a look-back only ever waits for CTAs that run, however
// many of the grid's CTAs the GPU has room for beside other work.
// All the regions' dependent loads overlap here, where one warp of a persistent
// encoder CTA went through them between two regions: encoder and plan of 1024
// buffers in 64 KiB regions 659 -> 542 us, of 4096 small buffers 170 -> 126, of
// one 16 MiB buffer 25 -> 26; one 256 MiB buffer pays its 7 us (237 -> 246).
__global__ void __launch_bounds__(kPlanThreads) enc_plan_kernel(const __grid_constant__ EncArgs a,
                                                                const __grid_constant__ EncTable tab) {
    __shared__ EncTable s_tab;
    const uint32_t tid = threadIdx.x, lane = tid & 31;
    uint32_t claim = 0;
    if (tid == 0) claim = atomicAdd(a.plan_counter, 1u);  // (beside the loads below)
    uint64_t nitems = a.nitems;
    if (a.jobs) {
        nitems = *a.nitems_dev;
    } else {
        s_tab.e[tid] = tab.e[tid];
        __syncthreads();
        // single path: the histograms in the workspace must come from this very input
        const bool fits = a.tag[0] == a.single.hi - a.single.lo &&
                          a.tag[1] == reinterpret_cast<uint64_t>(a.single.in_aligned) + a.single.lo;
        if (blockIdx.x == 0 && tid == 0) {
            *a.nitems_dev = fits ? nitems : 0;
            if (!fits) atomicOr(a.status, kDevPlan);
        }
        if (!fits) return;
    }
    __shared__ uint64_t s_agg[kPlanWarps], s_excl;
    __shared__ uint32_t s_first[kPlanWarps], s_next;
    const uint32_t warp = tid >> 5;
    if (tid == 0) s_next = claim;
    __syncthreads();
    for (uint64_t g = s_next; g * kPlanWarps < nitems; g = s_next) {
        const uint64_t item = g * kPlanWarps + warp;
        const bool valid = item < nitems;  // uniform over the warp
        uint32_t job = 0;
        if (a.jobs && valid) {  // the last job with item0 <= item: 32 probes a round
            uint32_t lo = 0, hi = a.count;
            while (hi - lo > 1) {
                const uint32_t step = (hi - lo + 31) / 32, at = lo + lane * step;
                const uint32_t le = __ballot_sync(kFull, at < hi && a.item0s[at] <= item);  // lane 0's always is
                const uint32_t k = 31 - __clz(le);
                lo += k * step;
                hi = lo + step < hi ? lo + step : hi;
            }
            job = lo;
        }
        const EncJob& J = a.jobs ? a.jobs[job] : a.single;
        const EncTable& T = a.jobs ? a.tables[job] : s_tab;
        const uint64_t st = item - J.item0;
        uint64_t part = 0;
        bool absent = false;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const uint32_t b = lane + 32 * j;
            const uint32_t len = (T.e[b] >> 16) & 31u;
            const uint32_t n = valid ? a.st_hist[item * 256 + b] : 0u;
            absent |= n != 0 && len == 0;
            part += (uint64_t)n * len;
        }
        if (absent) atomicOr(a.status, kDevNoCode);
        const uint64_t agg = warp_sum_u64(part);
        if (lane == 0) {
            s_agg[warp] = agg;
            s_first[warp] = valid && st == 0;
        }
        __syncthreads();
        const uint32_t starts = __ballot_sync(kFull, lane < (uint32_t)kPlanWarps && s_first[lane]);  // of jobs, in the group
        const uint64_t mine = lane < (uint32_t)kPlanWarps ? s_agg[lane] : 0;
        const bool held = a.hook.hold_plus1 && (a.hook.hold_plus1 - 1) / kPlanWarps == g;
        if (warp == 0) {
            const uint32_t from = starts ? 31 - __clz(starts) : 0u;
            const uint64_t sum = warp_sum_u64(lane >= from ? mine : 0);
            if (lane == 0 && !held) lookback_publish(a.st_rec, g, sum, starts != 0);
            if (lane == 0) claim = atomicAdd(a.plan_counter, 1u);
            const uint64_t e = lookback_resolve(a.st_rec, g, sum, (starts & 1u) != 0, a.status, lane, wait_limit(a.hook),
                                                !held && starts == 0);
            if (lane == 0) {
                s_excl = e;
                s_next = claim;
            }
        }
        // the job's bits before this region: in the group, and before it unless the job starts in it
        const uint32_t upto = starts & ((2u << warp) - 1u);
        const uint32_t from = upto ? 31 - __clz(upto) : 0u;
        uint64_t excl = warp_sum_u64(lane >= from && lane < warp ? mine : 0);
        __syncthreads();
        if (!upto) excl += s_excl;
        // (test hook: the regions after a held one in its own group wait for it, too)
        if (held && item >= a.hook.hold_plus1)
            lookback_resolve(a.st_rec, g + 1, 0, false, a.status, lane, wait_limit(a.hook), false);
        const uint64_t vfirst = st * (uint64_t)J.st_bytes;  // first byte of this region
        const uint64_t G = J.bit0 + excl;
        uint32_t head = 0, gap_head = 0;
        const uint32_t r = (uint32_t)(G & 31);
        const bool odd = ((G >> 7) & 1) != 0;
        if (valid && G > 0 && (r != 0 || odd)) {
            // walk the previous region's codes backwards from G
            const uint64_t wstart = G - r;              // the word's first bit
            const uint64_t bnd = G & ~127ull;           // the segment end at or before G
            // codes starting at or below `stop` can no longer reach the head
            // word (bits >= wstart) nor cross or end at bnd
            uint64_t stop = r ? wstart : ~0ull;
            if (odd && bnd - 1 < stop) stop = bnd - 1;
            uint64_t end = G;
            for (uint64_t base = 0;; base += 32) {  // 32 bytes a round, one per lane, going backwards
                const uint64_t v = vfirst - 1 - base - lane;  // may wrap below lo: no byte
                uint32_t c = 0, len = 0;
                if (vfirst >= base + lane + 1 && v >= J.lo) code_of(T.e[__ldg(J.in_aligned + v)], c, len);
                const uint32_t incl = warp_incl_scan(len, lane);
                const uint64_t ce = end - (incl - len);  // this code's end bit
                const uint64_t cs = ce - len;            // and start bit
                if (len) {
                    if (r && ce > wstart)  // the code's right-aligned value, placed to end at ce
                        head |= (uint32_t)(((uint64_t)(c >> (32 - len))) << (wstart + 32 - ce));
                    if (odd && cs < bnd && bnd <= ce) gap_head = (uint32_t)(ce - bnd);
                }
                const uint32_t total = __shfl_sync(kFull, incl, 31);
                end -= total;  // start of the round's last code
                if (end <= stop || total == 0) break;  // uniform
            }
            head = __reduce_or_sync(kFull, head);
            gap_head = __reduce_or_sync(kFull, gap_head);
        }
        if (lane == 0 && valid) {
            const uint64_t base = G & ~1023ull;
            auto room = [](uint64_t total, uint64_t from) {
                return total <= from ? 0u : total - from < 0x40000000ull ? (uint32_t)(total - from) : 0x40000000u;
            };
            const bool last = st + 1 == J.nst;
            EncRegion R;
            R.in = J.in_aligned + vfirst;
            R.bits = J.bits + (base >> 5);
            R.gaps = J.gaps + (base >> 10);
            R.nwords = room(J.words, base >> 5);
            R.ngaps = room(J.gap_words, base >> 10);
            R.lo = st == 0 ? (uint32_t)J.lo : 0u;
            R.hi = (uint32_t)(region_end(J, st) - vfirst);
            R.first_bit = (uint32_t)(G - base);
            R.nbits = (uint32_t)agg;
            R.tail = r ? head >> (32 - r) : 0u;
            R.gap_head = gap_head;
            R.job = job;
            R.flags = (st == 0 ? kRegionFirst : 0u) | (last ? kRegionLast : 0u) | (J.bits_aligned16 ? kRegionVec : 0u);
            R.pad[0] = R.pad[1] = 0;
            a.plan[item] = R;
            const uint64_t E = G + agg;
            if (last && ((E + 31) / 32 != J.words || (E + 127) / 128 != J.segments)) atomicOr(a.status, kDevSize);
        }
    }
}

__device__ __forceinline__ uint32_t region_steps(const EncRegion& R) { return (R.hi + kStepBytes - 1) / kStepBytes; }

// The bulk-copy producer: thread 0 at region boundaries, the last warp's first
// thread after each step's barrier (never both at once; barriers order them).
// Copies go out in the order the CTA encodes steps: the rest of region cur,
// then region next (null: not known yet); at most kRing beyond the last step
// whose buffer is free again.  Its state lives in shared memory (one thread
// touches it at a time), sparing every thread the registers.
__device__ __forceinline__ void produce(uint8_t* ring, EncShared& sh, uint32_t freed, const EncRegion* cur,
                                        const EncRegion* next) {
    uint32_t issued = sh.p_issued, ps = sh.p_step;
    int which = sh.p_which;
    while (issued < freed + kRing) {
        const EncRegion* const R = which ? next : cur;
        if (!R || R->hi == 0) break;
        if (ps >= region_steps(*R)) {
            if (which == 0) {
                which = 1;
                ps = 0;
                continue;
            }
            break;  // wait for the next region
        }
        const uint32_t v = ps * (uint32_t)kStepBytes;
        const uint32_t rem = ((R->hi + 15) & ~15u) - v;  // through the last 16-byte group
        const uint32_t bytes = rem >= (uint32_t)kStepBytes ? (uint32_t)kStepBytes : rem;
        const uint32_t s = issued % kRing;
        bulk_load(ring + s * (uint32_t)kStepBytes, R->in + v, bytes, &sh.mbar[s]);
        ++issued;
        ++ps;
    }
    sh.p_issued = issued;
    sh.p_step = ps;
    sh.p_which = which;
}

// A lane's 32 bytes as eight 64-bit pieces of four codes, left-aligned in
// hi:lo; byte b of q is 0x7f + the bits of the piece's first b + 1 codes.
struct Pieces {
    uint32_t hi[kPieces], lo[kPieces], q[kPieces];
};

__device__ __forceinline__ uint32_t piece_bits(uint32_t q) { return (q >> 24) - 0x7fu; }

// One input word (four bytes) to a piece.  `lane8`: the lane's byte offset in a
// table row.
__device__ __forceinline__ void join_piece(const uint2 (&e)[4], uint32_t& hi, uint32_t& lo, uint32_t& q) {
    // lengths are at most 16: a pair has at most 32 bits, and shifts by a pair's length clamp at 32
    const uint32_t c01 = e[0].x | __funnelshift_r(e[1].x, 0u, e[0].y);
    const uint32_t c23 = e[2].x | __funnelshift_r(e[3].x, 0u, e[2].y);
    const uint32_t l01 = e[0].y + e[1].y;
    hi = c01 | __funnelshift_rc(c23, 0u, l01);
    lo = __funnelshift_rc(0u, c23, l01);
    q = e[3].y * 0x01000000u + (e[2].y * 0x01010000u + (e[1].y * 0x01010100u + (e[0].y * kLen4 + kPieceBias)));
}

__device__ __forceinline__ void make_piece(const char* lut, uint32_t lane8, uint32_t w, uint32_t& hi, uint32_t& lo,
                                           uint32_t& q) {
    uint2 e[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const uint32_t b = __byte_perm(w, 0, 0x4440 + k);
        e[k] = *reinterpret_cast<const uint2*>(lut + (b * (kLutRep * 8) + lane8));
    }
    join_piece(e, hi, lo, q);
}

// Bits of the lane's first i bytes (i <= 32).
__device__ __forceinline__ uint32_t bits_before(const Pieces& pc, uint32_t i) {
    uint32_t n = 0;
#pragma unroll
    for (int j = 0; j < kPieces; ++j) {
        const uint32_t m = i > 4u * j ? (i - 4 * j < 4 ? i - 4 * j : 4u) : 0u;  // of piece j's four codes
        if (m) n += ((pc.q[j] >> (8 * m - 8)) & 0xffu) - 0x7fu;
    }
    return n;
}

// The last 32 bits of the lane's codes, right-aligned (all of them if fewer).
__device__ __forceinline__ uint32_t last_bits(const Pieces& pc) {
    // a piece's low 32 bits are hi:lo >> (64 - l), its bits in hi alone if l <= 32
    auto low = [](uint32_t hi, uint32_t lo, uint32_t l) {
        return l > 32 ? __funnelshift_r(lo, hi, 64 - l) : __funnelshift_rc(hi, 0u, 32 - l);
    };
    uint32_t n = piece_bits(pc.q[kPieces - 1]);
    uint32_t tail = low(pc.hi[kPieces - 1], pc.lo[kPieces - 1], n);
#pragma unroll
    for (int j = kPieces - 2; j >= 0; --j) {
        const uint32_t l = piece_bits(pc.q[j]);
        tail |= __funnelshift_lc(0u, low(pc.hi[j], pc.lo[j], l), n);  // (shifted out where n >= 32)
        n += l;
        if (j < kPieces - 2 && n >= 32) break;  // two more pieces nearly always do
    }
    return tail;
}

// Packs the lane's pieces from bit p of the warp's image on (image bit
// kSlackBits = the start of the segment that the warp's first bit is in).
// `cur` is what the lane's first word holds before p; stores every word
// completed, returns the unfinished last one, and the end bit in p.  Every
// segment end reached leaves a record (see the top): they are indexed by
// segment, rec0 = 4 * (the segment of image bit 0, minus 1).
__device__ __forceinline__ uint32_t pack(const Pieces& pc, uint32_t* img, char* recs, uint32_t rec0, uint32_t& p,
                                         uint32_t cur) {
    uint32_t a = p >> 5;
#pragma unroll
    for (int j = 0; j < kPieces; ++j) {
        const uint32_t q = pc.q[j];
        const uint32_t x = q - (~p & 127u) * kLen4;  // per byte: 0x80 + running length - distance to the segment's end
        const uint32_t x0 = cur | __funnelshift_r(pc.hi[j], 0u, p);
        const uint32_t x1 = __funnelshift_r(pc.lo[j], pc.hi[j], p);
        const uint32_t x2 = __funnelshift_r(0u, pc.lo[j], p);
        p += piece_bits(q);
        const uint32_t b = p >> 5;
        if (b != a) img[a] = x0;
        if (b > a + 1) img[a + 1] = x1;
        cur = b == a ? x0 : b == a + 1 ? x1 : x2;
        if ((int32_t)x < 0) *reinterpret_cast<uint32_t*>(recs + ((b + rec0) & (4 * kRecs - 4))) = x;
        a = b;
    }
    return cur;
}

__global__ void __launch_bounds__(kEncThreads, 2)
    encode_kernel(const __grid_constant__ EncArgs a, const __grid_constant__ EncTable tab) {
    extern __shared__ __align__(16) unsigned char smem[];
    uint2* lut = reinterpret_cast<uint2*>(smem);                       // [byte][lane & 15]: {code << (32 - len), len}
    uint8_t* ring = smem + (size_t)256 * kLutRep * 8;                  // kRing input steps
    uint32_t* img_all = reinterpret_cast<uint32_t*>(ring + (size_t)kRing * kStepBytes);
    uint32_t* recs = img_all + kEncWarps * kImgWords;                  // gap records, by segment
    __shared__ EncShared sh;

    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t lane8 = (lane & (kLutRep - 1)) * 8;
    uint32_t* const img = img_all + warp * kImgWords;                  // this warp's output words
    auto load_lut = [&](const EncTable& t) {
        for (int i = tid; i < 256 * kLutRep / 2; i += kEncThreads) {  // two copies a store
            uint32_t c, l;
            code_of(t.e[i / (kLutRep / 2)], c, l);
            reinterpret_cast<uint4*>(lut)[i] = make_uint4(c, l, c, l);
        }
    };
    // warp 0: region `item` of the plan to reg[slot], and a job's codes to next_codes, asynchronously
    const uint64_t nitems = *a.nitems_dev;
    // the plan is made: its records are zero again when a prepared call follows (st_rec, hgap_internal.h)
    if (!a.jobs) {
        const uint64_t stride = (uint64_t)gridDim.x * kEncThreads;
        for (uint64_t g = (uint64_t)blockIdx.x * kEncThreads + tid; g * kPlanWarps < nitems; g += stride) a.st_rec[g] = 0;
    }
    auto fetch_region = [&](uint32_t slot, uint64_t item) {
        EncRegion* const to = &sh.reg[slot];
        if (item < nitems) {
            if (lane < sizeof(EncRegion) / 16)
                cp_async16(reinterpret_cast<uint4*>(to) + lane, reinterpret_cast<const uint4*>(a.plan + item) + lane);
        } else if (lane == 0) {
            to->hi = 0;
        }
        cp_async_commit();
    };
    auto fetch_codes = [&](uint32_t job) {
        const uint4* const from = reinterpret_cast<const uint4*>(a.tables + job);
        uint4* const to = reinterpret_cast<uint4*>(&sh.next_codes);
        for (uint32_t i = lane; i < sizeof(EncTable) / 16; i += 32) cp_async16(to + i, from + i);
        cp_async_commit();
    };
    if (!a.jobs) load_lut(tab);
    if (tid == 0) {
        sh.lut_job = a.jobs ? ~0u : 0u;
        sh.p_issued = 0;
        sh.p_step = 0;
        sh.p_which = 0;
        for (int s = 0; s < kRing; ++s) mbar_init(&sh.mbar[s], 1);
        mbar_init_fence();
    }
    if (warp == 0) {
        // the CTA's first region is the one of its number, the later ones are claimed
        uint32_t item = 0;
        if (lane == 0) item = atomicAdd(a.counter, 1u);
        fetch_region(0, blockIdx.x);
        item = __shfl_sync(kFull, item, 0);
        fetch_region(1, (uint64_t)gridDim.x + item);
        cp_async_wait_all();
        __syncwarp();
        if (a.jobs && sh.reg[0].hi) fetch_codes(sh.reg[0].job);
        if (lane == 0) produce(ring, sh, 0, &sh.reg[0], &sh.reg[1]);
        cp_async_wait_all();
    }
    __syncthreads();

    uint32_t cons = 0;  // steps consumed so far (the ring's sequence number)
    for (uint32_t slot = 0;; slot = slot == 2 ? 0 : slot + 1) {
        const EncRegion& R = sh.reg[slot];
        if (R.hi == 0) break;
        const EncRegion* const next = &sh.reg[slot == 2 ? 0 : slot + 1];
        // batched: the job's codes into the table (the previous region is done with it)
        if (a.jobs && R.job != sh.lut_job) load_lut(sh.next_codes);
        if (warp == 0) {
            if (lane == 0) sh.tail[(cons * kEncWarps) % (4 * kEncWarps)] = R.tail;
            cp_async_wait_all();  // the next region
        }
        __syncthreads();
        // warp 0: the next region's codes, if they are others, and the claim of the region after it
        uint32_t claim = 0;
        if (warp == 0 && next->hi) {
            if (a.jobs && next->job != R.job) fetch_codes(next->job);
            if (lane == 0) claim = atomicAdd(a.counter, 1u);
        }
        if (tid == 0) sh.lut_job = R.job;
        uint32_t P = R.first_bit;      // first bit of the step
        uint32_t gnext = 0;            // next gap word to write
        bool overflow = false;

        // Gap word g from the records of the region's segments before k_end; `bytes` of it: all
        // four, or, where the region ends inside it, those whose two entries are known.  A region's
        // first byte takes its even entry from gap_head; bytes before that belong to the previous
        // region (the job's first region writes them: entries of no segment are 0).
        auto emit_gap = [&](uint32_t g, uint32_t k_end, uint32_t bytes) {
            const uint4* r4 = reinterpret_cast<const uint4*>(recs + ((8 * g) & (kRecs - 1)));
            const uint4 r0 = r4[0], r1 = r4[1];
            const uint32_t rr[8] = {r0.x, r0.y, r0.z, r0.w, r1.x, r1.y, r1.z, r1.w};
            const uint32_t lo = g == 0 ? R.first_bit >> 7 : 0u;  // first segment that ends in the region
            const uint32_t hi = k_end - 8 * g < 8 ? k_end - 8 * g : 8u;
            uint32_t v = 0;
#pragma unroll
            for (uint32_t i = 0; i < 8; ++i) {
                // the first byte with its top bit set: 0x80 + the spill of the code that reached the end
                const uint32_t s = (__ffs(rr[i] & 0x80808080u) - 8) & 31;
                v |= ((rr[i] >> s) & 0xfu) << (4 * i);
            }
            v &= (hi == 8 ? ~0u : (1u << (4 * hi)) - 1u) & (~0u << (4 * lo));
            if (lo & 1u) v |= R.gap_head << (4 * (lo - 1));
            const uint32_t b0 = R.flags & kRegionFirst ? 0u : lo >> 1;
            if (g >= R.ngaps) {
                overflow = true;
            } else if (b0 == 0 && bytes == 4) {
                R.gaps[g] = v;
            } else {
                uint8_t* const out = reinterpret_cast<uint8_t*>(R.gaps + g);
#pragma unroll 1
                for (uint32_t b = b0; b < bytes; ++b) out[b] = (uint8_t)(v >> (8 * b));
            }
        };

        // ---- stream the steps ---------------------------------------------------
        uint32_t off = warp * (uint32_t)kWarpBytes;              // the warp's first byte in the region
        for (const uint32_t nsteps_end = cons + (R.hi + kStepBytes - 1) / kStepBytes; cons != nsteps_end;
             ++cons, off += kStepBytes) {
            const uint32_t stage = cons % kRing, par = cons & 1;
            mbar_wait(&sh.mbar[stage], (cons / kRing) & 1, a.status, true);
            const bool have = off < R.hi;  // the warp's 1 KiB is in the region (whole, unless the job ends in it)
            // an end of the job in it: bytes before and after the job's are encoded too (the ring holds
            // something there), but count for nothing and are not written out
            const bool edge = off < R.lo || ((R.flags & kRegionLast) && off + kWarpBytes >= R.hi);
            Pieces pc;
            uint32_t nbits = 0;
            if (have) {
                const uint4* src = reinterpret_cast<const uint4*>(ring + stage * (uint32_t)kStepBytes + tid * kLaneBytes);
                const uint4 q0 = src[0], q1 = src[1];
                const uint32_t w[kPieces] = {q0.x, q0.y, q0.z, q0.w, q1.x, q1.y, q1.z, q1.w};
                const char* const l8 = reinterpret_cast<const char*>(lut);
#pragma unroll
                for (int j = 0; j < kPieces; ++j) {
                    make_piece(l8, lane8, w[j], pc.hi[j], pc.lo[j], pc.q[j]);
                    nbits += piece_bits(pc.q[j]);
                }
                if (edge) {
                    const uint32_t o = off + lane * (uint32_t)kLaneBytes;
                    const uint32_t b1 = o >= R.hi ? 0u : R.hi - o < 32u ? R.hi - o : 32u;
                    nbits = b1 ? bits_before(pc, b1) - (o < R.lo ? bits_before(pc, R.lo - o) : 0u) : 0u;
                }
            }
            const uint32_t incl = warp_incl_scan(nbits, lane);
            if (lane == 31) {
                sh.tot[par][warp] = incl;
                if (have) sh.tail[(cons * kEncWarps + warp + 1) % (4 * kEncWarps)] = last_bits(pc);
            }
            __syncthreads();  // counts and tails visible; this ring buffer read; the previous step's records complete
            // the last warp refills the ring
            if (tid == kEncThreads - 32) {
                fence_proxy_async_smem();
                produce(ring, sh, cons + 1, &R, next);
            }
            const uint32_t t = lane < (uint32_t)kEncWarps ? sh.tot[par][lane] : 0u;
            const uint32_t L = __reduce_add_sync(kFull, t);
            const uint32_t before = __reduce_add_sync(kFull, lane < warp ? t : 0u);

            // Gap words of the steps before this one, once there are enough to occupy half the warps
            // (a warp's 32 words take it as long as a fifth of a step, and every warp waits for it at
            // the next barrier), or before this step's records would reach them.
            const uint32_t gend = P >> 10;
            const bool wrap = ((P + L) >> 7) - 8 * gnext >= kRecs - 8;  // (8: segments of bytes after the job's)
            if (wrap || gend - gnext >= kEncThreads / 2) {  // uniform
#pragma unroll 1
                for (uint32_t g = gnext + (kEncThreads - 1 - tid); g < gend; g += kEncThreads) emit_gap(g, P >> 7, 4);
                gnext = gend;
                if (wrap) __syncthreads();
            }

            if (have) {
                const uint32_t Pw = P + before;
                uint32_t gw = (Pw >> 7) * 4 - kSlackBits / 32;       // output word of image word 0
                uint32_t p1 = (Pw & 127u) + kSlackBits + incl;       // image bit of the lane's end
                uint32_t p = p1 - nbits;
                // lane 0: what the warp's first word already holds
                const uint32_t before32 = sh.tail[(cons * kEncWarps + warp) % (4 * kEncWarps)];
                uint32_t cur = lane == 0 ? __funnelshift_r(0u, before32, p) : 0u;
                // more bits than the image holds: the warp's two halves one after the other
                const uint32_t pe = __shfl_sync(kFull, p1, 31);
                const bool split = (pe + (edge ? kLaneMaxBits : 0u)) >> 5 >= (uint32_t)kImgWords;
                for (uint32_t half = 0;; half = 1) {
                    const uint32_t pa = __shfl_sync(kFull, p, 16 * half);              // first and end bit
                    const uint32_t pz = __shfl_sync(kFull, p1, split && !half ? 15 : 31);
                    const bool act = split ? (lane >> 4) == half : true;
                    const bool ends = (R.flags & kRegionLast) && off + kWarpBytes >= R.hi && (half || !split);  // the job's end
                    if (edge) {
                        const uint32_t o = off + lane * (uint32_t)kLaneBytes;
                        if (o < R.lo) p -= bits_before(pc, R.lo - o);
                        // words that no lane may complete
                        if (act && nbits) img[(p + bits_before(pc, 32)) >> 5] = 0;
                        if (half && lane == 16 && !nbits) img[p >> 5] = cur;
                        __syncwarp();
                    }
                    const bool packs = act && (nbits || !edge);
                    if (packs) cur = pack(pc, img, reinterpret_cast<char*>(recs), gw - 4, p, cur);
                    __syncwarp();
                    // a lane's unfinished word: the next lane stored that word's other bits
                    if (packs) atomicOr(img + (p >> 5), cur);
                    __syncwarp();
                    // words to write: [j0, j1), the last one unfinished only where the job ends
                    const uint32_t j0 = pa >> 5;
                    uint32_t j1 = ends ? (pz + 31) >> 5 : pz >> 5;
                    if (edge) {
                        // (the job starts in the first half: the second one's first word holds the first's last bits)
                        if (lane == 0 && !half && off < R.lo) img[j0] &= ~0u >> (pa & 31);
                        if (lane == 31 && ends && (pz & 31)) img[pz >> 5] &= ~(~0u >> (pz & 31));
                        __syncwarp();
                    }
                    uint32_t* const bits = R.bits + (int32_t)gw;
                    if (gw + j1 > R.nwords) {
                        overflow = true;
                        j1 = R.nwords > gw ? R.nwords - gw : 0u;
                    }
                    if (R.flags & kRegionVec) {
                        // whole 16-byte groups, then the words before and after them
                        const uint32_t g0 = (j0 + 3) & ~3u, g1 = j1 & ~3u;
#pragma unroll 1
                        for (uint32_t j = g0 + 4 * lane; j < g1; j += 128)
                            *reinterpret_cast<uint4*>(bits + j) = *reinterpret_cast<const uint4*>(img + j);
                        const uint32_t jw = (lane < 4 ? j0 & ~3u : g1 - 4) + lane;
                        if (jw < j1 && (lane < 4 ? jw >= j0 && jw < g0 : lane < 8 && jw >= g0)) bits[jw] = img[jw];
                    } else {
#pragma unroll 1
                        for (uint32_t j = j0 + lane; j < j1; j += 32) bits[j] = img[j];
                    }
                    if (!split || half) break;
                    // the second half's image starts at the segment of its first bit
                    const uint32_t by = (__shfl_sync(kFull, p, 16) & ~127u) - kSlackBits;
                    cur = __shfl_sync(kFull, cur, 15);
                    if (lane != 16) cur = 0;
                    p -= by;
                    p1 -= by;
                    gw += by >> 5;
                    __syncwarp();
                }
            }
            P += L;
        }
        if (warp == 0) {
            cp_async_wait_all();  // the next region's codes
            // the region after the next into the slot that the last barrier freed
            claim = __shfl_sync(kFull, claim, 0);
            if (next->hi) fetch_region(slot == 0 ? 2 : slot - 1, (uint64_t)gridDim.x + claim);
            else if (lane == 0) sh.reg[slot == 0 ? 2 : slot - 1].hi = 0;
        }
        __syncthreads();  // every record of the region visible

        // ---- end of the region --------------------------------------------------
        {
            const uint32_t k_end = P >> 7;
#pragma unroll 1
            for (uint32_t g = gnext + (kEncThreads - 1 - tid); g <= (k_end >> 3); g += kEncThreads) {
                uint32_t bytes = 4;
                if (g == (k_end >> 3)) bytes = !(R.flags & kRegionLast) ? (k_end & 7) >> 1 : g < R.ngaps ? 4u : 0u;  // the region ends in it
                if (bytes) emit_gap(g, k_end, bytes);
            }
        }
        if (overflow) atomicOr(a.status, kDevSize);
        if (tid == 0) {
            if (P - R.first_bit != R.nbits) atomicOr(a.status, kDevPlan);  // histograms were not this input's
            // the producer's cursor follows its region, which becomes the current one
            if (sh.p_which == 1) sh.p_which = 0;
            else sh.p_step = 0;
            fence_proxy_async_smem();
            produce(ring, sh, cons, next, nullptr);
        }
    }

    // every copy issued has been consumed, unless a wait gave up: never leave
    // the CTA with a copy still in flight into its shared memory
    if (tid == 0) {
        const uint32_t issued = sh.p_issued;
        const uint32_t first = issued > (uint32_t)kRing ? issued - kRing : 0u;
        for (uint32_t i = first; i < issued; ++i)
            mbar_wait(&sh.mbar[i % kRing], (i / kRing) & 1, a.status, false);
    }
}

// ------------------------------------------------------------- launchers ---

int launch_encode(const EncArgs& a, const EncTable& t, int ctas_per_sm, void* stream) {
    static LaunchCache cache, plan_cache;
    const LaunchFacts f = cache.get(reinterpret_cast<const void*>(encode_kernel), kEncThreads, kEncSmem);
    if (f.err != cudaSuccess) return f.err;
    const LaunchFacts pf = plan_cache.get(reinterpret_cast<const void*>(enc_plan_kernel), kPlanThreads, 0);
    if (pf.err != cudaSuccess) return pf.err;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    // as many plan warps as there are regions, at most what the GPU holds at once
    const uint64_t regions = a.nitems ? a.nitems : 1;
    const uint64_t plan_want = (regions + kPlanWarps - 1) / kPlanWarps;
    const uint64_t plan_cap = (uint64_t)pf.sms * pf.per_sm;
    enc_plan_kernel<<<(unsigned)(plan_want < plan_cap ? plan_want : plan_cap), kPlanThreads, 0, st>>>(a, t);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    const int k = (ctas_per_sm > 0 && ctas_per_sm < f.per_sm) ? ctas_per_sm : f.per_sm;
    const uint64_t cap = (uint64_t)f.sms * k;
    encode_kernel<<<(unsigned)(regions < cap ? regions : cap), kEncThreads, kEncSmem, st>>>(a, t);
    return cudaGetLastError();
}

}  // namespace hgap
