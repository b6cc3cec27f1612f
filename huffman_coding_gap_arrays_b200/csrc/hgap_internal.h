// hgap_internal.h -- types shared by the host code and the sm_100a kernels.
#pragma once

#include <cstddef>
#include <cstdint>

#include "../../include/hgap.h"

#ifdef __CUDACC__
#define HGAP_HD __host__ __device__
#else
#define HGAP_HD
#endif

namespace hgap {

// ---------------------------------------------------------------- format ---
constexpr int kMaxLen = HGAP_MAX_CODE_LEN;  // encoder/include/constants.hpp:5
constexpr int kSegBits = HGAP_SEGMENT_BITS; // encoder/include/constants.hpp:12

// ------------------------------------------------------- device status bits -
// OR-ed into the workspace status word by the kernels; read back by
// hgap_workspace_status().  No kernel traps: every failure is a bit here.
enum : uint32_t {
    kDevTimeout = 1u,   // a bounded inter-tile wait gave up
    kDevCorrupt = 2u,   // decoder: invalid codeword / segment end != next gap
    kDevNoCode = 4u,    // encoder: an input byte has no codeword
    kDevSize = 8u,      // total bits / symbols disagree with W, S or n
    kDevPlan = 16u,     // encoder: workspace histograms are not this input's
};

// Look-back record: 2 flag bits over a 62-bit value (aggregate or inclusive
// prefix).  Zero = not yet published.
constexpr uint64_t kFlagA = 1ull << 62;
constexpr uint64_t kFlagP = 2ull << 62;
constexpr uint64_t kFlagMask = 3ull << 62;
constexpr uint64_t kValueMask = ~kFlagMask;

// Bounded-wait test hook, all zero in every product call: the work item
// (encoder region / decoder tile, in the launch's numbering) plus one whose
// look-back records are never published, and the limit of every look-back
// wait in ns (0: the default, kWaitLimitNs).
struct LookbackHook {
    uint64_t hold_plus1;
    uint64_t wait_ns;
};

// Workspace header (both kernels): status word, tile counter, padding.
constexpr size_t kWsHeader = 256;

// ---------------------------------------------------------------- encoder ---
// Per byte value: code in bits 0..15, length in bits 16..20; an absent byte
// is 0x80000000 (length field 0, and 0x8000 when summed as e >> 16 so that a
// thread's bit count reveals it without a per-byte test).
struct EncTable {
    uint32_t e[256];
};
constexpr uint32_t kEncAbsent = 0x80000000u;

// The encoder works on super-tiles: `st_chunks` chunks of kEncChunkBytes input
// bytes each.  The histogram pass that precedes it also records one 256-bin
// histogram per super-tile, so a super-tile's bit count -- and, after one
// look-back (enc_plan_kernel), its first output bit -- is known before any of
// its bytes are encoded.  st_chunks depends on n only (hgap_internal
// encode_st_chunks), so both passes and the workspace query agree.
constexpr int kEncChunkBytes = 8192;
constexpr int kEncMaxStChunks = 32;
// The super-tile size minimises the encoder's modelled makespan: persistent CTAs
// (2 per SM, 296 on a 148-SM B200) take equal super-tiles of c chunks in waves,
// each costing c chunks plus about one chunk's worth of fixed work (a last step
// partly empty, its gap words, two more barriers).  Measured on 16 MiB (2048
// chunks), encoder and histogram pass: 1-chunk super-tiles (7 waves) 0.070 ms, 2
// chunks 0.055, 4 chunks 0.047, 7 chunks (one wave) 0.041 ms; with the regions
// planned by a kernel of their own, sizes of 4 to 24 chunks still found none
// better.  The count is kept under encode_super_tiles_cap, so a workspace sized
// for n bytes serves every smaller input.
constexpr uint64_t kEncCtas = 296;
constexpr uint64_t kEncStOverhead = 1;  // chunks

// Encoder workspace for nst super-tiles:
//   [status u32][counter u32][super-tiles to encode u64][plan counter u32, 12 bytes of padding]
//                                                         cleared by every call
//   [tag: n u64, input u64][st_rec u64 x nst][scratch histogram u32 x 256]
//                                                         these by the histogram pass, and st_rec by
//                                                         the encoder again, for the next prepared call
//   [plan EncRegion x nst][st_hist u32 x 256 x nst]
// The tag's place depends on no input: a histogram pass over any other one writes over it.
constexpr size_t kEncWsTag = 32;
struct EncWorkspace {
    size_t st_rec, scratch, plan, st_hist, bytes;
};
inline uint64_t encode_chunks(uint64_t n) { return (n + 15 + kEncChunkBytes - 1) / kEncChunkBytes; }
// An upper bound of the super-tile count of every input of up to n bytes (at any
// alignment), non-decreasing in n: what a workspace for inputs of up to n bytes holds.
inline uint64_t encode_super_tiles_cap(uint64_t n) {
    const uint64_t ch = encode_chunks(n);
    const uint64_t a = ch < 2 * kEncCtas ? ch : 2 * kEncCtas;
    const uint64_t b = (ch + 15) / 16;
    return a > b ? a : b;
}
inline uint64_t encode_st_chunks(uint64_t n) {
    const uint64_t chunks = encode_chunks(n), cap = encode_super_tiles_cap(n);
    uint64_t best = kEncMaxStChunks, best_cost = ~0ull;
    for (uint64_t c = 1; c <= (uint64_t)kEncMaxStChunks; ++c) {
        const uint64_t tiles = (chunks + c - 1) / c;
        if (tiles > cap) continue;  // within the workspace bound (c = 32 always is)
        const uint64_t cost = (tiles + kEncCtas - 1) / kEncCtas * (c + kEncStOverhead);
        if (cost < best_cost) {  // ties keep the smaller super-tile (finer balance)
            best = c;
            best_cost = cost;
        }
    }
    return best;
}
inline uint64_t encode_super_tiles(uint64_t lo_plus_n, uint64_t n) {
    const uint64_t st = encode_st_chunks(n) * kEncChunkBytes;
    return (lo_plus_n + st - 1) / st;
}

// One buffer to encode.  The single-buffer entry points pass one job by value;
// the batched ones keep an array of them in the workspace.  Regions (units of
// st_bytes input bytes) are numbered globally over the jobs of a launch: job
// j owns regions [item0, item0 + nst).
// 16-byte aligned (and a multiple of 16 bytes): the one-CTA setup kernels write
// whole jobs with vector stores
struct alignas(16) EncJob {
    const uint8_t* in_aligned;  // input rounded down to 16 bytes
    uint64_t lo;                // virtual index of the first input byte (in & 15)
    uint64_t hi;                // lo + n
    uint32_t* bits;
    uint64_t words;
    uint32_t* gaps;
    uint64_t gap_words;
    uint64_t segments;
    uint64_t item0;             // global index of the job's first region
    uint64_t nst;               // its regions
    uint32_t st_bytes;          // region size in input bytes (a multiple of kEncChunkBytes)
    uint32_t bits_aligned16;    // bits is 16-byte aligned: vector stores allowed
    uint64_t bit0;              // stream bit of the job's first code: 0, unless the job is one
                                // part of a stream split across devices (bits / gaps then
                                // address stream word / gap word 0 of a window)
};
static_assert(sizeof(EncJob) == 96, "EncJob: six 16-byte groups");

// One region as the encoder takes it, made by enc_plan_kernel once the code
// lengths are known: all that a CTA needs to start on it without another
// dependent load.  Output words and bit positions count from the gap word (1024
// bits, so also the 16-byte group of output words) that holds the region's first
// bit.
struct alignas(16) EncRegion {
    const uint8_t* in;          // its bytes are [lo, hi) from here (16-byte aligned)
    uint32_t* bits;             // output and gap words,
    uint32_t* gaps;
    uint32_t nwords, ngaps;     // and how many of them exist
    uint32_t lo, hi;            // hi = 0: no region
    uint32_t first_bit;         // the region's first bit
    uint32_t nbits;             // and bit count
    uint32_t tail;              // the code bits before it in its first word, right-aligned
    uint32_t gap_head;          // spill at the segment end at or before it, if its first gap entry is an odd one
    uint32_t job;
    uint32_t flags;             // kRegion...
    uint32_t pad[2];
};
static_assert(sizeof(EncRegion) == 80, "EncRegion: five 16-byte groups");
constexpr uint32_t kRegionFirst = 1u;  // of its job
constexpr uint32_t kRegionLast = 2u;
constexpr uint32_t kRegionVec = 4u;    // output words are 16-byte aligned

inline EncWorkspace encode_workspace(uint64_t nst) {
    EncWorkspace w;
    w.st_rec = kEncWsTag + 16;
    w.scratch = (w.st_rec + 8 * (size_t)nst + 15) & ~(size_t)15;
    w.plan = w.scratch + 1024;
    w.st_hist = w.plan + sizeof(EncRegion) * (size_t)nst;
    w.bytes = w.st_hist + 1024 * (size_t)nst;
    return w;
}

struct EncArgs {
    EncJob single;              // the job, when jobs == nullptr
    const EncJob* jobs;         // batched: [count]
    const uint64_t* item0s;     // batched: [count + 1], item0 of each job and the total
    const EncTable* tables;     // batched: [count]
    uint32_t count;             // jobs (1 for the single-buffer path)
    uint64_t nitems;            // regions over all jobs (batched: an upper bound)
    uint64_t* nitems_dev;       // the region count in device memory; single path: written by the plan (0: not this input's)
    EncRegion* plan;            // [nitems]
    uint64_t* st_rec;           // [nitems] look-back records over regions
    const uint32_t* st_hist;    // [nitems][256] per-region histograms
    const uint64_t* tag;        // single path: {n, input address} written by the histogram pass
    uint32_t* counter;          // regions claimed by the encoder
    uint32_t* plan_counter;     // groups of regions claimed by the plan
    uint32_t* status;
    LookbackHook hook;
};

// A batched region as the histogram pass takes it: its bytes are [lo, hi) from `in`.
struct alignas(16) HistRegion {
    const uint8_t* in;  // 16-byte aligned
    uint32_t lo, hi;
    uint32_t job;
    uint32_t pad[3];
};
static_assert(sizeof(HistRegion) == 32, "HistRegion: two 16-byte groups");

struct HistStArgs {
    EncJob single;              // the job, when regions == nullptr
    uint64_t nitems;
    const uint64_t* nitems_dev; // batched: the region count in device memory (overrides nitems)
    uint32_t* hist;             // [count][256] histograms (zeroed before the launch)
    uint32_t* st_hist;          // [nitems][256]
    uint64_t* tag;              // single path: receives {n, input address}
    uint32_t* counter;          // batched: zeroed region counter (regions claimed one at a time)
    const HistRegion* regions;  // batched: [nitems]
};

// ---------------------------------------------------------------- decoder ---
// Two-level table.  Level 1 is indexed by the next kDecPrefix bits:
//   direct entry : bit15=0, bit14 = invalid, bits 8..11 = length-1, bits 0..7 = symbol
//   pointer entry: bit15=1, bits 12..14 = extra width w, bits 0..11 = level-2 offset
// Level 2 holds direct entries, 2^w per level-1 prefix whose codes are longer.
constexpr int kDecPrefix = 11;
// Decoder stage rows (of 4 symbols) for a book whose shortest code has
// min_len bits: a 128-bit segment holds at most ceil(128 / min_len) symbols.
HGAP_HD constexpr int dec_stage_rows(uint32_t min_len) {
    return min_len >= 4 ? 8 : min_len == 3 ? 11 : min_len == 2 ? 16 : 32;
}
// Segments per decoder tile for a stage of R rows: 512, for which the tile's
// fixed work (claim, look-back, barrier) counts least (256 MiB at 256 -> 512
// segments: mixed, R = 11, 546 -> 428 us; BF16 mantissa, R = 8, 576 -> 385); 256
// for 32 rows, whose 512-segment tile would leave one CTA per SM.
HGAP_HD constexpr int dec_tile_segs(int R) { return R >= 32 ? 256 : 512; }
// The same with a launch-shape override of 256 or 512 segments (0: the
// default; 32 rows keep 256), or what a batch takes for 16 rows by itself:
//   kDecTileBatch  480: 15 warps of one segment a lane and the extra one, three
//     CTAs and 48 warps an SM where 512 leaves two and 34 (batches of 10 to 80 MB
//     within 2 %, 291 MB 420 -> 413 us, 593 MB 766 -> 754, 256 buffers of 1 MiB of
//     Zipf(1.2) 410 -> 394).  Not for the single-buffer calls, whose every CTA
//     makes its own table: 256 MiB take the same time, 16 MiB 71 -> 79 us a call.
//     (8 and 11 rows are better off with two segments a lane: mixed 256 MiB
//     400 us, with 15 warps of one 444.)
//   kDecTileSmall  256, for small buffers, whose last tiles are mostly empty (4096
//     buffers of 4-64 KiB: that class 81 -> 67 us with 512 -> 256; 11 rows 58 -> 61
//     and 8 rows 12.7 -> 11.7, left alone).
constexpr uint32_t kDecTileBatch = ~0u, kDecTileSmall = ~1u;
HGAP_HD constexpr int dec_tile_segs_for(int R, uint32_t override_segs) {
    if (R >= 32) return 256;
    if (override_segs == kDecTileBatch) return R == 16 ? 480 : dec_tile_segs(R);
    if (override_segs == kDecTileSmall) return R == 16 ? 256 : dec_tile_segs(R);
    return override_segs == 256 ? 256 : dec_tile_segs(R);
}
constexpr int kDecT2Cap = 2560;  // >= the largest complete 16-bit book (see host.cpp)
constexpr uint16_t kDecInvalid = 0x4000;
struct alignas(16) DecTable {
    uint16_t t1[1 << kDecPrefix];
    uint16_t t2[kDecT2Cap];
};

// Multi entries (up to three symbols per level-1 lookup) pay for their wider
// stores and tail test only where codes are very short: complete books whose
// stage has at least this many rows (32: a shortest code of 1 bit).  Measured
// per 256 MiB: 2.2 bits/byte 0.518 -> 0.484 ms; from 16 rows on, Zipf(1.2)
// (shortest code 2 bits) 0.699 -> 0.722 ms.
constexpr int kDecMultiMinRows = 32;
HGAP_HD constexpr bool dec_multi(int rows, bool complete) { return complete && rows >= kDecMultiMinRows; }

// The decode kernel's table in shared memory.  A canonical code's long codes
// are the last in code order, so ONE table serves all lengths: a 32-bit window
// x at a code's start has the entry max(x >> (32 - P), (x >> shift) + offset) --
// below the first P-bit prefix with codes of more than P bits that prefix, from
// there on its first bits up to the book's longest length, counted on from that
// prefix (both lines meet there, and the second is the steeper one).  No second
// lookup, no branch.  P is 11, or 10 for the 32-row decoder, whose stage leaves
// room for three CTAs an SM only with a table this small (its books' codes are
// short: three fit 10 bits nearly as often; 1024 buffers of 4 KiB-4 MiB, that
// class's launch: 179 us with 11 bits and two CTAs, 150 us).  Of 1500 books of the batched
// workload's distributions 96 % (99.5 % of the bytes) fit dec_table_cap entries;
// the others ("wide") keep two levels: 2048 entries for 11 bits, and a level-2
// table in global memory for longer codes, reached by a branch.
HGAP_HD constexpr uint32_t dec_prefix(int rows) { return rows >= 32 ? 10u : (uint32_t)kDecPrefix; }
HGAP_HD constexpr uint32_t dec_table_cap(int rows) { return rows >= 32 ? 2176u : 2432u; }
struct DecIndex {
    uint32_t used;        // entries
    uint32_t shift;       // of x
    int32_t offset;
    uint32_t first_long;  // the first prefix with longer codes; kDecWide: two levels instead
};
constexpr uint32_t kDecWide = ~0u;
// From the first such prefix (2^P: none), the longest length, and whether the
// book is complete (an incomplete one is wide: its prefixes without a code have
// no place in one table).
HGAP_HD inline DecIndex dec_index(uint32_t first_long, uint32_t max_len, bool complete, int rows) {
    const uint32_t P = dec_prefix(rows), n1 = 1u << P;
    DecIndex d;
    const uint32_t extra = max_len > P && first_long < n1 ? max_len - P : 0u;
    const uint32_t used = extra ? first_long + ((n1 - first_long) << extra) : n1;
    const bool wide = !complete || used > dec_table_cap(rows);
    d.used = wide ? 1u << kDecPrefix : (used + 3) & ~3u;
    d.shift = wide ? 32 - kDecPrefix : 32 - P - extra;
    d.offset = wide || !extra ? 0 : (int32_t)first_long - (int32_t)(first_long << extra);
    d.first_long = wide ? kDecWide : first_long;
    return d;
}

// The same table in global memory, built once per buffer on the batched path
// so that a CTA moving to another buffer's tile gets it (symlen and the used
// entries) with one bulk copy.  A wide book's level-2 table is read from here.
struct alignas(16) DecTableW {
    DecIndex index;
    uint8_t symlen[256];  // each symbol's code length
    uint32_t t1[(1 << kDecPrefix) + kDecT2Cap / 2];
    HGAP_HD uint16_t* t2() { return reinterpret_cast<uint16_t*>(t1 + (1 << kDecPrefix)); }
    HGAP_HD const uint16_t* t2() const { return reinterpret_cast<const uint16_t*>(t1 + (1 << kDecPrefix)); }
};
static_assert((1 << kDecPrefix) + kDecT2Cap / 2 >= (int)dec_table_cap(8), "room for every table");
static_assert(sizeof(DecTableW) % 16 == 0, "16-byte copies");

// One stream to decode (same single / batched scheme as EncJob).  Its tiles
// use look-back records [item0, item0 + ntiles).
struct alignas(16) DecJob {
    const uint32_t* bits;
    uint64_t words;
    const uint32_t* gaps;
    uint64_t gap_words;
    uint64_t segments;
    uint8_t* out_aligned;  // output rounded down to 16 bytes
    uint64_t out_lo;       // out & 15
    uint64_t n;
    uint64_t item0;        // first look-back record of the job
    uint64_t ntiles;
};
static_assert(sizeof(DecJob) == 80, "DecJob: five 16-byte groups");

struct DecArgs {
    DecJob single;              // the job, when jobs == nullptr
    const DecJob* jobs;         // batched: [count]
    const uint32_t* job_of;     // batched: [nitems] job of each tile of this launch
    const uint64_t* item0s;     // batched: [count] first tile of each job in this launch's numbering
    const DecTableW* tables;    // batched: [count]
    DecIndex index;             // single path: the table's
    uint64_t nitems;            // tiles in this launch
    const uint64_t* nitems_dev; // batched: the tile count in device memory (overrides nitems)
    uint64_t* lookback;
    uint32_t* counter;
    uint32_t* status;
    LookbackHook hook;
};

// --------------------------------------------------------------- launchers --
// Implemented in the .cu files; return cudaError_t as int.
int launch_histogram(const void* d_in, uint64_t n, uint32_t* d_hist, void* stream);
// The plan, then the encoder.
int launch_encode(const EncArgs& a, const EncTable& t, int ctas_per_sm, void* stream);
int launch_hist_st(const HistStArgs& a, int ctas_per_sm, void* stream);
int launch_decode(const DecArgs& a, const DecTable& t, uint32_t min_len, bool complete, bool pairs,
                  int ctas_per_sm, uint32_t tile_segs, void* stream);
// Fraction of level-1 entries that decode two symbols (the decoder's pair
// rate under the code's own distribution, where every 11-bit prefix is
// equally likely).
double dec_pair_fraction(const hgap_codebook& cb);
// DecIndex of a book on the host.
DecIndex dec_index_of(const hgap_codebook& cb, bool complete, int rows);
// Tiles of a stream for a book whose shortest code is min_len bits (the
// decoder's tile size depends on it, and on a tile-size override, 0: none);
// min_len = 1 with 256-segment tiles gives the most.
uint64_t decode_tiles(uint64_t segments, uint32_t min_len, uint32_t tile_segs = 0);

// ------------------------------------------------------------- host helpers -
void make_enc_table(const hgap_codebook& cb, EncTable* t);
hgap_status make_dec_table(const hgap_codebook& cb, DecTable* t);

}  // namespace hgap
