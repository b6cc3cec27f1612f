// dec_entry.cuh -- the decoder's level-1 entries in the u32 form the decode
// kernel keeps in shared memory, made from the u16 table (DecTable).  Used by
// the decode kernel (single path: once per CTA) and by the batched path's
// per-buffer table build (bdec_table_kernel: once per buffer, copied per tile).
#pragma once

#include "hgap_internal.h"

namespace hgap {

// Entry forms.  Pointer: bit 31 | extra width << 16 | level-2 offset; invalid:
// bit 30.  Otherwise symbols from the low byte up, and
//   one or two symbols:   bits of the codes << 16 | number of symbols << 24 (e >> 16 is what the
//                         decoder's state, address << 8 | position, advances by);
//   up to three (multi):  bits of the codes << 24 | (number - 1) << 29.
constexpr uint32_t kEntPointer = 0x80000000u;
constexpr uint32_t kEntInvalidBit = 0x40000000u;
// (the lengths in it, 32 and 16 bits: a decoder that does not test the bit still ends its phase)
constexpr uint32_t kEntInvalid = kEntInvalidBit | 0x10200000u;

// The entry of one u16 table entry (level 1 or 2).
template <bool MULTI>
__device__ __forceinline__ uint32_t entry_single(uint32_t e) {
    if (e & 0x8000u) return kEntPointer | (((e >> 12) & 7u) << 16) | (e & 0xfffu);
    if (e & kDecInvalid) return kEntInvalid;
    const uint32_t len = ((e >> 8) & 15u) + 1u;
    return MULTI ? (len << 24) | (e & 0xffu) : 0x01000000u | (len << 16) | (e & 0xffu);
}

// The first code in the low bits of an 11-bit window x: its length, 0 if it is
// longer than the window or does not exist; its symbol in `sym`.
__device__ __forceinline__ uint32_t code_in_window(const uint16_t* t1src, uint32_t x, uint32_t& sym) {
    const uint32_t e = t1src[x & ((1u << kDecPrefix) - 1u)];
    sym = e & 0xffu;
    return e & (0x8000u | kDecInvalid) ? 0u : ((e >> 8) & 15u) + 1u;
}

// The entry of P-bit window x: when the first code leaves room for a whole
// second code inside the same window, both at once.  The second code is known
// from the bits after the first alone, because it ends inside the window.
template <uint32_t P>
__device__ __forceinline__ uint32_t entry_pair(const uint16_t* t1src, uint32_t x) {
    const uint32_t x11 = x << (kDecPrefix - P);
    uint32_t s1, s2;
    const uint32_t l1 = code_in_window(t1src, x11, s1);
    if (l1 == 0 || l1 >= P) return entry_single<false>(t1src[x11]);
    const uint32_t l2 = code_in_window(t1src, x11 << l1, s2);
    if (l2 == 0 || l1 + l2 > P) return entry_single<false>(t1src[x11]);
    return s1 | (s2 << 8) | ((l1 + l2) << 16) | 0x02000000u;
}

// The same with up to three codes (multi form; complete books).
template <uint32_t P>
__device__ __forceinline__ uint32_t entry_multi(const uint16_t* t1src, uint32_t x) {
    const uint32_t x11 = x << (kDecPrefix - P);
    uint32_t s1, s2, s3;
    const uint32_t l1 = code_in_window(t1src, x11, s1);
    if (l1 == 0 || l1 >= P) return entry_single<true>(t1src[x11]);
    const uint32_t l2 = code_in_window(t1src, x11 << l1, s2);
    if (l2 == 0 || l1 + l2 > P) return entry_single<true>(t1src[x11]);
    const uint32_t l12 = l1 + l2;
    const uint32_t two = s1 | (s2 << 8) | (l12 << 24) | (1u << 29);
    if (l12 >= P) return two;
    const uint32_t l3 = code_in_window(t1src, x11 << l12, s3);
    if (l3 == 0 || l12 + l3 > P) return two;
    return s1 | (s2 << 8) | (s3 << 16) | ((l12 + l3) << 24) | (2u << 29);
}

}  // namespace hgap
