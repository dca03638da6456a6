// Device-side look-up of Huffman codes that the first level of a table does not resolve.
#pragma once
#include "types.h"

namespace ffcvb {

// An invalid code acts as 16 bits that end the block, so that speculative decoding always makes
// progress.
static __device__ __noinline__ uint32_t huff_by_length(const HuffTable *__restrict__ t, uint32_t w) {
    const int code = w >> 16;
#pragma unroll 1
    for (int l = kHuffBits + 1; l <= 16; l++) {
        const int c = code >> (16 - l);
        if (c <= t->maxcode[l]) return huff_entry(l, t->vals[(t->valoff[l] + c) & 255], t->is_dc != 0);
    }
    return huff_invalid(t->is_dc != 0);
}
// Entry of the code at the top of w, which the first level answered with e (kHuffLong set): second
// level, or, when a table has more long-code prefixes than sub-tables (never with the tables encoders
// emit), the code-length walk.
__device__ __forceinline__ uint32_t huff_long(const HuffTable *__restrict__ t, uint32_t e, uint32_t w) {
    if (e == 0xFFFFu) return huff_by_length(t, w);
    return t->sub[e & (kHuffSubTables - 1)][(w >> 16) & ((1 << (16 - kHuffBits)) - 1)];
}
// Value of a symbol of n bits, `size` (>= 1) of them magnitude bits, that begins at the top of w.
__device__ __forceinline__ int huff_value(uint32_t w, uint32_t n, uint32_t size) {
    const uint32_t bits = w << (n - size);
    return (int)(bits >> (32 - size)) + ((int)bits < 0 ? 0 : 1 - (1 << size));
}

} // namespace ffcvb
