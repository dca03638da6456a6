// Triangle ("fancy") chroma upsampling and the 16.16 fixed-point YCbCr -> RGB transform of libjpeg, eight or
// four pixels at a time in packed arithmetic.  A pixel is a word: red in its low byte, then green, blue.
#pragma once
#include "types.h"

namespace ffcvb {

// Bytes of (a, b) by the nibbles of `sel`; a nibble's top bit replicates the byte's sign instead.
__device__ __forceinline__ uint32_t pick(uint32_t a, uint32_t b, uint32_t sel) {
    uint32_t r;
    asm("prmt.b32 %0, %1, %2, %3;" : "=r"(r) : "r"(a), "r"(b), "r"(sel));
    return r;
}

// One pixel.  lum: luma << 16 | 32768, cb and cr: chroma - 128.  What lies above bit 16 is the value, so it is
// clamped in place and its byte picked.
__device__ __forceinline__ uint32_t ycc_pixel(int lum, int cb, int cr) {
    const int r = __vimin_s32_relu(91881 * cr + lum, 0xffffff);
    const int g = __vimin_s32_relu(-22554 * cb + (-46802 * cr + lum), 0xffffff);
    const int b = __vimin_s32_relu(116130 * cb + lum, 0xffffff);
    return pick(pick((uint32_t)r, (uint32_t)g, 0x0062), (uint32_t)b, 0x6610);
}
__device__ __forceinline__ int luma_fixed(uint32_t word, int k) { return (int)pick(word, 0x8000u, 0x6054u | (uint32_t)k << 8); }

// Planes of a 4:2:0 image: pitches, and the real size of the chroma planes.
struct QuadPlanes {
    const uint8_t *y, *cb, *cr;
    int yw, cw, real_w, real_h;
};

// The 8 x 2 pixels of the chroma samples cx .. cx + 3 (cx a multiple of 4, below real_w) of row cy.  The filter
// reads a 3 x 6 neighbourhood (image edges replicate, which is what its edge formulas amount to): vertical blends
// once per column, two samples per register, then the horizontal ones.  21 instructions per pixel; one thread
// per two chroma samples in plain integers took 37.
__device__ __forceinline__ void quad_pixels(const QuadPlanes &p, int cx, int cy, uint32_t (&px)[2][8]) {
    const int xl = max(cx - 1, 0), xr = min(cx + 4, p.real_w - 1), last = p.real_w - 1 - cx;
    const uint32_t edge = last >= 3 ? 0x3210u : (last == 2 ? 0x2210u : (last == 1 ? 0x1110u : 0x0000u));
    const size_t rows[3] = {(size_t)max(cy - 1, 0) * p.cw, (size_t)cy * p.cw, (size_t)min(cy + 1, p.real_h - 1) * p.cw};
    uint32_t val[2][2][4]; // [Cb, Cr][row][samples 0|1 even, odd, 2|3 even, odd], minus 128 as signed bytes 0 and 2
#pragma unroll
    for (int k = 0; k < 2; k++) {
        const uint8_t *plane = k == 0 ? p.cb : p.cr;
        uint32_t s01[3], s23[3], ends[3];
#pragma unroll
        for (int r = 0; r < 3; r++) {
            const uint8_t *row = plane + rows[r];
            const uint32_t w = pick(*reinterpret_cast<const uint32_t *>(row + cx), 0, edge);
            ends[r] = (uint32_t)row[xl] | (uint32_t)row[xr] << 16;
            s01[r] = pick(w, 0, 0x4140);
            s23[r] = pick(w, 0, 0x4342);
        }
#pragma unroll
        for (int r = 0; r < 2; r++) {
            const uint32_t a = 3 * s01[1] + s01[2 * r], b = 3 * s23[1] + s23[2 * r], e = 3 * ends[1] + ends[2 * r];
            const uint32_t left = pick(e, a, 0x5410), mid = pick(a, b, 0x5432), right = pick(b, e, 0x7632);
            auto blend = [](uint32_t v, uint32_t beside, uint32_t round) {
                return ((3 * v + beside + round) >> 4 & 0x00ff00ffu) ^ 0x00800080u;
            };
            val[k][r][0] = blend(a, left, 0x00080008u);
            val[k][r][1] = blend(a, mid, 0x00070007u);
            val[k][r][2] = blend(b, mid, 0x00080008u);
            val[k][r][3] = blend(b, right, 0x00070007u);
        }
    }
#pragma unroll
    for (int r = 0; r < 2; r++) {
        const uint2 lum = *reinterpret_cast<const uint2 *>(p.y + (size_t)(2 * cy + r) * p.yw + 2 * cx);
#pragma unroll
        for (int q = 0; q < 8; q++) {
            const int v = (q >> 2) * 2 + (q & 1); // pixel q belongs to sample q / 2
            const uint32_t lane = (q & 2) ? 0xaaa2 : 0x8880;
            px[r][q] = ycc_pixel(luma_fixed(q < 4 ? lum.x : lum.y, q & 3), (int)pick(val[0][r][v], 0, lane), (int)pick(val[1][r][v], 0, lane));
        }
    }
}

// Four pixels of planes of one resolution, whose samples begin at offset s; `words`: the three addresses are
// multiples of 4, else `count` of them are fetched one by one.
__device__ __forceinline__ void plain_pixels(const uint8_t *y, const uint8_t *cb, const uint8_t *cr, size_t s, int count, bool words, uint32_t (&px)[4]) {
    uint32_t l = 0, b = 0, r = 0;
    if (words) {
        l = *reinterpret_cast<const uint32_t *>(y + s);
        b = *reinterpret_cast<const uint32_t *>(cb + s);
        r = *reinterpret_cast<const uint32_t *>(cr + s);
    } else {
        for (int q = 0; q < count; q++) {
            l |= (uint32_t)y[s + q] << (8 * q);
            b |= (uint32_t)cb[s + q] << (8 * q);
            r |= (uint32_t)cr[s + q] << (8 * q);
        }
    }
    b ^= 0x80808080u;
    r ^= 0x80808080u;
#pragma unroll
    for (int q = 0; q < 4; q++) px[q] = ycc_pixel(luma_fixed(l, q), (int)pick(b, 0, 0x8880u + 0x1111u * q), (int)pick(r, 0, 0x8880u + 0x1111u * q));
}

} // namespace ffcvb
