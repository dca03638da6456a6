// AC symbol decode + dequantisation + fast integer inverse DCT + chroma upsampling + colour
// conversion (sm_100a).
//
// The arithmetic is the variant TurboJPEG selects for the reference's call
// (libffcv/libffcv.cpp:104-106, TJFLAG_FASTDCT without TJFLAG_FASTUPSAMPLE): the AAN fast integer
// IDCT evaluated in wrapping 16-bit lanes with 8-bit constants and truncating shifts, the 3:1
// triangle ("fancy") chroma upsampler, and the 16.16 fixed-point YCbCr->RGB transform.  These are
// integer butterflies in registers; they are not a dense contraction and must not be reordered,
// so no tensor cores.
#include "color.h"
#include "huffman.h"
#include "kernels.h"
#include "two.h"

namespace ffcvb {

// Natural position (row-major) of the coefficient at a place in zig-zag order.
__constant__ uint8_t c_natural[64] = {0, 1, 8, 16, 9, 2, 3, 10, 17, 24, 32, 25, 18, 11, 4, 5, 12, 19, 26, 33, 40, 48, 41, 34, 27, 20, 13, 6, 7, 14, 21, 28, 35, 42, 49, 56, 57, 50, 43, 36, 29, 22, 15, 23, 30, 37, 44, 51, 58, 59, 52, 45, 38, 31, 39, 46, 53, 60, 61, 54, 47, 55, 62, 63};

// Coefficient of natural position n out of a block's words, two per register.
__device__ __forceinline__ int coef_at(const int (&w)[32], int n) {
    return (n & 1) ? (w[n >> 1] >> 16) : (int)(short)(w[n >> 1] & 0xffff);
}

__device__ __forceinline__ int w16(int v) { return (int)(short)v; }
__device__ __forceinline__ int mul8(int v, int c) { return w16((v * c) >> 8); }

// One 8-point pass.  Inputs and outputs are sign-extended 16-bit lane values.
__device__ __forceinline__ void idct8(int &v0, int &v1, int &v2, int &v3, int &v4, int &v5, int &v6,
                                      int &v7) {
    int t10 = w16(v0 + v4), t11 = w16(v0 - v4);
    int t13 = w16(v2 + v6);
    int t12 = w16(mul8(w16(v2 - v6), 362) - t13);
    int t0 = w16(t10 + t13), t3 = w16(t10 - t13), t1 = w16(t11 + t12), t2 = w16(t11 - t12);
    int z13 = w16(v5 + v3), z10 = w16(v5 - v3), z11 = w16(v1 + v7), z12 = w16(v1 - v7);
    int t7 = w16(z11 + z13);
    int t11b = mul8(w16(z11 - z13), 362);
    int z5 = mul8(w16(z10 + z12), 473);
    int t10b = w16(mul8(z12, 277) - z5);
    int t12b = w16(mul8(z10, -669) + z5);
    int t6 = w16(t12b - t7);
    int t5 = w16(t11b - t6);
    int t4 = w16(t10b + t5);
    v0 = w16(t0 + t7);
    v7 = w16(t0 - t7);
    v1 = w16(t1 + t6);
    v6 = w16(t1 - t6);
    v2 = w16(t2 + t5);
    v5 = w16(t2 - t5);
    v4 = w16(t3 + t4);
    v3 = w16(t3 - t4);
}

// The full-size transform of a block in floating point, two columns or two rows per instruction.  It gives the
// wrapping 16-bit result because sums and differences may wrap anywhere as long as what is multiplied, and what is
// shifted in the end, lies in 16 bits: integers below 2^24 are exact in a float, and a product rounded down onto
// 1.5 * 2^23 is the shifted one.  `peak` gathers the largest of those values.  Up to kPeak the result is exact (the sum
// of z10 and z12 is then below 2^15 as well); beyond it, which the streams of encoders do not reach, the integer
// transform below has to be taken.  Kernel on 1024 photographs to 160x160, 256x256, 64 of 4:4:4 to 384x384: 110, 145 and
// 596 us in integers, 94, 124 and 500 this way, with the six CTAs per SM that its registers allow by themselves.
constexpr float kPeak = 16383.f;
constexpr float kOnes = 12582912.f; // 1.5 * 2^23: what is added to it leaves as an integer
__device__ __forceinline__ Two both(float v) { return Two(v, v); }
__device__ __forceinline__ void peak_of(Two v, float &peak) { peak = fmaxf(fmaxf(peak, fabsf(v.lo())), fabsf(v.hi())); }
__device__ __forceinline__ void idct8(Two &v0, Two &v1, Two &v2, Two &v3, Two &v4, Two &v5, Two &v6, Two &v7, float &peak) {
    const Two ones = both(kOnes);
    const Two t10 = add_rn(v0, v4), t11 = sub_rn(v0, v4), t13 = add_rn(v2, v6), d26 = sub_rn(v2, v6);
    const Two t12 = sub_rn(sub_rn(fma_rd(d26, both(362.f / 256), ones), ones), t13);
    const Two t0 = add_rn(t10, t13), t3 = sub_rn(t10, t13), t1 = add_rn(t11, t12), t2 = sub_rn(t11, t12);
    const Two z13 = add_rn(v5, v3), z10 = sub_rn(v5, v3), z11 = add_rn(v1, v7), z12 = sub_rn(v1, v7);
    const Two t7 = add_rn(z11, z13), d = sub_rn(z11, z13);
    const Two z5 = fma_rd(add_rn(z10, z12), both(473.f / 256), ones); // (on top of `ones`, as the two it is added to)
    const Two t10b = sub_rn(fma_rd(z12, both(277.f / 256), ones), z5);
    const Two t12b = add_rn(fma_rd(z10, both(-669.f / 256), both(-kOnes)), z5);
    const Two t6 = sub_rn(t12b, t7);
    const Two t5 = sub_rn(sub_rn(fma_rd(d, both(362.f / 256), ones), ones), t6);
    const Two t4 = add_rn(t10b, t5);
    peak_of(d26, peak);
    peak_of(z10, peak);
    peak_of(z12, peak);
    peak_of(d, peak);
    v0 = add_rn(t0, t7);
    v7 = sub_rn(t0, t7);
    v1 = add_rn(t1, t6);
    v6 = sub_rn(t1, t6);
    v2 = add_rn(t2, t5);
    v5 = sub_rn(t2, t5);
    v4 = add_rn(t3, t4);
    v3 = sub_rn(t3, t4);
}

// Smaller of two pairs of 16-bit values and `most`, not below 0.
__device__ __forceinline__ uint32_t clamp_halves(uint32_t v, uint32_t most) { return __vimin_s16x2_relu(v, most); }

// Block out of 32 words of coefficients (one per kBlockTile words at `coef`), each value on top of 2^15.
// Returns whether the result, which is stored in any case, is exact.
__device__ __forceinline__ bool block_in_floats(const uint32_t *coef, uint8_t *__restrict__ dst, int pitch) {
    float peak = 0.f;
    Two a[8][4]; // [row][pair of columns]
#pragma unroll
    for (int k = 0; k < 4; k++) {
#pragma unroll
        for (int r = 0; r < 8; r++) {
            const uint32_t w = coef[(4 * r + k) * kBlockTile]; // (each value becomes 2^23 + 2^15 + itself)
            a[r][k] = sub_rn(Two(__uint_as_float(pick(w, 0x4B000000u, 0x7410u)), __uint_as_float(pick(w, 0x4B000000u, 0x7432u))), both(8388608.f + 32768.f));
        }
        idct8(a[0][k], a[1][k], a[2][k], a[3][k], a[4][k], a[5][k], a[6][k], a[7][k], peak);
    }
#pragma unroll
    for (int q = 0; q < 4; q++) {
        Two b[8]; // a column of two rows
#pragma unroll
        for (int c = 0; c < 8; c++) b[c] = Two(a[2 * q][c >> 1].half(c & 1), a[2 * q + 1][c >> 1].half(c & 1));
        idct8(b[0], b[1], b[2], b[3], b[4], b[5], b[6], b[7], peak);
#pragma unroll
        for (int c = 0; c < 8; c++) {
            peak_of(b[c], peak);
            b[c] = fma_rd(b[c], both(1.f / 32), both(kOnes + 128.f)); // 16 bits of the sample, beyond its range as yet
        }
#pragma unroll
        for (int r = 0; r < 2; r++) {
            uint32_t w[4];
#pragma unroll
            for (int c = 0; c < 4; c++)
                w[c] = clamp_halves(pick(__float_as_uint(b[2 * c].half(r)), __float_as_uint(b[2 * c + 1].half(r)), 0x5410u), 0x00ff00ffu);
            *reinterpret_cast<uint2 *>(dst + (size_t)(2 * q + r) * pitch) = make_uint2(pick(w[0], w[1], 0x6420u), pick(w[2], w[3], 0x6420u));
        }
    }
    return peak <= kPeak;
}

// Reduced-size inverse transforms for decoding at 1/2, 1/4, 1/8 scale (the scale_num / scale_denom
// arguments of libffcv/libffcv.cpp:59,89-90): a block goes straight to N x N samples, N = 8 / R, each
// the mean of the R x R samples of the full transform it replaces.  Per dimension, in the scaling
// of the integer transforms, the sum of R neighbouring outputs is
//     S[m] = R a0 + sum_k a_k C(k, m),   C(k, m) = sqrt(2) sum_{j<R} cos((2 (R m + j) + 1) k pi / 16),
// evaluated as libjpeg-turbo does: constants round(|C| 2^13), 32-bit sums, plain quantiser steps,
// two extra fraction bits after the column pass, one rounding shift per pass that also divides by R.
template <int R>
__device__ __forceinline__ int reduced_constant(int k, int m) {
    // C(k, m) * 2^13 for R = 2 (k = 4 contributes nothing) and R = 4 (only odd k contribute)
    constexpr int c2[8][4] = {{0, 0, 0, 0},          {20995, 8697, -8697, -20995}, {15137, -15137, -15137, 15137},
                              {7373, -17799, 17799, -7373}, {0, 0, 0, 0},          {-4926, 11893, -11893, 4926},
                              {-6270, 6270, 6270, -6270},   {-4176, -1730, 1730, 4176}};
    constexpr int c4[8][2] = {{0, 0}, {29692, -29692}, {0, 0}, {-10426, 10426}, {0, 0}, {6967, -6967}, {0, 0}, {-5906, 5906}};
    return R == 2 ? c2[k][m & 3] : c4[k][m & 1];
}

template <int R>
__device__ __forceinline__ void reduced_block(const int (&cw)[32], const uint16_t *__restrict__ q,
                                              uint8_t *__restrict__ dst, int pitch) {
    constexpr int N = 8 / R, L = R == 2 ? 1 : 2;
    int a[8][8];
#pragma unroll
    for (int r = 0; r < 8; r++) {
        const int4 qw = reinterpret_cast<const int4 *>(q)[r];
        const int qq[4] = {qw.x, qw.y, qw.z, qw.w};
#pragma unroll
        for (int k = 0; k < 4; k++) {
            a[r][2 * k] = coef_at(cw, r * 8 + 2 * k) * (qq[k] & 0xffff);
            a[r][2 * k + 1] = coef_at(cw, r * 8 + 2 * k + 1) * (int)((uint32_t)qq[k] >> 16);
        }
    }
    int ws[8][N]; // [column of the block][row of the result]
#pragma unroll
    for (int col = 0; col < 8; col++)
#pragma unroll
        for (int m = 0; m < N; m++) {
            int acc = a[0][col] * (1 << (13 + L));
#pragma unroll
            for (int k = 1; k < 8; k++) acc += a[k][col] * reduced_constant<R>(k, m);
            ws[col][m] = (acc + (1 << (11 + L - 1))) >> (11 + L);
        }
#pragma unroll
    for (int row = 0; row < N; row++) {
        uint32_t packed = 0;
#pragma unroll
        for (int m = 0; m < N; m++) {
            int acc = ws[0][row] * (1 << (13 + L));
#pragma unroll
            for (int k = 1; k < 8; k++) acc += ws[k][row] * reduced_constant<R>(k, m);
            const int v = min(255, max(0, ((acc + (1 << (18 + L - 1))) >> (18 + L)) + 128));
            packed |= (uint32_t)v << (8 * m);
        }
        if (N == 4)
            *reinterpret_cast<uint32_t *>(dst + (size_t)row * pitch) = packed;
        else
            *reinterpret_cast<uint16_t *>(dst + (size_t)row * pitch) = (uint16_t)packed;
    }
}

constexpr uint32_t kCoefZero = 0x80008000u; // coefficients wait for the transform on top of 2^15

// One thread per block: decodes the block's AC symbols from the place the entropy decoder recorded,
// dequantising each value as it is stored (the block lies in shared memory, two coefficients per word,
// one bank per lane), then transforms it in registers.  Only blocks inside the crop's reach run.
// A warp takes blocks of one component that are neighbours in the plane: their symbol counts are
// alike, their bits are near one another and their rows leave as one run.
// Bound by instruction issue (61 % of the cycles) and the arithmetic pipe (53 %): about 30 instructions per symbol, of
// which a warp's longest block has some 28.  CTAS: as many per SM, by its registers.  Eight (64 registers, 40 words of the
// transform in local memory) where there are tiles for them; 4:4:4 images 500 us with six, 473 with seven, 461 with eight,
// 1024 photographs to 256x256 123, 119, 119.  Few tiles are done sooner without the detour.
template <int CTAS>
__global__ void __launch_bounds__(kBlockTile, CTAS)
blocks_kernel(const ImageDesc *__restrict__ descs, const uint2 *__restrict__ tiles, const HuffTable *__restrict__ huff,
              const MultTable *__restrict__ mult, EntropyScratch scratch, uint8_t *__restrict__ planes) {
    constexpr int kLook = 1 << kHuffBits;
    __shared__ __align__(16) uint32_t s_coef[32][kBlockTile];
    __shared__ __align__(16) uint16_t s_look[2][kLook]; // AC tables of luma and of the first chroma component
    __shared__ uint32_t s_mult[3][64]; // by zig-zag position: multiplier, and where the value goes << 16
    next_may_begin();
    const uint2 tile = tiles[blockIdx.x];
    const ImageDesc &d = descs[tile.x];
    const int tid = threadIdx.x;
    const int nx = d.idct_col1 - d.idct_col0, ny = d.mcu_rows - d.idct_row0, hs = d.hs, vs = d.vs;
    const int mcus = nx * ny, luma = hs * vs, n_luma = mcus * luma, luma_pad = (n_luma + 31) & ~31, chroma_pad = (mcus + 31) & ~31;
    const bool scaled = d.bs_luma != 8; // the coefficients stay as they are: the reduced transforms dequantise
    {
        const int first = (int)tile.y * kBlockTile; // which tables this tile needs
        for (int t = 0; t < (d.ncomp == 3 ? 2 : 1); t++) {
            if (t == 0 ? first >= luma_pad : first + kBlockTile <= luma_pad) continue;
            const uint4 *src = reinterpret_cast<const uint4 *>(huff[d.tab_id[d.ac_tab[t]]].look);
            for (int k = tid; k < kLook / 8; k += kBlockTile) reinterpret_cast<uint4 *>(s_look[t])[k] = src[k];
        }
        for (int k = tid; k < 64 * d.ncomp; k += kBlockTile) {
            const uint32_t m = scaled && (k < 64 || d.bs_chroma != 8) ? 1 : (uint16_t)mult[d.q_tab[k >> 6]].m[k & 63], n = c_natural[k & 63];
            s_mult[k >> 6][k & 63] = m | ((n >> 1) * kBlockTile * 4 + (n & 1) * 2) << 16;
        }
    }
    await_previous();
    __syncthreads();
    int item = (int)tile.y * kBlockTile + tid, comp = 0, bx, by, plane_w, bs;
    uint32_t blk;
    if (item < luma_pad) {
        if (item >= n_luma) return;
        const int row = nx * hs;
        by = item / row;
        bx = item - by * row + d.idct_col0 * hs;
        by += d.idct_row0 * vs;
        const int my = by / vs, mx = bx / hs;
        blk = (uint32_t)(my * d.mcus_x + mx) * d.bpm + (by - my * vs) * hs + (bx - mx * hs);
        bs = d.bs_luma;
        plane_w = d.mcus_x * hs * bs;
    } else {
        item -= luma_pad;
        comp = 1 + item / chroma_pad;
        item -= (comp - 1) * chroma_pad;
        if (d.ncomp != 3 || comp > 2 || item >= mcus) return;
        by = item / nx;
        bx = item - by * nx + d.idct_col0;
        by += d.idct_row0;
        blk = (uint32_t)(by * d.mcus_x + bx) * d.bpm + luma + comp - 1;
        bs = d.bs_chroma;
        plane_w = d.mcus_x * bs;
    }
    // ---- the block's coefficients
    const uint32_t p0 = scratch.pos[d.block_base + blk];
    int dc = scratch.dc[d.block_base + blk];
    if (d.seg_count > 1 && p0 != kNoBlock) dc += scratch.seg_dc[((size_t)d.seg_first + p0 / (d.seg_stride * 8)) * 4 + comp];
    const uint32_t *m = s_mult[comp];
    unsigned char *coef = reinterpret_cast<unsigned char *>(&s_coef[0][tid]);
#pragma unroll
    for (int k = 0; k < 32; k++) s_coef[k][tid] = kCoefZero;
    *reinterpret_cast<uint16_t *>(coef) = (uint16_t)((uint32_t)dc * m[0] + 0x8000);
    if (p0 != kNoBlock) {
        const int t = comp == 0 ? 0 : 1, table = d.ac_tab[comp];
        const bool in_shared = comp < 2 || table == d.ac_tab[1]; // (a table of its own for Cr: read where it is)
        const HuffTable *full = huff + d.tab_id[table];
        const uint32_t *words = reinterpret_cast<const uint32_t *>(scratch.clean + d.clean_off);
        uint32_t p = p0;
        const uint32_t *w32 = words + (p >> 5);
        uint32_t hi = w32[0], lo = w32[1], nx_ = w32[2], edge = (p & ~31u) + 32;
        w32 += 3;
        int z = 1;
        do {
            const uint32_t w = __funnelshift_l(lo, hi, p);
            uint32_t e = in_shared ? s_look[t][w >> (32 - kHuffBits)] : full->look[w >> (32 - kHuffBits)];
            if (e & kHuffLong) e = huff_long(full, e, w);
            const uint32_t n = e & 31, size = (e >> 5) & 15;
            p += n;
            const bool next = p >= edge;
            hi = next ? lo : hi;
            lo = next ? nx_ : lo;
            if (next) nx_ = *w32++;
            edge += next ? 32 : 0;
            z += (int)(e >> 9);
            const int at = z - 1; // where the value goes
            if (size != 0 && at < 64) { // (the low 16 bits of the product are the value's)
                const uint32_t to = m[at];
                *reinterpret_cast<uint16_t *>(coef + (to >> 16)) = (uint16_t)((uint32_t)huff_value(w, n, size) * to + 0x8000);
            }
        } while (z < 64);
    }
    uint8_t *dst = planes + d.plane_off[comp] + (size_t)(by * bs) * plane_w + bx * bs;
    if (bs == 8 && block_in_floats(&s_coef[0][tid], dst, plane_w)) return;
    asm volatile("" ::: "memory"); // (the words are read again: held since the first time they would cost 40 registers)
    int cw[32];
#pragma unroll
    for (int k = 0; k < 32; k++) cw[k] = (int)(s_coef[k][tid] ^ kCoefZero);
    if (bs != 8) { // scaled decode: this block becomes bs x bs samples
        const MultTable &mt = mult[d.q_tab[comp]];
        if (bs == 4) {
            reduced_block<2>(cw, mt.q, dst, plane_w);
        } else if (bs == 2) {
            reduced_block<4>(cw, mt.q, dst, plane_w);
        } else {
            const int a0 = coef_at(cw, 0) * (int)mt.q[0];
            dst[0] = (uint8_t)min(255, max(0, ((a0 + 4) >> 3) + 128));
        }
        return;
    }
    int v[8][8];
#pragma unroll
    for (int r = 0; r < 8; r++)
#pragma unroll
        for (int c = 0; c < 8; c++) v[r][c] = coef_at(cw, r * 8 + c);
#pragma unroll
    for (int c = 0; c < 8; c++)
        idct8(v[0][c], v[1][c], v[2][c], v[3][c], v[4][c], v[5][c], v[6][c], v[7][c]);
#pragma unroll
    for (int r = 0; r < 8; r++) {
        idct8(v[r][0], v[r][1], v[r][2], v[r][3], v[r][4], v[r][5], v[r][6], v[r][7]);
        uint32_t lo = 0, hi = 0;
#pragma unroll
        for (int c = 0; c < 8; c++) {
            int s = v[r][c] >> 5;
            s = min(127, max(-128, s)) + 128;
            if (c < 4)
                lo |= (uint32_t)s << (8 * c);
            else
                hi |= (uint32_t)s << (8 * (c - 4));
        }
        *reinterpret_cast<uint2 *>(dst + (size_t)r * plane_w) = make_uint2(lo, hi);
    }
}

void launch_blocks(const ImageDesc *descs, const uint2 *tiles, int n_tiles, const HuffTable *huff, const MultTable *mult,
                   const EntropyScratch &scratch, uint8_t *planes, bool early, cudaStream_t stream) {
    auto run = [&](auto kernel) { launch(early, n_tiles, kBlockTile, 0, stream, kernel, descs, tiles, huff, mult, scratch, planes); };
    if (n_tiles >= 148 * 8) run(blocks_kernel<8>);
    else if (n_tiles > 0) run(blocks_kernel<5>);
}

// ------------------------------------------------------------------------------------------

__device__ __forceinline__ int chroma_sample(const uint8_t *__restrict__ p, int W, int real_w,
                                             int real_h, int hs, int vs, int x, int y) {
    if (hs == 1) return p[(size_t)y * W + x];
    const int cx = x >> 1, cy = vs == 2 ? (y >> 1) : y;
    const uint8_t *row = p + (size_t)cy * W;
    if (real_w < 3) return row[cx];
    if (vs == 1) {
        const int cur = row[cx];
        if ((x & 1) == 0) return cx == 0 ? cur : (3 * cur + row[cx - 1] + 1) >> 2;
        return cx == real_w - 1 ? cur : (3 * cur + row[cx + 1] + 2) >> 2;
    }
    int ny = (y & 1) ? cy + 1 : cy - 1;
    ny = max(0, min(real_h - 1, ny));
    const uint8_t *far = p + (size_t)ny * W;
    const int cur = 3 * row[cx] + far[cx];
    if ((x & 1) == 0) {
        if (cx == 0) return (cur * 4 + 8) >> 4;
        return (cur * 3 + 3 * row[cx - 1] + far[cx - 1] + 8) >> 4;
    }
    if (cx == real_w - 1) return (cur * 4 + 7) >> 4;
    return (cur * 3 + 3 * row[cx + 1] + far[cx + 1] + 7) >> 4;
}

// Four pixels as three words of packed RGB.
__device__ __forceinline__ void pack_rgb4(uint32_t *w, const uint32_t *px) {
    w[0] = pick(px[0], px[1], 0x4210);
    w[1] = pick(px[1], px[2], 0x5421);
    w[2] = pick(px[2], px[3], 0x6542);
}

// Stores four RGB pixels at `o`: three words when the address allows and all four pixels exist, else the first
// `count` pixels by bytes.
__device__ __forceinline__ void store_rgb4(uint8_t *o, const uint32_t *px, int count, bool words) {
    if (words && count == 4) {
        pack_rgb4(reinterpret_cast<uint32_t *>(o), px);
    } else {
#pragma unroll
        for (int k = 0; k < 4; k++) {
            if (k >= count) break;
            o[3 * k] = (uint8_t)px[k];
            o[3 * k + 1] = (uint8_t)(px[k] >> 8);
            o[3 * k + 2] = (uint8_t)(px[k] >> 16);
        }
    }
}

// A warp stores `bytes` bytes of a row at `row` (shared memory, whole words; a word behind them may be read) to dst:
// consecutive words whatever dst's alignment, because the rows of a caller's image begin anywhere and may
// lie in host memory, where every partial sector is a transaction of its own.  With the six words of each
// thread stored one by one the kernel for 4:2:0 took 37 us for a 224x256 image in host memory (now 14) and 20 for one of
// 1213x1617 pixels on the GPU (now 11); calls with 4:4:4 images of 224x253 and 401x419 pixels took 283 and 565 us
// with single bytes (now 94 and 117).
constexpr int kRowPixels = 128, kRowWords = kRowPixels * 3 / 4 + 4;
__device__ __forceinline__ void store_row(uint8_t *dst, const uint32_t *row, int bytes, int lane) {
    const int head = min((int)(-reinterpret_cast<uintptr_t>(dst) & 3), bytes), words = (bytes - head) >> 2;
    const uint8_t *b = reinterpret_cast<const uint8_t *>(row);
    if (lane < head) dst[lane] = b[lane];
    for (int k = lane; k < words; k += 32)
        reinterpret_cast<uint32_t *>(dst + head)[k] = __funnelshift_r(row[k], row[k + 1], 8 * head);
    const int done = head + 4 * words;
    if (lane < bytes - done) dst[done + lane] = b[done + lane];
}

// The box of pixels to convert: the crop box when the batch has one (valid), else the image.
__device__ __forceinline__ void convert_box(const int32_t *params, int n_params, int img, int W, int H, int &x0,
                                            int &y0, int &x1, int &y1) {
    x0 = 0, y0 = 0, x1 = W, y1 = H;
    if (params) {
        const int32_t *p = params + (size_t)img * n_params;
        if (p[2] > 0 && p[3] > 0 && p[0] >= 0 && p[1] >= 0 && p[0] + p[2] <= H && p[1] + p[3] <= W) {
            y0 = p[0];
            x0 = p[1];
            y1 = p[0] + p[2];
            x1 = p[1] + p[3];
        }
    }
}

// 4:2:0 images: one thread per four chroma samples of a row = 8 x 2 output pixels (quad_pixels), a warp per
// 128 x 4, which leave through shared memory as whole rows.  Only the chroma cells the crop box touches are
// converted.
__global__ void __launch_bounds__(128)
color_quad_kernel(const ImageDesc *__restrict__ descs, const int32_t *__restrict__ list,
                  const uint2 *__restrict__ tiles, const uint8_t *__restrict__ planes, uint8_t *__restrict__ rgb,
                  const int32_t *__restrict__ params, int n_params) {
    next_may_begin();
    await_previous();
    // which sample and which tile of 64 x 8 chroma samples of its box: from the batch's tile table
    // (one CTA per tile that exists), or, without a table, from a grid that covers the largest box
    int img, tile_x, tile_y;
    if (tiles) {
        const uint2 t = tiles[blockIdx.x];
        img = (int)t.x;
        tile_x = (int)(t.y & 0xffff);
        tile_y = (int)(t.y >> 16);
    } else {
        img = list[blockIdx.z];
        tile_x = blockIdx.x;
        tile_y = blockIdx.y;
    }
    const ImageDesc &d = descs[img];
    if (d.host_status != 0 || d.ncomp != 3 || d.hs != 2 || d.vs != 2 || d.scale_shift != 0 || d.fuse_rows) return;
    const int W = d.width, H = d.height;
    const QuadPlanes p{planes + d.plane_off[0], planes + d.plane_off[1], planes + d.plane_off[2], d.mcus_x * 16, d.mcus_x * 8, (W + 1) >> 1, (H + 1) >> 1};
    if (p.real_w < 3) return; // too narrow for the filter: the per-pixel kernel replicates
    int x0, y0, x1, y1;
    convert_box(params, n_params, img, W, H, x0, y0, x1, y1);
    __shared__ __align__(16) uint32_t s_rows[8][2][kRowWords];
    const int first = ((x0 >> 1) & ~3) + 64 * tile_x, cx = first + 4 * threadIdx.x, cy = (y0 >> 1) + tile_y * 8 + threadIdx.y;
    if (cx <= ((x1 - 1) >> 1) && cy <= ((y1 - 1) >> 1)) {
        uint32_t px[2][8];
        quad_pixels(p, cx, cy, px);
#pragma unroll
        for (int r = 0; r < 2; r++) {
            pack_rgb4(&s_rows[threadIdx.y][r][6 * threadIdx.x], px[r]);
            pack_rgb4(&s_rows[threadIdx.y][r][6 * threadIdx.x + 3], px[r] + 4);
        }
    }
    __syncwarp();
    const int lane = threadIdx.x + 16 * (threadIdx.y & 1), count = min(kRowPixels, x1 - 2 * first);
    if (count <= 0) return;
    for (int k = 0; k < 4; k++) { // the warp's rows
        const int c = (threadIdx.y & ~1) + (k >> 1), y = 2 * ((y0 >> 1) + tile_y * 8 + c) + (k & 1);
        if (y < y1) store_row(rgb + d.rgb_off + (size_t)y * d.rgb_pitch + (size_t)first * 6, s_rows[c][k & 1], 3 * count, lane);
    }
}

// 4:4:4 images, and images decoded at reduced scale (whose chroma blocks were inverted to the luma
// resolution): no upsampling, one thread per four pixels of a row of the crop box (one word of each
// plane in, three words out), every thread walking a column strip so that the grid stays small
// for very large images.  kRows: rows leave whole (store_row), for results whose rows do not begin on words or that
// lie in host memory; on the GPU the three words of each thread are better (64 images of 1200x1400: 190 us, 231
// with whole rows).
template <bool kRows>
__global__ void __launch_bounds__(256)
color_444_kernel(const ImageDesc *__restrict__ descs, const int32_t *__restrict__ list,
                 const uint8_t *__restrict__ planes, uint8_t *__restrict__ rgb,
                 const int32_t *__restrict__ params, int n_params) {
    next_may_begin();
    await_previous();
    const int img = list[blockIdx.z];
    const ImageDesc &d = descs[img];
    if (d.host_status != 0 || d.ncomp != 3 || !(d.scale_shift != 0 || (d.hs == 1 && d.vs == 1)) || d.fuse_rows) return;
    const int W = d.dec_width, H = d.dec_height;
    int x0, y0, x1, y1;
    convert_box(params, n_params, img, W, H, x0, y0, x1, y1);
    const int pw = d.mcus_x * d.hs * d.bs_luma; // = the chroma planes' pitch: all planes have one resolution here
    const uint8_t *Y = planes + d.plane_off[0], *Cb = planes + d.plane_off[1], *Cr = planes + d.plane_off[2];
    uint8_t *out = rgb + d.rgb_off;
    __shared__ __align__(16) uint32_t s_rows[kRows ? 8 : 1][kRowWords];
    const int first = (x0 & ~3) + kRowPixels * blockIdx.x, x = first + 4 * threadIdx.x;
    if (kRows ? first >= x1 : x >= x1) return;
    const int count = min(4, W - x);
    // a plane's pitch is a multiple of 8 only at full scale; reduced planes may be narrower
    const bool words_in = ((pw | (int)(d.plane_off[0] | d.plane_off[1] | d.plane_off[2])) & 3) == 0;
    const bool words_out = ((reinterpret_cast<uintptr_t>(out) | d.rgb_pitch) & 3) == 0;
    for (int y = y0 + blockIdx.y * 8 + threadIdx.y; y < y1; y += gridDim.y * 8) {
        uint32_t px[4];
        if (!kRows) {
            plain_pixels(Y, Cb, Cr, (size_t)y * pw + x, count, words_in, px);
            store_rgb4(out + (size_t)y * d.rgb_pitch + (size_t)x * 3, px, count, words_out);
            continue;
        }
        if (x < x1) {
            plain_pixels(Y, Cb, Cr, (size_t)y * pw + x, count, words_in, px);
            pack_rgb4(&s_rows[threadIdx.y][3 * threadIdx.x], px);
        }
        __syncwarp();
        store_row(out + (size_t)y * d.rgb_pitch + (size_t)first * 3, s_rows[threadIdx.y], 3 * min(kRowPixels, x1 - first), threadIdx.x);
        __syncwarp();
    }
}

// Per-pixel kernel for everything the kernels above leave out (4:2:2, greyscale, 4:2:0 images
// narrower than the triangle filter).  kRows: where rows follow one another without a gap, as those of a single
// image do, a warp's 32 pixels leave as 24 words (a choice at run time costs batches a third: 211 -> 277 us for 256
// 4:2:2 images of 300x400).
template <bool kRows>
__global__ void __launch_bounds__(256)
color_other_kernel(const ImageDesc *__restrict__ descs, const int32_t *__restrict__ list,
                   const uint8_t *__restrict__ planes, uint8_t *__restrict__ rgb) {
    next_may_begin();
    await_previous();
    const ImageDesc &d = descs[list[blockIdx.y]];
    if (d.host_status != 0) return;
    const int W = d.width, H = d.height;
    const int real_w = (W + d.hs - 1) / d.hs, real_h = (H + d.vs - 1) / d.vs;
    if (d.scale_shift != 0) return;                                      // equal-resolution kernel's
    if (d.ncomp == 3 && d.hs == 2 && d.vs == 2 && real_w >= 3) return; // quad kernel's
    if (d.ncomp == 3 && d.hs == 1 && d.vs == 1) return;                  // 4:4:4 kernel's
    const int npix = W * H;
    const int yw = d.mcus_x * d.hs * 8, cw = d.mcus_x * 8;
    const uint8_t *Y = planes + d.plane_off[0];
    const uint8_t *Cb = planes + d.plane_off[1];
    const uint8_t *Cr = planes + d.plane_off[2];
    uint8_t *out = rgb + d.rgb_off;
    __shared__ __align__(16) uint8_t s_pixels[kRows ? 256 / 32 : 1][32 * 3];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const bool gapless = kRows && d.rgb_pitch == (uint32_t)W * 3 && (reinterpret_cast<uintptr_t>(out) & 3) == 0;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < npix; i += gridDim.x * blockDim.x) {
        const int y = i / W, x = i - y * W;
        const int lum = Y[(size_t)y * yw + x];
        int r = lum, g = lum, b = lum;
        if (d.ncomp == 3) {
            const int cb = chroma_sample(Cb, cw, real_w, real_h, d.hs, d.vs, x, y) - 128;
            const int cr = chroma_sample(Cr, cw, real_w, real_h, d.hs, d.vs, x, y) - 128;
            r = lum + ((91881 * cr + 32768) >> 16);
            g = lum + ((-22554 * cb - 46802 * cr + 32768) >> 16);
            b = lum + ((116130 * cb + 32768) >> 16);
        }
        const bool whole = gapless && i - lane + 32 <= npix; // (uniform in the warp)
        uint8_t *o = whole ? &s_pixels[warp][3 * lane] : out + (size_t)y * d.rgb_pitch + (size_t)x * 3;
        o[0] = (uint8_t)min(255, max(0, r));
        o[1] = (uint8_t)min(255, max(0, g));
        o[2] = (uint8_t)min(255, max(0, b));
        if (whole) {
            __syncwarp();
            if (lane < 24) reinterpret_cast<uint32_t *>(out + 3 * (size_t)(i - lane))[lane] = reinterpret_cast<const uint32_t *>(s_pixels[warp])[lane];
            __syncwarp();
        }
    }
}

void launch_color(const ImageDesc *descs, const int32_t *list, int n_list, int n_quad, int n_444, int n_other,
                  int max_w, int max_h, const uint2 *quad_tiles, int n_quad_tiles, const uint8_t *planes, uint8_t *rgb, const int32_t *crop_params,
                  int n_params, bool whole_rows, bool early, cudaStream_t stream) {
    if (n_list == 0) return;
    if (n_444 > 0) {
        int gy = (max_h + 7) / 8;
        if (gy > 64) gy = 64;
        dim3 grid(((max_w + 3) / 4 + 1 + 31) / 32, gy, n_list); // + 1: a box starts up to 3 pixels into its first group
        launch(early, grid, dim3(32, 8), 0, stream, whole_rows ? color_444_kernel<true> : color_444_kernel<false>, descs, list, planes, rgb, crop_params, n_params);
    }
    if (n_quad > 0 && quad_tiles != nullptr) {
        if (n_quad_tiles > 0)
            launch(early, n_quad_tiles, dim3(16, 8), 0, stream, color_quad_kernel, descs, list, quad_tiles, planes, rgb, crop_params, n_params);
    } else if (n_quad > 0) {
        launch(early, dim3(quad_tiles_x(max_w), quad_tiles_y(max_h), n_list), dim3(16, 8), 0, stream, color_quad_kernel, descs, list, nullptr, planes, rgb,
               crop_params, n_params);
    }
    if (n_other > 0) {
        int bx = (max_w * max_h + 256 * 4 - 1) / (256 * 4);
        bx = bx < 1 ? 1 : (bx > 1024 ? 1024 : bx);
        launch(early, dim3(bx, n_list), 256, 0, stream, whole_rows ? color_other_kernel<true> : color_other_kernel<false>, descs, list, planes, rgb);
    }
}

} // namespace ffcvb
