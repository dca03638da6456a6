// Fused crop + INTER_AREA resize + flip / translate / cutout + lookup-table normalise (sm_100a).
//
// Replaces, in one pass over the output, the chain the reference runs as separate CPU loops:
//   cv::resize(roi, dst, INTER_AREA)      libffcv/libffcv.cpp:33-42 (from rgb_image.py:205-208)
//   RandomHorizontalFlip                  ffcv/transforms/flip.py:31-39
//   RandomTranslate                       ffcv/transforms/translate.py:35-44
//   Cutout                                ffcv/transforms/cutout.py:36-46
//   NormalizeImage (256x3 table gather)   ffcv/transforms/normalize.py:58-109
// Every output pixel traces backwards through the augmentations to either a fill colour or a
// pixel of the resized crop, whose value is computed with OpenCV's INTER_AREA arithmetic:
//   equal size -> copy; integer factors -> box sum ((s+2)>>2 for 2x2, else
//   round-half-even(float(s) * float(1/area))); both factors >= 1 -> separable fractional
//   coverage accumulated in fp32 in source order (no FMA contraction); any factor < 1 -> 2-tap
//   interpolation on both axes with 11-bit fixed-point weights.
// Byte work bound by instruction issue: a few CTAs per sample, each producing every k-th band of output rows;
// tap positions and weights are computed once per CTA into shared memory and serve all its bands.  The
// source pixels a band reads are gathered in a window in shared memory first, one word per pixel, so
// that a tap is one load for three channels.  For JPEG samples the window is filled from the decoded
// planes: chroma upsampling and colour conversion happen there and no RGB image travels through global
// memory (taps come from global memory byte by byte when too few rows fit).  Every band's normalised tile is
// assembled in shared memory and leaves with coalesced 16-byte stores.  In the fractional shrinking and the
// enlarging regime a thread owns an output column for a run of rows, so that what a source row contributes
// (its horizontal sums, its interpolated values) is shared by the output rows that touch it; what a
// translation or a cutout fills is painted over the band afterwards.
#include "color.h"
#include "kernels.h"
#include "two.h"

#include <type_traits>

namespace ffcvb {

enum { kOpFlip = 1, kOpTranslate = 2, kOpCutout = 3 };
enum { kOutU8 = 0, kOutF16Nhwc = 1, kOutF16Nchw = 2, kOutF32Nhwc = 3, kOutF32Nchw = 4 };

struct AreaTaps {
    int first, n;
    float wl, wm, wr;
    bool has_l, has_r;
};

// a / b correctly rounded, given the correctly rounded 1 / b: the product with the reciprocal is
// within 1.5 ulp, a first remainder step makes it faithful, a second one correctly rounded
// (Markstein); three double-precision divisions per tap would otherwise dominate the CTA's set-up.
__device__ __forceinline__ double quotient(double a, double b, double inv_b) {
    double q = a * inv_b;
    q = fma(fma(-b, q, a), inv_b, q);
    return fma(fma(-b, q, a), inv_b, q);
}

// Source cells covering destination cell d of an axis shrunk by `scale` (>= 1).
__device__ __forceinline__ AreaTaps area_taps(int d, int ssize, double scale) {
    AreaTaps t;
    const double f1 = d * scale, f2 = f1 + scale;
    const double cell = fmin(scale, ssize - f1);
    int s1 = (int)ceil(f1), s2 = (int)floor(f2);
    s2 = min(s2, ssize - 1);
    s1 = min(s1, s2);
    t.has_l = (s1 - f1) > 1e-3;
    t.has_r = (f2 - s2) > 1e-3;
    const double inv_cell = 1.0 / cell;
    t.wl = (float)quotient(s1 - f1, cell, inv_cell);
    t.wm = (float)inv_cell;
    t.wr = (float)quotient(fmin(fmin(f2 - s2, 1.0), cell), cell, inv_cell);
    t.first = t.has_l ? s1 - 1 : s1;
    t.n = (t.has_l ? 1 : 0) + (s2 - s1) + (t.has_r ? 1 : 0);
    return t;
}

// Two-tap position and 11-bit weights of destination index d when some axis is enlarged.
__device__ __forceinline__ void linear_taps(int d, int ssize, double inv, double scale, bool clamp_last,
                                            int &s, int &w0, int &w1) {
    s = (int)floor(d * scale);
    float f = (float)((d + 1) - (s + 1) * inv);
    f = f <= 0.f ? 0.f : f - floorf(f);
    if (clamp_last && s >= ssize - 1) {
        f = 0.f;
        s = ssize - 1;
    }
    w0 = min(32767, __float2int_rn(__fmul_rn(__fsub_rn(1.f, f), 2048.f)));
    w1 = min(32767, __float2int_rn(__fmul_rn(f, 2048.f)));
    if (clamp_last && s + 1 >= ssize) {
        w0 = 2048;
        w1 = 0;
    }
}

__device__ __forceinline__ int sat_round(float v) { return min(255, max(0, __float2int_rn(v))); }

// Byte k of a pixel -> float without the conversion pipe: 2^23 + v is representable; the 2^23 is taken off
// again inside the multiplication, fma(2^23 + v, w, -2^23 * w)
constexpr uint32_t kBias = 0x4B000000u; // the bits of 2^23
template <int k>
__device__ __forceinline__ float biased(uint32_t px) {
    return __uint_as_float(pick(px, kBias, 0x7440u | k));
}

// A pixel of a row: of the window's words, or of packed bytes.  (Those one by one: the aligned words that hold a pixel are
// fewer requests, but took 276 us instead of 258 for 64 images of 1200x1400 pixels to 224x224.)
__device__ __forceinline__ uint32_t pixel(const uint32_t *row, int x) { return row[x]; }
__device__ __forceinline__ uint32_t pixel(const uint8_t *row, int x) {
    const uint8_t *p = row + 3 * x;
    return (uint32_t)p[0] | (uint32_t)p[1] << 8 | (uint32_t)p[2] << 16;
}

// Taps of an output column or row, computed once per CTA (double-precision position arithmetic as
// OpenCV does it, then only fp32 / integer work per pixel).  Area: first and number of the source indices, weights
// of the first, the middle and the last tap (0 if there is only one).
__device__ __forceinline__ uint4 make_area_taps(int d, int ssize, double scale) {
    const AreaTaps a = area_taps(d, ssize, scale);
    const float last = a.has_r ? a.wr : a.wm, first = a.has_l ? a.wl : (a.n == 1 ? last : a.wm);
    return make_uint4((uint32_t)a.first | (uint32_t)a.n << 16, __float_as_uint(first), __float_as_uint(a.wm),
                      __float_as_uint(a.n == 1 ? 0.f : last));
}
// Linear: the two source indices and their weights.
__device__ __forceinline__ uint4 make_linear_taps(int d, int ssize, double inv, double scale, bool clamp_last) {
    int s, w0, w1;
    linear_taps(d, ssize, inv, scale, clamp_last, s, w0, w1);
    return make_uint4((uint32_t)min(s, ssize - 1), (uint32_t)min(s + 1, ssize - 1), __float_as_uint((float)w0), __float_as_uint((float)w1));
}

// Two neighbouring columns' horizontal sums: first tap, the whole cells between, last tap, rounded after every
// operation.  fma(2^23 + v, w, -2^23 * w) is the correctly rounded v * w, exactly what the multiplication of the
// converted value gives (2^23 * w is exact).  The columns share their instructions, one channel at a time.  A cell of
// `scale` pixels has scale - 0.002 <= n < scale + 1.998 taps (area_taps), so the columns have equally many or one has
// one more; the other's pixel there may be the one behind the crop's last, and its weight is zero, which changes no sum.
// (V = One: a single column; b is a's.)
template <class V>
struct AreaColumns {
    int first[2], mids, taps; // tap `mids` + 1 is the first that is the last one of either column
    V w_first, w_mid, w_tail[2];
    __device__ __forceinline__ AreaColumns(uint4 a, uint4 b) {
        const int na = (int)(a.x >> 16), nb = (int)(b.x >> 16);
        first[0] = (int)(a.x & 0xffff);
        first[1] = (int)(b.x & 0xffff);
        taps = max(na, nb);
        mids = max(min(na, nb) - 2, 0);
        w_first = V(__uint_as_float(a.y), __uint_as_float(b.y));
        w_mid = V(__uint_as_float(a.z), __uint_as_float(b.z));
#pragma unroll
        for (int k = 0; k < 2; k++) w_tail[k] = V(weight(a, mids + 1 + k), weight(b, mids + 1 + k));
    }
    // of tap k >= 1
    static __device__ __forceinline__ float weight(uint4 t, int k) {
        const int last = (int)(t.x >> 16) - 1;
        return k < last ? __uint_as_float(t.z) : (k == last ? __uint_as_float(t.w) : 0.f);
    }
    static __device__ __forceinline__ void tap(uint32_t p, uint32_t q, V w, V (&v)[3]) {
        const V c = mul_rn(w, V(-8388608.0f, -8388608.0f));
        v[0] = fma_rn(V(biased<0>(p), biased<0>(q)), w, c);
        v[1] = fma_rn(V(biased<1>(p), biased<1>(q)), w, c);
        v[2] = fma_rn(V(biased<2>(p), biased<2>(q)), w, c);
    }
    template <class Row>
    __device__ __forceinline__ void more(Row row, int k, V w, V (&sum)[3]) const {
        V v[3];
        tap(pixel(row, first[0] + k), pixel(row, first[1] + k), w, v);
#pragma unroll
        for (int c = 0; c < 3; c++) sum[c] = add_rn(sum[c], v[c]);
    }
    template <class Row>
    __device__ __forceinline__ void across(Row row, V (&sum)[3]) const {
        tap(pixel(row, first[0]), pixel(row, first[1]), w_first, sum);
        for (int k = 1; k <= mids; k++) more(row, k, w_mid, sum);
        if (taps > mids + 1) more(row, mids + 1, w_tail[0], sum);
        if (taps > mids + 2) more(row, mids + 2, w_tail[1], sum);
    }
};

// OpenCV's fixed-point bilinear, in floating point whose roundings do what the shifts do: with S the two taps'
// weighted sum (an exact integer below 2^20), 2^27 + S rounded down is 2^27 + 16 * (S >> 4), and
// fma(b, that, 2^43 - 2^27 * b) rounded down is 2^43 + 2^20 * (b * (S >> 4) >> 16), the product of the integers
// in the low bits of its mantissa.  Two neighbouring columns share their instructions.
template <class V>
struct LinearColumns {
    int x0[2], x1[2];
    V w0, w1, c0, c1;
    __device__ __forceinline__ LinearColumns(uint4 a, uint4 b) {
        x0[0] = (int)a.x, x1[0] = (int)a.y;
        x0[1] = (int)b.x, x1[1] = (int)b.y;
        w0 = V(__uint_as_float(a.z), __uint_as_float(b.z));
        w1 = V(__uint_as_float(a.w), __uint_as_float(b.w));
        c0 = mul_rn(w0, V(-8388608.0f, -8388608.0f));
        c1 = mul_rn(w1, V(-8388608.0f, -8388608.0f));
    }
    template <class Row>
    __device__ __forceinline__ void across(Row row, V (&h)[3]) const {
        const uint32_t p0 = pixel(row, x0[0]), q0 = pixel(row, x0[1]), p1 = pixel(row, x1[0]), q1 = pixel(row, x1[1]);
        auto one = [&](float a0, float b0, float a1, float b1) {
            const V s = add_rn(fma_rn(V(a0, b0), w0, c0), fma_rn(V(a1, b1), w1, c1));
            return add_rd(s, V(134217728.f, 134217728.f));
        };
        h[0] = one(biased<0>(p0), biased<0>(q0), biased<0>(p1), biased<0>(q1));
        h[1] = one(biased<1>(p0), biased<1>(q0), biased<1>(p1), biased<1>(q1));
        h[2] = one(biased<2>(p0), biased<2>(q0), biased<2>(p1), biased<2>(q1));
    }
};
// A column's value out of the two rows' products.  (The weights' sum is at most 2049, so 255 is not exceeded.)
__device__ __forceinline__ uint32_t blended(float upper, float lower) { return (__float_as_uint(upper) + __float_as_uint(lower) + 2u - 2u * (170u << 23)) >> 2; }

// a / n for a, n < 2^16, inv_n = ceil(2^32 / n)
__device__ __forceinline__ int divided(uint32_t a, uint32_t inv_n, int n) { return n == 1 ? (int)a : (int)__umulhi(a, inv_n); }
__host__ __device__ __forceinline__ uint32_t inverse(int n) { return 0xFFFFFFFFu / (uint32_t)n + 1u; }

// One of SmallCopies, by a CTA of 256 threads: every thread has its words (at most kSmallCopyWords / 256) under way
// at once.
template <typename Word>
__device__ __forceinline__ void copy_words(const uint8_t *__restrict__ src, uint8_t *__restrict__ dst, uint32_t bytes) {
    constexpr int kEach = kSmallCopyWords / 256;
    const uint32_t n = bytes / sizeof(Word);
    const Word *from = reinterpret_cast<const Word *>(src);
    Word *to = reinterpret_cast<Word *>(dst), v[kEach];
#pragma unroll
    for (int k = 0; k < kEach; k++)
        if (threadIdx.x + 256 * k < n) v[k] = from[threadIdx.x + 256 * k];
#pragma unroll
    for (int k = 0; k < kEach; k++)
        if (threadIdx.x + 256 * k < n) to[threadIdx.x + 256 * k] = v[k];
    const uint32_t done = n * (uint32_t)sizeof(Word);
    if (threadIdx.x < bytes - done) dst[done + threadIdx.x] = src[done + threadIdx.x];
}
__device__ __noinline__ void copy_small(const uint8_t *src, uint8_t *dst, uint32_t bytes) {
    const uint32_t word = copy_word(src, dst);
    if (word == 16)
        copy_words<uint4>(src, dst, bytes);
    else if (word == 4)
        copy_words<uint32_t>(src, dst, bytes);
    else
        copy_words<uint8_t>(src, dst, bytes);
}

// kPlain: for batches with crops that are interpolated without a window.  Where there are none the kernel does without that way, which
// costs the other one 3 % by being there (1024 images to 160x160 252 and 258 us).
template <typename OutT, bool kPlain>
__global__ void __launch_bounds__(256, 4)
resize_augment_kernel(const __grid_constant__ ResizeSource src, const int32_t *__restrict__ params, int n_params,
                      const ResizeItem *__restrict__ items,
                      const __grid_constant__ OpList ops,
                      int resize, int out_h, int out_w, const __grid_constant__ ResizeShape shape, int planar,
                      const OutT *__restrict__ lut, OutT *__restrict__ out,
                      const int32_t *__restrict__ status, const __grid_constant__ SmallCopies small) {
    extern __shared__ __align__(16) unsigned char s_raw[];
    await_previous();
    constexpr bool kU8 = sizeof(OutT) == 1;
    // shared layout: [lut][x taps][y taps][out tile][window of source pixels]; y taps are indexed by the row of
    // the resized crop (a translation can move a band anywhere)
    int band0 = 0, rows = 0; // the band of output rows being produced (see the loop below)
    OutT *s_lut = reinterpret_cast<OutT *>(s_raw);
    uint4 *tx = reinterpret_cast<uint4 *>(s_raw + 768 * sizeof(OutT)), *ty = tx + out_w;
    OutT *s_out = reinterpret_cast<OutT *>(ty + out_h);
    const size_t tile_row = (size_t)out_w * 3 * sizeof(OutT);

    const int i = blockIdx.y;
    if (blockIdx.x == 0 && i == 0)
        for (int k = 0; k < small.n; k++) copy_small(small.src[k], small.dst[k], (uint32_t)small.bytes[k]);
    ResizeItem item{};
    if (resize) item = items[i];

    // ---- where the sample's pixels are
    const uint8_t *base;
    int stride, row0 = 0, col0 = 0, img_h, img_w;
    // rows of a gathered crop box start at their source alignment inside their slot (raw_skew)
    uint32_t skew_base = 0, skew_pitch = 0;
    bool skew = false;
    bool ok = true;
    bool fuse = false; // a sample whose planes are converted here
    if (src.descs) {
        const ImageDesc &d = src.descs[i];
        img_h = d.dec_height; // the decoded size: smaller than the stored one after a scaled decode
        img_w = d.dec_width;
        stride = (int)d.rgb_pitch;
        if (d.mode == 1) {
            base = src.blob + d.payload_off;
            row0 = d.row0;
            col0 = d.col0;
            stride = (int)d.raw_pitch;
            ok = d.host_status == 0;
            if (d.raw_skew) {
                skew = true;
                skew_base = (uint32_t)(d.src_addr & 15);
                skew_pitch = (uint32_t)d.width * 3;
            }
        } else {
            base = src.rgb + d.rgb_off;
            fuse = d.fuse_rows != 0;
            ok = d.host_status == 0 && (status == nullptr || status[i] == 0);
        }
    } else {
        img_h = src.uniform_h;
        img_w = src.uniform_w;
        stride = img_w * 3;
        base = src.uniform + (size_t)i * img_h * stride;
    }
    const int32_t *prm = params + (size_t)i * n_params;
    int ci = 0, cj = 0, ch = out_h, cw = out_w;
    if (resize) {
        ci = prm[0];
        cj = prm[1];
        ch = prm[2];
        cw = prm[3];
        ok = ok && ch > 0 && cw > 0 && ci >= 0 && cj >= 0 && ci + ch <= img_h && cj + cw <= img_w;
    } else {
        ok = ok && img_h == out_h && img_w == out_w;
    }
    // What is not filled maps to the crop's rows and columns with an offset and a direction.
    bool flips_only = true; // nothing is ever filled
    int dy = 0, dx = 0, step_x = 1;
    for (int k = ops.n_ops - 1; k >= 0; k--) {
        flips_only = flips_only && ops.type[k] == kOpFlip;
        if (ops.type[k] == kOpTranslate) {
            dy += prm[4 + 2 * k] - ops.arg[k];
            dx += prm[5 + 2 * k] - ops.arg[k];
        } else if (ops.type[k] == kOpFlip && prm[4 + 2 * k]) {
            dx = out_w - 1 - dx;
            step_x = -step_x;
        }
    }

    const int window = ok ? item.window : 0, band_rows = window ? window : shape.band;
    const int lead = item.lead, wpitch = window_pitch(cw), groups = item.groups;
    uint32_t *s_win = reinterpret_cast<uint32_t *>(reinterpret_cast<unsigned char *>(s_out) + (((size_t)band_rows * tile_row + 15) & ~(size_t)15));
    const int nbands = (out_h + band_rows - 1) / band_rows;
    if ((int)blockIdx.x >= nbands) return;
    if (!kU8)
        for (int k = threadIdx.x; k < 768; k += blockDim.x) s_lut[(k % 3) * 256 + k / 3] = lut[k]; // per channel
    const int regime = ok ? item.regime : kCopy, isx = item.isx, isy = item.isy;
    if (regime == kArea || regime == kLinear) {
        // x taps of every column, y taps of the rows of the crop that this CTA needs
        const int my_bands = (nbands - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x;
        for (int e = threadIdx.x; e < out_w + my_bands * band_rows; e += blockDim.x) {
            const bool column = e < out_w;
            const int k = e - out_w, b = column ? 0 : k / band_rows;
            const int at = column ? e : ((int)blockIdx.x + b * (int)gridDim.x) * band_rows + (k - b * band_rows) + dy;
            if (at < 0 || at >= (column ? out_w : out_h)) continue;
            const int ssize = column ? cw : ch;
            const double inv = column ? item.inv_x : item.inv_y, scale = column ? item.sc_x : item.sc_y;
            (column ? tx : ty)[at] = regime == kArea ? make_area_taps(at, ssize, scale) : make_linear_taps(at, ssize, inv, scale, column);
        }
    }
    __syncthreads();

    const int roff = ci - row0, coff = (cj - col0) * 3;
    auto row_ptr = [&](int y) -> const uint8_t * { // first pixel of row y of the crop
        const int rr = roff + y;
        const uint8_t *p = base + (ptrdiff_t)rr * stride + coff;
        if (skew) p += (skew_base + (uint32_t)rr * skew_pitch) & 15u;
        return p;
    };
    int npix = 0;
    const uint32_t inv_w = inverse(out_w), inv_pairs = inverse((out_w + 1) >> 1);
    // Traces an output pixel back through the augmentations: either a fill colour, or the position
    // (y, x) of a pixel of the resized crop.
    auto trace = [&](int oy, int ox, int &y, int &x, int *val) -> bool {
        y = oy;
        x = ox;
        bool filled = false;
        for (int k = ops.n_ops - 1; k >= 0 && !filled; k--) {
            const int a = prm[4 + 2 * k], b = prm[5 + 2 * k];
            const int type = ops.type[k], arg = ops.arg[k];
            if (type == kOpCutout) {
                filled = y >= a && y < a + arg && x >= b && x < b + arg;
            } else if (type == kOpTranslate) {
                y += a - arg;
                x += b - arg;
                filled = y < 0 || y >= out_h || x < 0 || x >= out_w;
            } else if (type == kOpFlip) {
                if (a) x = out_w - 1 - x;
            }
            if (filled) {
                val[0] = ops.fill[k][0];
                val[1] = ops.fill[k][1];
                val[2] = ops.fill[k][2];
            }
        }
        return filled;
    };
    // normalise (table gather, one 256-entry table per channel) into the shared tile, in final
    // memory order: element = pix * pix_step + c * chan_step
    int pix_step = 3, chan_step = 1;
    auto emit = [&](OutT *o, int v0, int v1, int v2) {
        if constexpr (kU8) {
            o[0] = (OutT)v0;
            o[chan_step] = (OutT)v1;
            o[2 * chan_step] = (OutT)v2;
        } else {
            o[0] = s_lut[v0];
            o[chan_step] = s_lut[256 + v1];
            o[2 * chan_step] = s_lut[512 + v2];
        }
    };
    // The same for two neighbouring pixels of a row, the first of an even column; `bias` is on top of every value.
    // They leave as whole words (bytes: half-words) where rows have an even number of pixels.  width 1: only the first.
    const bool even = (out_w & 1) == 0;
    const uint32_t lut_address = (uint32_t)__cvta_generic_to_shared(s_lut);
    auto emit_pair = [&](OutT *o, const uint32_t (&v)[2][3], uint32_t bias, bool both, int width) {
        uint32_t e[2][3];
#pragma unroll
        for (int p = 0; p < 2; p++)
#pragma unroll
            for (int c = 0; c < 3; c++) {
                // (the bias goes out of the address, which has 32 bits like the product)
                const uint32_t at = lut_address - bias * (uint32_t)sizeof(OutT) + v[p][c] * (uint32_t)sizeof(OutT);
                if constexpr (kU8)
                    e[p][c] = v[p][c];
                else if constexpr (sizeof(OutT) == 2)
                    asm("{\n\t.reg .u16 h;\n\tld.shared.u16 h, [%1];\n\tcvt.u32.u16 %0, h;\n\t}" : "=r"(e[p][c]) : "r"(at + 256 * 2 * c));
                else
                    asm("ld.shared.u32 %0, [%1];" : "=r"(e[p][c]) : "r"(at + 256 * 4 * c));
            }
        if (width == 1 || !even) {
#pragma unroll
            for (int p = 0; p < 2; p++) {
                if (p == 1 && !both) break;
#pragma unroll
                for (int c = 0; c < 3; c++) o[p * pix_step + c * chan_step] = (OutT)e[p][c];
            }
        } else if constexpr (kU8) {
            uint16_t *w = reinterpret_cast<uint16_t *>(o);
            w[0] = (uint16_t)pick(e[0][0], e[0][1], 0x0040);
            w[1] = (uint16_t)pick(e[0][2], e[1][0], 0x0040);
            w[2] = (uint16_t)pick(e[1][1], e[1][2], 0x0040);
        } else if constexpr (sizeof(OutT) == 2) {
            if (planar) {
#pragma unroll
                for (int c = 0; c < 3; c++) *reinterpret_cast<uint32_t *>(o + c * chan_step) = pick(e[0][c], e[1][c], 0x5410);
            } else {
                uint32_t *w = reinterpret_cast<uint32_t *>(o);
                w[0] = pick(e[0][0], e[0][1], 0x5410);
                w[1] = pick(e[0][2], e[1][0], 0x5410);
                w[2] = pick(e[1][1], e[1][2], 0x5410);
            }
        } else {
            if (planar) {
#pragma unroll
                for (int c = 0; c < 3; c++) *reinterpret_cast<uint2 *>(o + c * chan_step) = make_uint2(e[0][c], e[1][c]);
            } else {
                uint2 *w = reinterpret_cast<uint2 *>(o);
                w[0] = make_uint2(e[0][0], e[0][1]);
                w[1] = make_uint2(e[0][2], e[1][0]);
                w[2] = make_uint2(e[1][1], e[1][2]);
            }
        }
    };
    // A CTA produces every gridDim.x-th band of its image: what was set up above (descriptor, tap
    // tables, lookup table) serves all of them.
    for (int band = blockIdx.x; band < nbands; band += gridDim.x) {
    band0 = band * band_rows;
    rows = min(band_rows, out_h - band0);
    npix = rows * out_w;
    pix_step = planar ? 1 : 3;
    chan_step = planar ? npix : 1;
    // The source pixels this band reads, in the window: rows win_lo .. of the crop, `wpitch` words apart, the crop's
    // first column at `lead`.
    int win_lo = 0;
    const int y_lo = max(0, band0 + dy), y_hi = min(out_h, band0 + rows + dy); // rows of the crop in this band
    if (window && y_lo < y_hi) {
        const uint4 top = ty[y_lo], bottom = ty[y_hi - 1];
        win_lo = (int)(regime == kArea ? top.x & 0xffff : top.x);
        const int hi = (int)(regime == kArea ? (bottom.x & 0xffff) + (bottom.x >> 16) - 1 : bottom.y);
        const int units = item.units;
        const uint32_t inv_units = item.inv_units;
        if (fuse) {
            const ImageDesc &d = src.descs[i];
            const uint8_t *py = src.planes + d.plane_off[0], *pb = src.planes + d.plane_off[1], *pr = src.planes + d.plane_off[2];
            const int r0 = ci + win_lo, r1 = ci + hi; // rows of the image
            if (d.scale_shift == 0 && d.hs == 2) {
                const QuadPlanes p{py, pb, pr, d.mcus_x * 16, d.mcus_x * 8, (d.width + 1) >> 1, (d.height + 1) >> 1};
                const int n_items = units * ((r1 >> 1) - (r0 >> 1) + 1);
                for (int e = threadIdx.x; e < n_items; e += blockDim.x) {
                    const int v = divided(e, inv_units, units), u = e - v * units, cy = (r0 >> 1) + v;
                    uint32_t px[2][8];
                    quad_pixels(p, ((cj - lead) >> 1) + 4 * u, cy, px);
#pragma unroll
                    for (int r = 0; r < 2; r++) {
                        const int y = 2 * cy + r;
                        if (y < r0 || y > r1) continue;
                        uint4 *w = reinterpret_cast<uint4 *>(s_win + (y - r0) * wpitch + 8 * u);
                        w[0] = make_uint4(px[r][0], px[r][1], px[r][2], px[r][3]);
                        w[1] = make_uint4(px[r][4], px[r][5], px[r][6], px[r][7]);
                    }
                }
            } else {
                const int pw = d.mcus_x * d.hs * d.bs_luma;
                const bool words = (pw & 3) == 0; // (planes begin at multiples of 16)
                const int n_items = units * (r1 - r0 + 1);
                for (int e = threadIdx.x; e < n_items; e += blockDim.x) {
                    const int v = divided(e, inv_units, units), x = cj - lead + 4 * (e - v * units);
                    uint32_t px[4];
                    plain_pixels(py, pb, pr, (size_t)(r0 + v) * pw + x, min(4, img_w - x), words, px);
                    *reinterpret_cast<uint4 *>(s_win + v * wpitch + (x - cj + lead)) = make_uint4(px[0], px[1], px[2], px[3]);
                }
            }
        } else { // packed pixels: four at a time out of the aligned words that hold them
            const int n_items = units * (hi - win_lo + 1);
            for (int e = threadIdx.x; e < n_items; e += blockDim.x) {
                const int v = divided(e, inv_units, units), u = e - v * units;
                const uint8_t *p = row_ptr(win_lo + v) + 12 * u;
                const uint32_t phase = (uint32_t)(reinterpret_cast<uintptr_t>(p) & 3), bytes = phase + 3 * min(4, cw - 4 * u);
                const uint32_t *g = reinterpret_cast<const uint32_t *>(p - phase);
                uint32_t w[4];
#pragma unroll
                for (int k = 0; k < 4; k++) w[k] = 4 * k < bytes ? g[k] : 0;
#pragma unroll
                for (int k = 0; k < 3; k++) w[k] = __funnelshift_r(w[k], w[k + 1], 8 * phase);
                *reinterpret_cast<uint4 *>(s_win + v * wpitch + 4 * u) =
                    make_uint4(w[0], pick(w[0], w[1], 0x0543), pick(w[1], w[2], 0x0432), w[2] >> 8);
            }
        }
        __syncthreads();
    }
    auto window_row = [&](int y) -> const uint32_t * { return s_win + (y - win_lo) * wpitch + lead; };
    if (regime == kArea || regime == kLinear) { // (and ok)
        // OpenCV first sums every source row horizontally with the x weights, then combines those row sums with
        // the y weights; likewise for its two-tap interpolation.  A thread therefore owns two neighbouring output
        // columns for a run of consecutive output rows: the taps and weights of its columns live in registers for the
        // whole run, what a source row contributes is computed once for neighbouring output rows that share
        // it, and the columns share instructions and the loop around them.
        // Same operations in the same order as the per-pixel form, so the same bits.
        // Without a window a thread has one column: the taps come through the first-level cache, which four CTAs' shared memory leaves
        // 28 KB of, and there 32 warps hold 600 bytes of a row each, at a scale of 6, but not 1200 (64 images of
        // 1200x1400 pixels to 224x224 240 us, 304 with two columns; 400 of them 1250 and 1697; 64 of 1200x1500 to 384x384 266 and 310).
        const int run = (rows + groups - 1) / groups;
        // row_of: a row of the crop, in the window or in global memory.  A loop for either way to interpolate: in one the
        // linear way is 1 % slower (1024 images to 256x256 273 and 277 us).
        auto columns = [&](auto row_of, auto value, auto way) {
            using V = decltype(value);
            constexpr bool area = decltype(way)::value;
            const int per_row = V::width == 2 ? (out_w + 1) >> 1 : out_w;
            const uint32_t inv_per_row = V::width == 2 ? inv_pairs : inv_w;
            for (int t = threadIdx.x; t < groups * per_row; t += blockDim.x) {
                const int g = divided(t, inv_per_row, per_row), ox = V::width * (t - g * per_row);
                const bool both = V::width == 2 && ox + 1 < out_w;
                const int begin = max(y_lo, band0 + g * run + dy), end = min(y_hi, band0 + (g + 1) * run + dy);
                auto taps_of = [&](int x) { return tx[min(max(step_x * x + dx, 0), out_w - 1)]; };
                const uint4 taps = taps_of(ox), beside = taps_of(both ? ox + 1 : ox);
                OutT *o = s_out + ((begin - dy - band0) * out_w + ox) * pix_step;
                const int row_step = out_w * pix_step;
                if constexpr (area) {
                    const AreaColumns<V> pair(taps, beside);
                    int pj = -1; // source row whose horizontal sums are held
                    V row[3];
                    row[0] = row[1] = row[2] = V(0.f, 0.f);
                    for (int y = begin; y < end; y++, o += row_step) {
                        const uint4 c = ty[y];
                        const int yf = (int)(c.x & 0xffff), ye = yf + (int)(c.x >> 16) - 1;
                        // only the first source row can be the one the previous output row ended with
                        if (yf != pj) pair.across(row_of(yf), row);
                        float beta = __uint_as_float(c.y);
                        V sum[3];
#pragma unroll
                        for (int k = 0; k < 3; k++) sum[k] = mul_rn(V(beta, beta), row[k]);
                        for (int j = yf + 1; j <= ye; j++) {
                            pair.across(row_of(j), row);
                            beta = __uint_as_float(j == ye ? c.w : c.z);
#pragma unroll
                            for (int k = 0; k < 3; k++) sum[k] = add_rn(sum[k], mul_rn(V(beta, beta), row[k]));
                        }
                        pj = ye;
                        // 2^23 + the rounded value.  (The weights of an axis sum up to 1 but for rounding, so 255 is not exceeded.)
                        uint32_t v[2][3];
#pragma unroll
                        for (int k = 0; k < 3; k++) {
                            const V r = add_rn(sum[k], V(8388608.f, 8388608.f));
                            v[0][k] = __float_as_uint(r.lo());
                            v[1][k] = __float_as_uint(r.hi());
                        }
                        emit_pair(o, v, kBias, both, V::width);
                    }
                } else {
                    const LinearColumns<V> pair(taps, beside);
                    int ra = -1, rb = -1; // source rows whose interpolated values ha / hb hold
                    V ha[3], hb[3];
                    ha[0] = ha[1] = ha[2] = hb[0] = hb[1] = hb[2] = V(0.f, 0.f);
                    for (int y = begin; y < end; y++, o += row_step) {
                        const uint4 c = ty[y];
                        const int r0 = (int)c.x, r1 = (int)c.y;
                        // rows only move forward: the upper row is the former upper or lower one, or both are new
                        if (r0 != ra) {
                            if (r0 == rb) {
#pragma unroll
                                for (int k = 0; k < 3; k++) ha[k] = hb[k];
                            } else {
                                pair.across(row_of(r0), ha);
                            }
                            ra = r0;
                        }
                        if (r1 != rb) {
                            pair.across(row_of(r1), hb);
                            rb = r1;
                        }
                        const V b0(__uint_as_float(c.z), __uint_as_float(c.z)), b1(__uint_as_float(c.w), __uint_as_float(c.w));
                        const V k0 = fma_rn(b0, V(-134217728.f, -134217728.f), V(8796093022208.f, 8796093022208.f));
                        const V k1 = fma_rn(b1, V(-134217728.f, -134217728.f), V(8796093022208.f, 8796093022208.f));
                        uint32_t v[2][3];
#pragma unroll
                        for (int k = 0; k < 3; k++) {
                            const V upper = fma_rd(b0, ha[k], k0), lower = fma_rd(b1, hb[k], k1);
                            v[0][k] = blended(upper.lo(), lower.lo());
                            v[1][k] = blended(upper.hi(), lower.hi());
                        }
                        emit_pair(o, v, 0, both, V::width);
                    }
                }
            }
        };
        auto both_ways = [&](auto row_of, auto value) {
            if (regime == kArea)
                columns(row_of, value, std::true_type{});
            else
                columns(row_of, value, std::false_type{});
        };
        if (window)
            both_ways(window_row, Two());
        else if constexpr (kPlain)
            both_ways(row_ptr, One());
        if (!flips_only) { // what is filled, over it
            __syncthreads();
            for (int pix = threadIdx.x; pix < npix; pix += blockDim.x) {
                const int r = divided(pix, inv_w, out_w), ox = pix - r * out_w;
                int y, x, val[3];
                if (trace(band0 + r, ox, y, x, val)) emit(s_out + pix * pix_step, val[0], val[1], val[2]);
            }
        }
    } else {
        for (int pix = threadIdx.x; pix < npix; pix += blockDim.x) {
            const int r = divided(pix, inv_w, out_w), ox = pix - r * out_w;
            int y, x, val[3] = {0, 0, 0};
            if (!trace(band0 + r, ox, y, x, val) && ok) {
                if (regime == kCopy) {
                    const uint8_t *p = row_ptr(y) + x * 3;
                    val[0] = p[0];
                    val[1] = p[1];
                    val[2] = p[2];
                } else if (regime == kInteger) {
                    int s0 = 0, s1 = 0, s2 = 0;
                    for (int j = 0; j < isy; j++) {
                        const uint8_t *p = row_ptr(y * isy + j) + (x * isx) * 3;
                        for (int k = 0; k < isx; k++, p += 3) {
                            s0 += p[0];
                            s1 += p[1];
                            s2 += p[2];
                        }
                    }
                    if (isx == 2 && isy == 2) {
                        val[0] = (s0 + 2) >> 2;
                        val[1] = (s1 + 2) >> 2;
                        val[2] = (s2 + 2) >> 2;
                    } else {
                        const float inv = __fdiv_rn(1.f, (float)(isx * isy));
                        val[0] = sat_round(__fmul_rn((float)s0, inv));
                        val[1] = sat_round(__fmul_rn((float)s1, inv));
                        val[2] = sat_round(__fmul_rn((float)s2, inv));
                    }
                }
            }
            emit(s_out + pix * pix_step, val[0], val[1], val[2]);
        }
    }
    __syncthreads();

    // ---- coalesced copy-out: one contiguous run (NHWC) or one per channel (NCHW), 16-byte vectors
    const size_t plane = (size_t)out_h * out_w;
    const int runs = planar ? 3 : 1;
    const int run_elems = planar ? npix : npix * 3;
    for (int c = 0; c < runs; c++) {
        OutT *dst = planar ? out + ((size_t)i * 3 + c) * plane + (size_t)band0 * out_w
                           : out + ((size_t)i * plane + (size_t)band0 * out_w) * 3;
        const OutT *srcp = s_out + (size_t)c * run_elems;
        constexpr int kVec = 16 / sizeof(OutT);
        const bool aligned = ((reinterpret_cast<uintptr_t>(dst) | reinterpret_cast<uintptr_t>(srcp)) & 15) == 0;
        const int nvec = aligned ? run_elems / kVec : 0;
        for (int k = threadIdx.x; k < nvec; k += blockDim.x)
            reinterpret_cast<uint4 *>(dst)[k] = reinterpret_cast<const uint4 *>(srcp)[k];
        for (int k = nvec * kVec + threadIdx.x; k < run_elems; k += blockDim.x) dst[k] = srcp[k];
    }
    __syncthreads(); // the tile is rewritten by the next band
    }
}

static size_t value_size(int out_kind) { return out_kind == kOutU8 ? 1 : (out_kind == kOutF16Nhwc || out_kind == kOutF16Nchw ? 2 : 4); }

ResizeShape resize_shape(int n, int out_h, int out_w, int out_kind) {
    const size_t elem = value_size(out_kind);
    ResizeShape s{};
    const size_t fixed = 768 * elem + sizeof(uint4) * ((size_t)out_w + out_h), row = (size_t)out_w * 3 * elem;
    // without a window: about 2048 pixels per band
    int band = (2048 + out_w - 1) / out_w;
    if (band > out_h) band = out_h;
    while (band > 1 && fixed + band * row > 200 * 1024) band /= 2;
    s.band = band;
    // With one: as many rows (up to 5120 pixels) as fit, with their window, in a quarter of the SM's shared memory; four
    // resident CTAs of 256 threads is what the registers allow.  Small batches get bands enough for all SMs.
    s.max_band = (5120 + out_w - 1) / out_w;
    const int64_t spread = (int64_t)out_h * n / (148 * 4);
    if (spread < s.max_band) s.max_band = spread < 4 ? 4 : (int)spread;
    if (s.max_band > out_h) s.max_band = out_h;
    const size_t quarter = (227 * 1024) / 4 - 1024;
    s.room = quarter > fixed ? (quarter - fixed) & ~(size_t)15 : 0;
    const size_t tile = (band * row + 15) & ~(size_t)15;
    s.smem = fixed + (s.room > tile ? s.room : tile) + 16; // (a zero weight's pixel lies up to one behind the window)
    return s;
}

constexpr int kWaves = 8, kWindowedWaves = 4;

ResizeItems::ResizeItems(int n, int out_h, int out_w, int out_kind)
    : out_h_(out_h), out_w_(out_w), most_((kWaves * 148 * 4 + n - 1) / n), most_windowed_((kWindowedWaves * 148 * 4 + n - 1) / n), tile_row_((size_t)out_w * 3 * value_size(out_kind)),
      shape_(resize_shape(n, out_h, out_w, out_kind)), groups_(shape_.max_band + 1, 0) {}

// The column paths deal a band's rows to this many runs per pair of columns (without a window: per column), so that the
// (pair, run) items fill the CTA's 256 threads evenly, with runs of at least 2 rows (3).
int ResizeItems::groups(int band, bool window) {
    uint8_t &known = window ? groups_[band] : plain_groups_;
    if (known) return known;
    const int width = window ? 2 : 1, per_row = (out_w_ + width - 1) / width;
    int groups = 1, best = 0;
    for (int g = 1; g <= 4 * width && (band + g - 1) / g >= 4 - width; g++) {
        const int items = g * per_row, use = items * 256 / ((items + 255) / 256 * 256);
        if (use > best) {
            best = use;
            groups = g;
        }
    }
    known = (uint8_t)groups;
    return groups;
}

ResizeItem ResizeItems::make(const int32_t *box, int img_h, int img_w, Fuse fuse) {
    ResizeItem item{};
    const int ch = box[2], cw = box[3];
    if (!(ch > 0 && cw > 0 && box[0] >= 0 && box[1] >= 0 && box[0] + ch <= img_h && box[1] + cw <= img_w)) return item;
    const Scaling sc = scaling_of(ch, cw, out_h_, out_w_);
    item.inv_x = sc.inv_x;
    item.inv_y = sc.inv_y;
    item.sc_x = sc.sc_x;
    item.sc_y = sc.sc_y;
    item.regime = sc.regime;
    item.isx = sc.isx;
    item.isy = sc.isy;
    if (sc.regime == kArea || sc.regime == kLinear) item.window = window_band(cw, sc.sc_y, tile_row_, shape_);
    if (item.window && fuse != kPacked) item.lead = fuse == kFuseQuad ? box[1] & 7 : box[1] & 3; // a unit begins at a multiple of its width
    item.units = item.window && fuse == kFuseQuad ? (item.lead + cw + 7) / 8 : (item.lead + cw + 3) / 4;
    item.inv_units = inverse(item.units);
    const int band = item.window ? item.window : shape_.band, bands = (out_h_ + band - 1) / band;
    item.groups = groups(band, item.window != 0);
    if (bands > bands_) bands_ = bands;
    windowed_ = windowed_ && item.window != 0;
    plain_ = plain_ || (item.window == 0 && (sc.regime == kArea || sc.regime == kLinear));
    return item;
}

template <typename OutT>
static void launch_typed(const ResizeSource &src, int n, const int32_t *params, int n_params, const ResizeItem *items, const OpList &ops,
                         int resize, int out_h, int out_w, int planar, const ResizeShape &shape, int bands, bool plain, const void *lut, void *out,
                         const int32_t *status, const SmallCopies &small, bool early, cudaStream_t stream) {
    auto run = [&](auto kern) {
        if (shape.smem > 48 * 1024) cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)shape.smem);
        dim3 grid(bands, n);
        launch(early, grid, 256, shape.smem, stream, kern, src, params, n_params, items, ops, resize, out_h, out_w, shape, planar, (const OutT *)lut, (OutT *)out,
               status, small);
    };
    if (plain)
        run(resize_augment_kernel<OutT, true>);
    else
        run(resize_augment_kernel<OutT, false>);
}

void launch_resize_augment(const ResizeSource &src, int n, const int32_t *params, int n_params, const ResizeItem *items,
                           const OpList &ops, int resize, int out_h, int out_w, int out_kind, int bands, bool plain,
                           const void *lut, void *out, const int32_t *status, const SmallCopies &small, bool early, cudaStream_t stream) {
    if (n <= 0) return;
    const int planar = out_kind == kOutF16Nchw || out_kind == kOutF32Nchw;
    const ResizeShape shape = resize_shape(n, out_h, out_w, out_kind);
    if (out_kind == kOutU8)
        launch_typed<uint8_t>(src, n, params, n_params, items, ops, resize, out_h, out_w, 0, shape, bands, plain, nullptr, out, status, small, early, stream);
    else if (out_kind == kOutF16Nhwc || out_kind == kOutF16Nchw)
        launch_typed<uint16_t>(src, n, params, n_params, items, ops, resize, out_h, out_w, planar, shape, bands, plain, lut, out, status, small, early, stream);
    else
        launch_typed<uint32_t>(src, n, params, n_params, items, ops, resize, out_h, out_w, planar, shape, bands, plain, lut, out, status, small, early, stream);
}

} // namespace ffcvb
