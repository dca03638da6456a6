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
template <int k>
__device__ __forceinline__ float biased(uint32_t px) {
    return __uint_as_float(pick(px, 0x4B000000u, 0x7440u | k));
}
// sat_round of a value that is not negative
__device__ __forceinline__ int round_byte(float v) { return (int)(__float_as_uint(__fadd_rn(fminf(v, 255.f), 8388608.f)) & 0xff); }

// A pixel of a row: of the window's words, or of packed bytes.
__device__ __forceinline__ uint32_t pixel(const uint32_t *row, int x) { return row[x]; }
__device__ __forceinline__ uint32_t pixel(const uint8_t *row, int x) {
    return (uint32_t)row[3 * x] | (uint32_t)row[3 * x + 1] << 8 | (uint32_t)row[3 * x + 2] << 16;
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

// Two floats per register pair, and two operations per instruction.
struct Two {
    unsigned long long v;
    __device__ __forceinline__ Two() {}
    __device__ __forceinline__ Two(float lo, float hi) { asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "f"(lo), "f"(hi)); }
    __device__ __forceinline__ float lo() const { return half(0); }
    __device__ __forceinline__ float hi() const { return half(1); }
    __device__ __forceinline__ float half(int k) const {
        float a, b;
        asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
        return k ? b : a;
    }
};
__device__ __forceinline__ Two fma_rn(Two a, Two b, Two c) {
    Two r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
    return r;
}
__device__ __forceinline__ Two fma_rd(Two a, Two b, Two c) {
    Two r;
    asm("fma.rm.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
    return r;
}
__device__ __forceinline__ Two add_rn(Two a, Two b) {
    Two r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
// (as a sum with zero: a product that is added next may be contracted into one rounding, which must not happen)
__device__ __forceinline__ Two mul_rn(Two a, Two b) { return fma_rn(a, b, Two(0.f, 0.f)); }

// A column's horizontal sums: first tap, the whole cells between, last tap, rounded after every operation.
// fma(2^23 + v, w, -2^23 * w) is the correctly rounded v * w, exactly what the multiplication of the
// converted value gives (2^23 * w is exact).  Red and green share their instructions.
struct AreaColumn {
    int first, last;
    float w_first, w_mid, w_last;
    __device__ __forceinline__ explicit AreaColumn(uint4 t) {
        first = (int)(t.x & 0xffff);
        last = first + (int)(t.x >> 16) - 1;
        w_first = __uint_as_float(t.y);
        w_mid = __uint_as_float(t.z);
        w_last = __uint_as_float(t.w);
    }
    static __device__ __forceinline__ void tap(uint32_t px, float w, Two &rg, float &b) {
        const float c = -8388608.0f * w;
        rg = fma_rn(Two(biased<0>(px), biased<1>(px)), Two(w, w), Two(c, c));
        b = __fmaf_rn(biased<2>(px), w, c);
    }
    template <class Row>
    __device__ __forceinline__ void across(Row row, Two &rg, float &b) const {
        Two rg2;
        float b2;
        tap(pixel(row, first), w_first, rg, b);
        for (int k = first + 1; k < last; k++) {
            tap(pixel(row, k), w_mid, rg2, b2);
            rg = add_rn(rg, rg2);
            b = __fadd_rn(b, b2);
        }
        tap(pixel(row, last), w_last, rg2, b2);
        rg = add_rn(rg, rg2);
        b = __fadd_rn(b, b2);
    }
};

// OpenCV's fixed-point bilinear, in floating point whose roundings do what the shifts do: with S the two taps'
// weighted sum (an exact integer below 2^20), 2^27 + S rounded down is 2^27 + 16 * (S >> 4), and
// fma(b, that, 2^43 - 2^27 * b) rounded down is 2^43 + 2^20 * (b * (S >> 4) >> 16), the product of the integers
// in the low bits of its mantissa.  The two taps of a channel share their instruction, and so do the two rows.
struct LinearColumn {
    int x0, x1;
    Two w, c;
    __device__ __forceinline__ explicit LinearColumn(uint4 t) {
        x0 = (int)t.x;
        x1 = (int)t.y;
        w = Two(__uint_as_float(t.z), __uint_as_float(t.w));
        c = mul_rn(w, Two(-8388608.0f, -8388608.0f));
    }
    template <class Row>
    __device__ __forceinline__ void across(Row row, float (&h)[3]) const {
        const uint32_t p = pixel(row, x0), q = pixel(row, x1);
        auto one = [&](float a, float b) {
            const Two s = fma_rn(Two(a, b), w, c);
            return __fadd_rd(__fadd_rn(s.lo(), s.hi()), 134217728.f);
        };
        h[0] = one(biased<0>(p), biased<0>(q));
        h[1] = one(biased<1>(p), biased<1>(q));
        h[2] = one(biased<2>(p), biased<2>(q));
    }
};
// (The weights' sum is at most 2049, so 255 is not exceeded.)
__device__ __forceinline__ int blend_rows(float upper, float lower, Two b, Two k) {
    const Two u = fma_rd(b, Two(upper, lower), k);
    return (int)((__float_as_uint(u.lo()) + __float_as_uint(u.hi()) + 2u - 2u * (170u << 23)) >> 2);
}

// The column paths deal a band's rows to this many runs per column, so that the (column, run) items fill the
// CTA's 256 threads evenly, with runs of at least 3 rows.
__device__ __forceinline__ int row_groups(int out_w, int band) {
    int groups = 1, best = 0;
    for (int g = 1; g <= 4 && (band + g - 1) / g >= 3; g++) {
        const int items = g * out_w, use = items * 256 / ((items + 255) / 256 * 256);
        if (use > best) {
            best = use;
            groups = g;
        }
    }
    return groups;
}

// a / n for a, n < 2^16, inv_n = ceil(2^32 / n)
__device__ __forceinline__ int divided(uint32_t a, uint32_t inv_n, int n) { return n == 1 ? (int)a : (int)__umulhi(a, inv_n); }
__device__ __forceinline__ uint32_t inverse(int n) { return (uint32_t)((0x100000000ull + n - 1) / n); }

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

template <typename OutT>
__global__ void __launch_bounds__(256, 4)
resize_augment_kernel(const __grid_constant__ ResizeSource src, const int32_t *__restrict__ params, int n_params,
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
    if (!kU8)
        for (int k = threadIdx.x; k < 768; k += blockDim.x) s_lut[(k % 3) * 256 + k / 3] = lut[k]; // per channel

    // ---- where the sample's pixels are
    const uint8_t *base;
    int stride, row0 = 0, col0 = 0, img_h, img_w;
    // rows of a gathered crop box start at their source alignment inside their slot (raw_skew)
    uint32_t skew_base = 0, skew_pitch = 0;
    bool skew = false;
    bool ok = true;
    int fuse = 0; // output rows per band of a sample whose planes are converted here
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
            fuse = d.fuse_rows;
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

    // The scale factors (four double-precision divisions) are worked out by one thread, and so are the
    // conversion units of a window row and the number of output rows whose source rows fit the window.
    __shared__ Scaling s_scaling;
    __shared__ int s_window, s_units, s_lead, s_groups;
    __shared__ uint32_t s_inv_units;
    if (threadIdx.x == 0 && ok) {
        s_scaling = scaling_of(ch, cw, out_h, out_w);
        const bool fits = s_scaling.regime == kArea || s_scaling.regime == kLinear;
        s_window = fuse ? fuse : (fits ? window_band(cw, s_scaling.sc_y, tile_row, shape) : 0);
        const bool quad = fuse && src.descs[i].scale_shift == 0 && src.descs[i].hs == 2;
        s_lead = fuse ? (quad ? cj & 7 : cj & 3) : 0; // a unit begins at a multiple of its width
        s_units = quad ? (s_lead + cw + 7) / 8 : (s_lead + cw + 3) / 4;
        s_inv_units = inverse(s_units);
        s_groups = row_groups(out_w, s_window ? s_window : shape.band);
    }
    __syncthreads();
    int regime = kCopy, isx = 1, isy = 1;
    const int window = ok ? s_window : 0, band_rows = window ? window : shape.band;
    const int lead = ok ? s_lead : 0, wpitch = window_pitch(cw), groups = ok ? s_groups : 1;
    uint32_t *s_win = reinterpret_cast<uint32_t *>(reinterpret_cast<unsigned char *>(s_out) + (((size_t)band_rows * tile_row + 15) & ~(size_t)15));
    const int nbands = (out_h + band_rows - 1) / band_rows;
    if ((int)blockIdx.x >= nbands) return;
    if (ok) {
        const Scaling &sc = s_scaling;
        regime = sc.regime;
        isx = sc.isx;
        isy = sc.isy;
        if (regime == kArea || regime == kLinear) {
            // x taps of every column, y taps of the rows of the crop that this CTA needs
            const int my_bands = (nbands - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x;
            for (int e = threadIdx.x; e < out_w + my_bands * band_rows; e += blockDim.x) {
                const bool column = e < out_w;
                const int k = e - out_w, b = column ? 0 : k / band_rows;
                const int at = column ? e : ((int)blockIdx.x + b * (int)gridDim.x) * band_rows + (k - b * band_rows) + dy;
                if (at < 0 || at >= (column ? out_w : out_h)) continue;
                const int ssize = column ? cw : ch;
                const double inv = column ? sc.inv_x : sc.inv_y, scale = column ? sc.sc_x : sc.sc_y;
                (column ? tx : ty)[at] = regime == kArea ? make_area_taps(at, ssize, scale) : make_linear_taps(at, ssize, inv, scale, column);
            }
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
    const uint32_t inv_w = inverse(out_w);
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
        const int units = s_units;
        const uint32_t inv_units = s_inv_units;
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
        // the y weights; likewise for its two-tap interpolation.  A thread therefore owns one output column for
        // a run of consecutive output rows: the taps and weights of its column live in registers for the whole
        // run, and what a source row contributes is computed once for neighbouring output rows that share it.
        // Same operations in the same order as the per-pixel form, so the same bits.
        const int run = (rows + groups - 1) / groups;
        // row_of: a row of the crop, in the window or in global memory
        auto columns = [&](auto row_of) {
            for (int t = threadIdx.x; t < groups * out_w; t += blockDim.x) {
                const int g = divided(t, inv_w, out_w), ox = t - g * out_w;
                const int begin = max(y_lo, band0 + g * run + dy), end = min(y_hi, band0 + (g + 1) * run + dy);
                const uint4 taps = tx[min(max(step_x * ox + dx, 0), out_w - 1)];
                OutT *o = s_out + ((begin - dy - band0) * out_w + ox) * pix_step;
                const int row_step = out_w * pix_step;
                if (regime == kArea) {
                    const AreaColumn column(taps);
                    int pj = -1; // source row whose horizontal sums are held
                    Two rg(0.f, 0.f);
                    float b = 0.f;
                    for (int y = begin; y < end; y++, o += row_step) {
                        const uint4 c = ty[y];
                        const int yf = (int)(c.x & 0xffff), ye = yf + (int)(c.x >> 16) - 1;
                        // only the first source row can be the one the previous output row ended with
                        if (yf != pj) column.across(row_of(yf), rg, b);
                        float beta = __uint_as_float(c.y);
                        Two sum_rg = mul_rn(Two(beta, beta), rg);
                        float sum_b = __fmul_rn(beta, b);
                        for (int j = yf + 1; j <= ye; j++) {
                            column.across(row_of(j), rg, b);
                            beta = __uint_as_float(j == ye ? c.w : c.z);
                            sum_rg = add_rn(sum_rg, mul_rn(Two(beta, beta), rg));
                            sum_b = __fadd_rn(sum_b, __fmul_rn(beta, b));
                        }
                        pj = ye;
                        emit(o, round_byte(sum_rg.lo()), round_byte(sum_rg.hi()), round_byte(sum_b));
                    }
                } else {
                    const LinearColumn column(taps);
                    int ra = -1, rb = -1; // source rows whose interpolated values ha / hb hold
                    float ha[3] = {0.f, 0.f, 0.f}, hb[3] = {0.f, 0.f, 0.f};
                    for (int y = begin; y < end; y++, o += row_step) {
                        const uint4 c = ty[y];
                        const int r0 = (int)c.x, r1 = (int)c.y;
                        // rows only move forward: the upper row is the former upper or lower one, or both are new
                        if (r0 != ra) {
                            if (r0 == rb) {
#pragma unroll
                                for (int k = 0; k < 3; k++) ha[k] = hb[k];
                            } else {
                                column.across(row_of(r0), ha);
                            }
                            ra = r0;
                        }
                        if (r1 != rb) {
                            column.across(row_of(r1), hb);
                            rb = r1;
                        }
                        const Two b(__uint_as_float(c.z), __uint_as_float(c.w));
                        const Two k = fma_rn(b, Two(-134217728.f, -134217728.f), Two(8796093022208.f, 8796093022208.f));
                        emit(o, blend_rows(ha[0], hb[0], b, k), blend_rows(ha[1], hb[1], b, k), blend_rows(ha[2], hb[2], b, k));
                    }
                }
            }
        };
        if (window)
            columns(window_row);
        else
            columns(row_ptr);
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

ResizeShape resize_shape(int n, int out_h, int out_w, int out_kind) {
    const size_t elem = out_kind == kOutU8 ? 1 : (out_kind == kOutF16Nhwc || out_kind == kOutF16Nchw ? 2 : 4);
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
    s.smem = fixed + (s.room > tile ? s.room : tile);
    return s;
}

int resize_bands(const int32_t *params, int n, int n_params, int resize, int out_h, int out_w, int out_kind) {
    const ResizeShape shape = resize_shape(n, out_h, out_w, out_kind);
    const size_t elem = out_kind == kOutU8 ? 1 : (out_kind == kOutF16Nhwc || out_kind == kOutF16Nchw ? 2 : 4), tile_row = (size_t)out_w * 3 * elem;
    const int plain = (out_h + shape.band - 1) / shape.band, most = (8 * 148 * 4 + n - 1) / n;
    int bands = 1;
    for (int i = 0; i < n && bands < most; i++) {
        const int32_t *box = params + (size_t)i * n_params;
        int mine = plain;
        if (resize && box[2] > 0 && box[3] > 0) {
            const Scaling sc = scaling_of(box[2], box[3], out_h, out_w);
            const int window = sc.regime == kArea || sc.regime == kLinear ? window_band(box[3], sc.sc_y, tile_row, shape) : 0;
            if (window) mine = (out_h + window - 1) / window;
        }
        if (mine > bands) bands = mine;
        if (!resize) break; // (all alike)
    }
    return bands < most ? bands : most;
}

template <typename OutT>
static void launch_typed(const ResizeSource &src, int n, const int32_t *params, int n_params, const OpList &ops,
                         int resize, int out_h, int out_w, int planar, const ResizeShape &shape, int bands, const void *lut, void *out,
                         const int32_t *status, const SmallCopies &small, bool early, cudaStream_t stream) {
    auto kern = resize_augment_kernel<OutT>;
    if (shape.smem > 48 * 1024) cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)shape.smem);
    dim3 grid(bands, n);
    launch(early, grid, 256, shape.smem, stream, kern, src, params, n_params, ops, resize, out_h, out_w, shape, planar, (const OutT *)lut, (OutT *)out,
           status, small);
}

void launch_resize_augment(const ResizeSource &src, int n, const int32_t *params, int n_params,
                           const OpList &ops, int resize, int out_h, int out_w, int out_kind, int bands,
                           const void *lut, void *out, const int32_t *status, const SmallCopies &small, bool early, cudaStream_t stream) {
    if (n <= 0) return;
    const int planar = out_kind == kOutF16Nchw || out_kind == kOutF32Nchw;
    const ResizeShape shape = resize_shape(n, out_h, out_w, out_kind);
    if (out_kind == kOutU8)
        launch_typed<uint8_t>(src, n, params, n_params, ops, resize, out_h, out_w, 0, shape, bands, nullptr, out, status, small, early, stream);
    else if (out_kind == kOutF16Nhwc || out_kind == kOutF16Nchw)
        launch_typed<uint16_t>(src, n, params, n_params, ops, resize, out_h, out_w, planar, shape, bands, lut, out, status, small, early, stream);
    else
        launch_typed<uint32_t>(src, n, params, n_params, ops, resize, out_h, out_w, planar, shape, bands, lut, out, status, small, early, stream);
}

} // namespace ffcvb
