// Per-pixel colour and blending transforms on uint8 device batches (sm_100a): brightness,
// contrast, saturation (ffcv/transforms/color_jitter.py), image mixup (ffcv/transforms/mixup.py)
// and poisoning (ffcv/transforms/poisoning.py).
//
// The reference evaluates these in float64 under numba's fastmath, which fuses some multiply-add
// pairs; which ones decides the last bit of a truncated result.  Every operation below is written
// with explicit rounding intrinsics (__dmul_rn, __dadd_rn, __fma_rn) so that nvcc fuses nothing
// by itself and the arithmetic is, operation for operation, the one the reference's compiled code
// performs:
//   grey      = (uint8) fma(0.114, b, fma(0.587, g, 0.2989 * r))
//   brightness, contrast:  fma(t, v, (1 - t) * s)     (s = 0, or the mean of the grey image)
//   saturation:            t * v + (1 - t) * grey      (not fused)
//   mixup:                 fma(1 - t, partner, t * v)
// Colour jitter, mixup and the normalisation behind them run as one chain: a thread takes four pixels
// through every operation in registers, so a batch is read once (twice with mixup, and once more for
// every contrast, which needs the mean of the image as the operations before it leave it) and written
// once.  Bound by HBM for one operation and by the double-precision pipe for longer chains: bytes become
// doubles, and doubles bytes, by an addition of 2^52 instead of the slow conversion instructions.
#include "kernels.h"

namespace ffcvb {

namespace {

// A byte as a double: 2^52 + v has v in its low word.
__device__ __forceinline__ double to_double(uint32_t v) { return __dsub_rn(__hiloint2double(0x43300000, (int)v), 4503599627370496.0); }

// A double truncated to a byte, clamped to 0 .. 255 (|v| < 2^31): the addition rounds down, and where
// that differs from truncation the value is negative and becomes 0.
__device__ __forceinline__ uint32_t clip_u8(double v) {
    const int i = __double2loint(__dadd_rd(v, 6755399441055744.0)); // 1.5 * 2^52
    return (uint32_t)min(255, max(0, i));
}

__device__ __forceinline__ uint32_t grey_u8(const uint32_t (&v)[3]) {
    return clip_u8(__fma_rn(0.114, to_double(v[2]), __fma_rn(0.587, to_double(v[1]), __dmul_rn(0.2989, to_double(v[0])))));
}

__device__ __forceinline__ uint32_t byte_of(const uint32_t (&w)[3], int k) { return (w[k >> 2] >> (8 * (k & 3))) & 255u; }

// Four pixels (12 bytes, three aligned words) at pixel p, or one by bytes.
template <bool VEC>
__device__ __forceinline__ void load_pixels(const uint8_t *base, int p, uint32_t (&w)[3]) {
    const uint8_t *src = base + (size_t)p * 3;
    if (VEC) {
        const uint32_t *src4 = reinterpret_cast<const uint32_t *>(src);
        w[0] = src4[0];
        w[1] = src4[1];
        w[2] = src4[2];
    } else {
        w[0] = src[0] | (src[1] << 8) | (src[2] << 16);
        w[1] = w[2] = 0;
    }
}

// The same the other way.
template <bool VEC>
__device__ __forceinline__ void store_pixels(uint8_t *base, int p, const uint32_t (&r)[3]) {
    uint8_t *to = base + (size_t)p * 3;
    if (VEC) {
        uint32_t *to4 = reinterpret_cast<uint32_t *>(to);
        to4[0] = r[0];
        to4[1] = r[1];
        to4[2] = r[2];
    } else {
        to[0] = (uint8_t)r[0];
        to[1] = (uint8_t)(r[0] >> 8);
        to[2] = (uint8_t)(r[0] >> 16);
    }
}

struct ChainStep {
    double t, u, c; // factor, 1 - factor, what brightness and contrast add
    int kind;       // < 0: not applied to this image
    bool wide;      // a factor so large (or not a number) that clip_u8 needs its argument clamped first
};

__device__ __forceinline__ ChainStep chain_step(int kind, double t, unsigned long long grey_sum, int pixels) {
    ChainStep st{t, __dsub_rn(1.0, t), 0.0, kind, !(fabs(t) < 1e6)};
    if (kind == kJitterBrightness) st.c = __dmul_rn(st.u, 0.0);
    if (kind == kJitterContrast) st.c = __dmul_rn(st.u, __ddiv_rn((double)grey_sum, (double)pixels));
    return st;
}
// The operations [0, n_ops) of image `img`, worked out by the first n_ops threads of the CTA.
__device__ __forceinline__ void chain_steps(ChainStep *s, const PixelChain &chain, int n_ops, int img, int pixels, int k) {
    if (k >= n_ops) return;
    const size_t at = (size_t)k * chain.n + img;
    ChainStep st = chain_step(chain.kind[k], chain.ratio[at], chain.kind[k] == kJitterContrast ? chain.grey_sum[at] : 0, pixels);
    if (!chain.apply[at]) st.kind = -1;
    s[k] = st;
}

__device__ __forceinline__ void apply_step(const ChainStep &s, uint32_t (&v)[3]) {
    const int kind = s.kind; // (uniform over the CTA)
    if (kind < 0) return;
    const double t = s.t;
    double x[3];
    if (kind == kJitterSaturation) {
        const double l = __dmul_rn(s.u, to_double(grey_u8(v)));
#pragma unroll
        for (int c = 0; c < 3; c++) x[c] = __dadd_rn(__dmul_rn(t, to_double(v[c])), l);
    } else {
#pragma unroll
        for (int c = 0; c < 3; c++) x[c] = __fma_rn(t, to_double(v[c]), s.c);
    }
    if (s.wide)
        for (int c = 0; c < 3; c++) x[c] = fmin(fmax(x[c], -1.0), 256.0);
#pragma unroll
    for (int c = 0; c < 3; c++) v[c] = clip_u8(x[c]);
}
__device__ __forceinline__ void apply_chain(const ChainStep *s, int n_ops, uint32_t (&v)[3]) {
    for (int k = 0; k < n_ops; k++) apply_step(s[k], v);
}

// One operation alone, in place (what a pipeline with a single jitter runs): its factors in registers, images
// that it does not apply to left alone, and the conversion instructions, which have a pipe of their own that is idle
// otherwise (16 images of 1024x1024: 44 us, 51 with the additions that a chain converts by, 61 as a chain).
template <int KIND, bool VEC>
__global__ void __launch_bounds__(256)
jitter_kernel(uint8_t *__restrict__ images, int pixels, const uint8_t *__restrict__ apply, const double *__restrict__ ratio,
              const unsigned long long *__restrict__ grey_sum) {
    constexpr int per = VEC ? 4 : 1;
    const int img = blockIdx.y;
    if (!apply[img]) return;
    const ChainStep s = chain_step(KIND, ratio[img], KIND == kJitterContrast ? grey_sum[img] : 0, pixels);
    uint8_t *base = images + (size_t)img * pixels * 3;
    for (int p0 = (blockIdx.x * blockDim.x + threadIdx.x) * per; p0 < pixels; p0 += gridDim.x * blockDim.x * per) {
        uint32_t w[3], r[3] = {0, 0, 0};
        load_pixels<VEC>(base, p0, w);
#pragma unroll
        for (int q = 0; q < per; q++) {
            uint32_t v[3] = {byte_of(w, 3 * q), byte_of(w, 3 * q + 1), byte_of(w, 3 * q + 2)};
            double l = 0.0;
            if (KIND == kJitterSaturation)
                l = __dmul_rn(s.u, (double)__double2uint_rz(__fma_rn(0.114, (double)v[2], __fma_rn(0.587, (double)v[1], __dmul_rn(0.2989, (double)v[0])))));
#pragma unroll
            for (int c = 0; c < 3; c++) {
                const double x = KIND == kJitterSaturation ? __dadd_rn(__dmul_rn(s.t, (double)v[c]), l) : __fma_rn(s.t, (double)v[c], s.c);
                v[c] = __double2uint_rz(fmin(fmax(x, 0.0), 255.0));
            }
#pragma unroll
            for (int c = 0; c < 3; c++) r[(3 * q + c) >> 2] |= v[c] << (8 * ((3 * q + c) & 3));
        }
        store_pixels<VEC>(base, p0, r);
    }
}

// One CTA column per image.  With MIX the image before it in the batch (the last one, for the first)
// takes the same chain and is blended in.  OutT: bytes, or the bits of the table's floats.
template <typename OutT, bool VEC, bool MIX>
__global__ void __launch_bounds__(256)
chain_kernel(const uint8_t *src, OutT *dst, int pixels, const __grid_constant__ PixelChain chain, const OutT *__restrict__ lut) {
    constexpr int per = VEC ? 4 : 1;
    __shared__ ChainStep s_steps[2][kMaxChainOps];
    __shared__ OutT s_lut[sizeof(OutT) == 1 ? 1 : 768]; // per channel
    const int img = blockIdx.y, partner = img == 0 ? chain.n - 1 : img - 1;
    chain_steps(s_steps[0], chain, chain.n_ops, img, pixels, threadIdx.x);
    if (MIX && threadIdx.x >= 32) chain_steps(s_steps[1], chain, chain.n_ops, partner, pixels, threadIdx.x - 32);
    if constexpr (sizeof(OutT) > 1)
        for (int k = threadIdx.x; k < 768; k += blockDim.x) s_lut[(k % 3) * 256 + k / 3] = lut[k];
    __syncthreads();
    const double lam = MIX ? chain.lam[img] : 1.0, rest = __dsub_rn(1.0, lam);
    const uint8_t *a = src + (size_t)img * pixels * 3, *b = src + (size_t)partner * pixels * 3;
    OutT *o = dst + (size_t)img * pixels * 3;
    for (int p0 = (blockIdx.x * blockDim.x + threadIdx.x) * per; p0 < pixels; p0 += gridDim.x * blockDim.x * per) {
        uint32_t w[3], x[3] = {0, 0, 0}, r[3] = {0, 0, 0};
        load_pixels<VEC>(a, p0, w);
        if (MIX) load_pixels<VEC>(b, p0, x);
        OutT out[3 * per];
#pragma unroll
        for (int q = 0; q < per; q++) {
            uint32_t v[3] = {byte_of(w, 3 * q), byte_of(w, 3 * q + 1), byte_of(w, 3 * q + 2)};
            apply_chain(s_steps[0], chain.n_ops, v);
            if (MIX) {
                uint32_t y[3] = {byte_of(x, 3 * q), byte_of(x, 3 * q + 1), byte_of(x, 3 * q + 2)};
                apply_chain(s_steps[1], chain.n_ops, y);
#pragma unroll
                for (int c = 0; c < 3; c++) v[c] = clip_u8(__fma_rn(rest, to_double(y[c]), __dmul_rn(lam, to_double(v[c]))));
            }
#pragma unroll
            for (int c = 0; c < 3; c++) {
                const int k = 3 * q + c;
                if constexpr (sizeof(OutT) == 1)
                    r[k >> 2] |= v[c] << (8 * (k & 3));
                else
                    out[k] = s_lut[c * 256 + v[c]];
            }
        }
        OutT *to = o + (size_t)p0 * 3;
        if constexpr (sizeof(OutT) == 1) {
            store_pixels<VEC>(o, p0, r);
        } else if (VEC) { // (12 values from a multiple of 12 on: 8-byte pieces are aligned)
#pragma unroll
            for (int k = 0; k < (int)(12 * sizeof(OutT) / 8); k++) {
                uint2 piece;
                if constexpr (sizeof(OutT) == 2)
                    piece = make_uint2(out[4 * k] | (uint32_t)out[4 * k + 1] << 16, out[4 * k + 2] | (uint32_t)out[4 * k + 3] << 16);
                else
                    piece = make_uint2(out[2 * k], out[2 * k + 1]);
                reinterpret_cast<uint2 *>(to)[k] = piece;
            }
        } else {
#pragma unroll
            for (int k = 0; k < 3; k++) to[k] = out[k];
        }
    }
}

// Sum of the (truncated) grey values, as the operations before operation `upto` leave them, of every
// image that operation (a contrast) applies to.  Integer sums, so the order of the additions does not
// matter.
template <bool VEC>
__global__ void __launch_bounds__(256)
grey_sum_kernel(const uint8_t *__restrict__ images, int pixels, const __grid_constant__ PixelChain chain, int upto) {
    constexpr int per = VEC ? 4 : 1;
    __shared__ ChainStep s_steps[kMaxChainOps];
    const int img = blockIdx.y;
    const size_t at = (size_t)upto * chain.n + img;
    if (!chain.apply[at]) return;
    chain_steps(s_steps, chain, upto, img, pixels, threadIdx.x);
    __syncthreads();
    const uint8_t *base = images + (size_t)img * pixels * 3;
    unsigned int acc = 0; // at most 2^31 / 255 pixels per thread
    for (int p0 = (blockIdx.x * blockDim.x + threadIdx.x) * per; p0 < pixels; p0 += gridDim.x * blockDim.x * per) {
        uint32_t w[3];
        load_pixels<VEC>(base, p0, w);
#pragma unroll
        for (int q = 0; q < per; q++) {
            uint32_t v[3] = {byte_of(w, 3 * q), byte_of(w, 3 * q + 1), byte_of(w, 3 * q + 2)};
            apply_chain(s_steps, upto, v);
            acc += grey_u8(v);
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, o);
    __shared__ unsigned int s_part[8];
    if ((threadIdx.x & 31) == 0) s_part[threadIdx.x >> 5] = acc;
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned long long total = 0;
        for (int k = 0; k < (int)(blockDim.x >> 5); k++) total += s_part[k];
        atomicAdd(&chain.grey_sum[at], total);
    }
}

// Mixup of images whose values do not group into pixels.
__global__ void __launch_bounds__(256)
mixup_bytes_kernel(const uint8_t *__restrict__ src, uint8_t *__restrict__ dst, long long count, const __grid_constant__ PixelChain chain) {
    const int img = blockIdx.y, partner = img == 0 ? chain.n - 1 : img - 1;
    const double lam = chain.lam[img], rest = __dsub_rn(1.0, lam);
    const uint8_t *a = src + (size_t)img * count, *b = src + (size_t)partner * count;
    for (long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x; k < count; k += (long long)gridDim.x * blockDim.x)
        dst[(size_t)img * count + k] = (uint8_t)clip_u8(__fma_rn(rest, to_double(b[k]), __dmul_rn(lam, to_double(a[k]))));
}

// Soft labels of mixup: row i holds lam[i] at label i and 1 - lam[i] at the label of the sample before
// it (which wins where the two are the same).
__global__ void __launch_bounds__(256)
onehot_mix_kernel(float *__restrict__ dst, int n, int classes, const int32_t *__restrict__ label, const float *__restrict__ lam) {
    const int i = blockIdx.x, l0 = label[i], l1 = label[i == 0 ? n - 1 : i - 1];
    const float a = lam[i], b = __fadd_rn(-a, 1.0f);
    for (int c = threadIdx.x; c < classes; c += blockDim.x) dst[(size_t)i * classes + c] = c == l1 ? b : (c == l0 ? a : 0.0f);
}

// Poison: float32 scratch value per element, two statements that each round a float64 result to
// float32, clamp, truncate (ffcv/transforms/poisoning.py:52-58).
__global__ void __launch_bounds__(256)
poison_kernel(uint8_t *__restrict__ images, long long count, const uint8_t *__restrict__ apply,
              const double *__restrict__ one_minus_alpha, const double *__restrict__ mask, float lo, float hi) {
    const int img = blockIdx.y;
    if (!apply[img]) return;
    uint8_t *p = images + (size_t)img * count;
    for (long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x; k < count;
         k += (long long)gridDim.x * blockDim.x) {
        float t = (float)p[k];
        t = __double2float_rn(__dmul_rn((double)t, one_minus_alpha[k]));
        t = __double2float_rn(__dadd_rn((double)t, mask[k]));
        t = fmaxf(t, lo);
        t = fminf(t, hi);
        p[k] = (uint8_t)__float2uint_rz(t);
    }
}

int blocks_for(long long items, int per_block) {
    long long b = (items + per_block - 1) / per_block;
    if (b < 1) b = 1;
    if (b > 148 * 8) b = 148 * 8; // grid-stride beyond eight CTAs per SM
    return (int)b;
}

} // namespace

void launch_pixel_chain(const uint8_t *src, void *dst, int pixels, const PixelChain &chain, int out_size, const void *lut,
                        cudaStream_t stream) {
    const bool vec = pixels % 4 == 0 && ((reinterpret_cast<uintptr_t>(src) & 3) | (reinterpret_cast<uintptr_t>(dst) & (out_size == 1 ? 3 : 7))) == 0;
    // a few passes per thread: what a CTA sets up serves more pixels
    const dim3 grid(blocks_for(pixels / (vec ? 4 : 1), 256 * 2), chain.n);
    for (int k = 0; k < chain.n_ops; k++)
        if (chain.kind[k] == kJitterContrast) {
            const dim3 sums(blocks_for(pixels / (vec ? 4 : 1), 256 * 4), chain.n);
            if (vec)
                grey_sum_kernel<true><<<sums, 256, 0, stream>>>(src, pixels, chain, k);
            else
                grey_sum_kernel<false><<<sums, 256, 0, stream>>>(src, pixels, chain, k);
        }
    if (chain.n_ops == 1 && out_size == 1 && !chain.lam && src == dst) {
        const dim3 all(blocks_for(pixels / (vec ? 4 : 1), 256), chain.n);
        auto one = [&](auto kernel) { kernel<<<all, 256, 0, stream>>>((uint8_t *)dst, pixels, chain.apply, chain.ratio, chain.grey_sum); };
        if (chain.kind[0] == kJitterBrightness)
            one(vec ? jitter_kernel<kJitterBrightness, true> : jitter_kernel<kJitterBrightness, false>);
        else if (chain.kind[0] == kJitterContrast)
            one(vec ? jitter_kernel<kJitterContrast, true> : jitter_kernel<kJitterContrast, false>);
        else
            one(vec ? jitter_kernel<kJitterSaturation, true> : jitter_kernel<kJitterSaturation, false>);
        return;
    }
    auto run = [&](auto zero) {
        using OutT = decltype(zero);
        auto *out = static_cast<OutT *>(dst);
        auto *table = static_cast<const OutT *>(lut);
        if (vec && chain.lam)
            chain_kernel<OutT, true, true><<<grid, 256, 0, stream>>>(src, out, pixels, chain, table);
        else if (vec)
            chain_kernel<OutT, true, false><<<grid, 256, 0, stream>>>(src, out, pixels, chain, table);
        else if (chain.lam)
            chain_kernel<OutT, false, true><<<grid, 256, 0, stream>>>(src, out, pixels, chain, table);
        else
            chain_kernel<OutT, false, false><<<grid, 256, 0, stream>>>(src, out, pixels, chain, table);
    };
    if (out_size == 1)
        run(uint8_t{});
    else if (out_size == 2)
        run(uint16_t{});
    else
        run(uint32_t{});
}

void launch_mixup_bytes(const uint8_t *src, uint8_t *dst, long long count, const PixelChain &chain, cudaStream_t stream) {
    mixup_bytes_kernel<<<dim3(blocks_for(count, 256), chain.n), 256, 0, stream>>>(src, dst, count, chain);
}

void launch_onehot_mix(float *dst, int n, int classes, const int32_t *label, const float *lam, cudaStream_t stream) {
    onehot_mix_kernel<<<n, 256, 0, stream>>>(dst, n, classes, label, lam);
}

void launch_poison(uint8_t *images, int n, long long count, const uint8_t *apply, const double *one_minus_alpha,
                   const double *mask, float lo, float hi, cudaStream_t stream) {
    poison_kernel<<<dim3(blocks_for(count, 256), n), 256, 0, stream>>>(images, count, apply, one_minus_alpha, mask,
                                                                      lo, hi);
}

} // namespace ffcvb
