// Launch wrappers of the CUDA kernels (sm_100a).  All pointers are device pointers unless noted.
#pragma once
#include <float.h>
#include <math.h>
#include <cuda_runtime.h>
#include <emmintrin.h>
#include <stdint.h>

#include <vector>

#include "types.h"

namespace ffcvb {

// Pulls samples' payloads from pinned host memory (descs[i].src_addr, read by the SMs over
// PCIe) into their places in the device blob.  Source and destination share their alignment mod 16, and the
// bytes up to the next 16-byte boundaries around a payload's place are overwritten too.  Where a piece has not arrived
// after limit_ns the samples of its CTA get host_status and their word in `status` set to kErrData, and `failed`
// (device-visible) is set.  `ranges` (device): what each of the `ctas` CTAs fetches.
constexpr int kGatherCtas = 148;
void launch_gather_payloads(ImageDesc *descs, const uint2 *ranges, int ctas, uint8_t *blob, int32_t *status, uint64_t limit_ns, int32_t *failed,
                            cudaStream_t stream);
// Shares the n samples out to the CTAs, equally many lines of 128 bytes to each: ctas + 1 places (sample, and there the
// row of a crop box or the byte of a run, counted from the 16-byte word of its first byte).  Whole samples, or equal parts of
// them, in turn left the CTAs unequal loads: crop rows alone 43.9 GB/s instead of 45.0, streams of 60 KB 48.9 and 50.0,
// 24 streams 36 to 38 and 39; 512 photographs, half of them raw crops, to 224x224 through the loader 6813 and 6664 us a pass.
void gather_ranges(const ImageDesc *descs, int n, int ctas, uint2 *ranges);

// The kernels of a small batch follow one another early: each is launched as soon as all CTAs of the one before
// have begun (next_may_begin, first thing), fetches its tables and then waits in hardware for the one before to
// end (await_previous, by every CTA before it reads or writes anything of the batch's, so that the end of the last
// kernel means the end of all).  Only where the batch leaves SMs free: waiting CTAs hold shared memory and
// registers that a large batch's neighbours on other streams need.  Per call: one
// image of 100x133 pixels 103 -> 90 us, 224x256 116 -> 105, 900x1200 286 -> 275; 16 requests 144.4 -> 141.4.
constexpr int kEarlySegments = 2 * 148;
#if defined(__CUDACC__)
__device__ __forceinline__ void next_may_begin() { asm volatile("griddepcontrol.launch_dependents;"); }
__device__ __forceinline__ void await_previous() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
template <class... P, class... A>
void launch(bool early, dim3 grid, dim3 block, size_t smem, cudaStream_t stream, void (*kernel)(P...), A... args) {
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t config{};
    config.gridDim = grid;
    config.blockDim = block;
    config.dynamicSmemBytes = smem;
    config.stream = stream;
    config.attrs = &attr;
    config.numAttrs = early ? 1 : 0;
    cudaLaunchKernelEx(&config, kernel, P(args)...);
}
#endif

// Scratch and results of the entropy decode of a batch (device memory, no initialisation needed
// except `done`, which starts at zero once and is left at zero).
constexpr size_t kSegScratch = sizeof(SegMeta) + (4 + 2) * kSegSubs + 16; // bytes per segment of meta, sub_info, sub_exit and seg_dc
struct EntropyScratch {
    uint8_t *clean;      // unstuffed streams (ImageDesc::clean_off), 512 spare bytes behind them
    SegMeta *meta;       // per segment
    uint32_t *sub_info;  // per segment kSegSubs words: state at the start of a subsequence, blocks << 16
    uint16_t *sub_exit;  // per segment kSegSubs: the state that leads to at its end
    uint16_t *records;   // of every image per segment seg_lanes x rec_room, from 4 * rec_first on: where the blocks of a subsequence begin (8-byte aligned; nullptr: not kept)
    SlotTables *slots;   // per segment of the samples with ImageDesc::slots
    int32_t *seg_dc;     // per segment four words: DC value of each component before the segment
    uint32_t *done;      // per sample
    uint32_t *pos;       // per block: bit position of its first AC symbol from its image's clean_off
    int16_t *dc;         // per block: DC value, relative to seg_dc of its segment
};

// What an entropy decode works on (device lists).
struct EntropyWork {
    const uint2 *segs;     // (sample, segment) of every segment of the samples without restart markers:
    int n_guess, n_slots;  // first the n_guess of samples decoded from one guess per subsequence, then those with ImageDesc::slots
    const uint4 *parts;    // (sample, first segment, segments) of the samples of the first kind in parts that are repaired
    int n_parts, n_whole;  // on their own, see repair_parts; then those of the n_whole samples in several parts as a whole
    const int32_t *slot_images; // samples of the second kind
    int n_slot_images;
    const int32_t *restart; // samples with restart markers
    int n_restart;
    uint32_t max_subseq_bits; // of the samples decoded from one guess
    bool local_repair;     // see local_repair
    uint32_t max_raw;      // bounds a segment's raw bytes with run-up and overlap
    int max_tables;        // bounds the tables of a sample in shared memory (its distinct DC tables and twice its AC tables)
    int max_slot_segs;     // most segments of one of slot_images
    bool alike;            // all samples in segs have the same tables and layout of an MCU
    bool early() const { return n_restart == 0 && n_guess + n_slots > 0 && n_guess + n_slots <= kEarlySegments; } // see kEarlySegments
};

// Entropy decode: finds every block of the listed scans.  status[sample] is set for every listed
// sample.  index_pool / index_stats: the decode index (see DecodeIndexHeader) and two counters (images
// decoded from their entry, entries written); both may be nullptr.
void launch_entropy_decode(const ImageDesc *descs, const EntropyWork &work, const uint8_t *blob, const HuffTable *huff,
                           const EntropyScratch &scratch, int32_t *status, uint8_t *index_pool, unsigned long long *index_stats,
                           cudaStream_t stream);

// How a scan of scan_len bytes is cut into subsequences and segments.  `target_bits`: wished length of
// a subsequence, see subseq_target; bpm: blocks of an MCU; indexed: with a decode index.
struct ScanLayout {
    uint32_t subseq_bits, seg_raw, seg_warm, seg_run_up, seg_stride, seg_count, seg_lanes;
};
ScanLayout layout_scan(uint32_t scan_len, uint32_t target_bits, int bpm, bool local_repair, bool indexed);
// Where a batch leaves SMs idle, subsequences that began in the wrong state are decoded again at once, by the threads that have
// their segment's bytes: a shorter way than scan_repair_kernel, but a segment keeps its shared memory until the last one
// is right.  So too for a single image, beside which nothing runs.  One of 24 Mbit (4:4:4) / 33 Mbit (4:2:0), all kernels of
// the entropy decode: 119 and 224 us with repairs behind, 91 and 182 this way.  Batches on both sides of the line (60 Mbit), all
// kernels alone / as one of four in flight, at once and behind: 44 Mbit of 4:2:0 278 / 189 us and 284 / 174, 57 Mbit
// 312 / 210 and 339 / 200, 65 Mbit 335 / 238 and 349 / 242, 53 Mbit of 4:4:4 212 / 121 and 243 / 130.
inline bool local_repair(uint32_t target_bits, int n_images) { return target_bits < kMaxSubseqBits / 2 || n_images == 1; }
// Otherwise a scan of seg_count segments is repaired in parts: one, or, of long scans, of kRepairPart segments each, and what
// they leave at their seams by one CTA afterwards.
constexpr uint32_t kRepairPart = 32;
inline uint32_t repair_parts(uint32_t seg_count, bool local) { return local || seg_count <= 2 * kRepairPart ? 1 : (seg_count + kRepairPart - 1) / kRepairPart; }
inline uint4 repair_part(uint32_t sample, uint32_t seg_count, uint32_t parts, uint32_t k) {
    if (parts == 1) return make_uint4(sample, 0, seg_count, 0);
    const uint32_t first = k * kRepairPart, left = seg_count - first;
    return make_uint4(sample, first, left < kRepairPart ? left : kRepairPart, 0);
}
// The same for a scan decoded from every slot at once, which is done while a batch's scans leave most of
// the GPU idle otherwise: three times the work, but a chain of 4 x 512 bits instead of 6 to 10 kbit.  Kernels of a
// batch of 4:2:0 photographs, alone / as one of four in flight, from every slot and from one guess: 0.2 Mbit 77 / 23
// and 96 / 27 us, 2.3 Mbit 95 / 43 and 135 / 61, 9.5 Mbit 153 / 76 and 164 / 74, 16 Mbit 195 / 125 and 200 / 98, 25 Mbit
// 274 / 203 and 240 / 140, 38 Mbit 362 / 289 and 279 / 190.
ScanLayout layout_scan_slots(uint32_t scan_len);
constexpr uint64_t kSlotModeBits = 16u << 20; // of a batch, at most
// Subsequence length for a batch with `total_bits` of scans: long ones re-synchronise fewer times,
// short ones spread few scans over the GPU.
uint32_t subseq_target(uint64_t total_bits);

// Block decode: AC symbols, dequantisation and inverse transform of the blocks the crops need, into
// the 8-bit component planes.  `tiles` (device): one entry (sample, k) per kBlockTile blocks of a
// sample, block_tiles() of them per sample.
constexpr int kBlockTile = 128;
FFCVB_HD inline uint32_t block_tiles(const ImageDesc &d) {
    const uint32_t mcus = (uint32_t)(d.idct_col1 - d.idct_col0) * (uint32_t)(d.mcu_rows - d.idct_row0);
    const uint32_t luma = (mcus * d.hs * d.vs + 31) / 32 * 32, chroma = d.ncomp == 3 ? (mcus + 31) / 32 * 32 : 0;
    return (luma + 2 * chroma + kBlockTile - 1) / kBlockTile;
}
void launch_blocks(const ImageDesc *descs, const uint2 *tiles, int n_tiles, const HuffTable *huff, const MultTable *mult,
                   const EntropyScratch &scratch, uint8_t *planes, bool early, cudaStream_t stream);

// Chroma upsampling (triangle filter) + YCbCr->RGB into h*w*3 images in `rgb` (rows rgb_pitch
// apart).  4:2:0 images (n_quad of them) go through the quad kernel and 4:4:4 images (n_444)
// through a 2-D kernel (neither counts those with ImageDesc::fuse_rows), both converting only the crop box given by `crop_params` (row, col, h, w
// per sample; nullptr = whole image); the other n_other images go through the generic kernel.
// max_w / max_h bound the boxes in the list.  quad_tiles (device; may be nullptr): one entry
// (sample, tile x | tile y << 16) per tile of 64 x 8 chroma samples the quad kernel has to
// convert, so that it launches exactly those CTAs instead of a grid over the largest box.  whole_rows: the
// images lie in host memory or their rows do not begin on words.
void launch_color(const ImageDesc *descs, const int32_t *list, int n_list, int n_quad, int n_444, int n_other,
                  int max_w, int max_h, const uint2 *quad_tiles, int n_quad_tiles, const uint8_t *planes,
                  uint8_t *rgb, const int32_t *crop_params, int n_params, bool whole_rows, bool early, cudaStream_t stream);

// Tiles of 64 x 8 chroma samples that cover a box of bw x bh pixels wherever it begins (a thread converts four
// samples of a row, beginning at a multiple of four).
inline uint32_t quad_tiles_x(int bw) { return (uint32_t)(((bw + 1) / 2 + 6) / 4 + 15) / 16; }
inline uint32_t quad_tiles_y(int bh) { return (uint32_t)((bh + 1) / 2 + 7) / 8; }

// Scaling regime of a crop of ch x cw pixels resized to out_h x out_w, as OpenCV decides it.
enum { kCopy = 0, kInteger = 1, kArea = 2, kLinear = 3 };
struct Scaling {
    int regime, isx, isy;
    double inv_x, inv_y, sc_x, sc_y;
};
FFCVB_HD inline int nearest(double v) { // (ties to even)
#if defined(__CUDA_ARCH__)
    return __double2int_rn(v);
#else
    return _mm_cvtsd_si32(_mm_set_sd(v)); // (rint is a call)
#endif
}
FFCVB_HD inline Scaling scaling_of(int ch, int cw, int out_h, int out_w) {
    Scaling s{kCopy, 1, 1, 1, 1, 1, 1};
    if (ch != out_h || cw != out_w) {
        s.inv_x = (double)out_w / cw;
        s.inv_y = (double)out_h / ch;
        s.sc_x = 1.0 / s.inv_x;
        s.sc_y = 1.0 / s.inv_y;
        if (s.sc_x >= 1 && s.sc_y >= 1) {
            s.isx = nearest(s.sc_x);
            s.isy = nearest(s.sc_y);
            s.regime = (fabs(s.sc_x - s.isx) < DBL_EPSILON && fabs(s.sc_y - s.isy) < DBL_EPSILON) ? kInteger : kArea;
        } else {
            s.regime = kLinear;
        }
    }
    return s;
}

// How the resize kernel works on an output: rows per band without and (at most) with a window of source
// pixels; bytes of shared memory for the output tile and the window, and of all.
struct ResizeShape {
    int band, max_band;
    size_t room, smem;
};
ResizeShape resize_shape(int n, int out_h, int out_w, int out_kind);
// Pixels (words) of a row of the window, and the output rows per band whose tile (rows of tile_row bytes) and source
// rows fit in the room; 0 when so few fit that a window does not pay.  b output rows span at most
// b * sc_y + 3 source rows, of which those that two bands share are fetched twice, so more is better.
FFCVB_HD inline int window_pitch(int cw) { return (cw + 14) & ~7; }
FFCVB_HD inline int window_band(int cw, double sc_y, size_t tile_row, const ResizeShape &shape) {
    const double pitch = 4.0 * window_pitch(cw), left = (double)shape.room - 16 - 3 * pitch;
    if (left <= 0) return 0;
    const double fit = left / ((double)tile_row + sc_y * pitch);
    if (fit >= shape.max_band) return shape.max_band;
    const int b = (int)fit & ~1; // (even: most bands then begin on 16 bytes)
    return b >= 4 ? b : 0;
}

// Source of the fused kernel.
struct ResizeSource {
    const ImageDesc *descs; // per-sample descriptors, or nullptr for a uniform device batch
    const uint8_t *blob;    // raw payloads live here (descs != nullptr)
    const uint8_t *rgb;     // decoded JPEG samples live here (descs != nullptr)
    const uint8_t *planes;  // ... or here, those with ImageDesc::fuse_rows
    const uint8_t *uniform; // [n, h, w, 3] uint8 (descs == nullptr)
    int uniform_h, uniform_w;
};

// Copies from one place in device memory to another that ride along: one CTA makes them, in words of 16, 4 or 1
// bytes as the two places' alignment allows, eight per thread at most.  Up to there they cost nothing (last kernel of
// 512 images of 32x32 pixels: 12.5-13 us with up to 32 KB, 15-17 with a copy of its own behind it); a copy
// of more is a cudaMemcpyAsync (4 MB: 15 us; bytewise by the one CTA it was 4.2 ms).
struct SmallCopies {
    int n;
    uint64_t bytes[8];
    const uint8_t *src[8];
    uint8_t *dst[8];
};
constexpr uint64_t kSmallCopyWords = 2048;
FFCVB_HD inline uint32_t copy_word(const void *src, const void *dst) {
    const uint32_t low = (uint32_t)(reinterpret_cast<uintptr_t>(src) | reinterpret_cast<uintptr_t>(dst));
    return (low & 15) == 0 ? 16 : ((low & 3) == 0 ? 4 : 1);
}
FFCVB_HD inline uint64_t small_copy_words(uint64_t bytes, const void *src, const void *dst) {
    const uint32_t word = copy_word(src, dst);
    return bytes / word + (bytes % word != 0);
}

// What the resize kernel's CTAs have to know about an image, worked out on the host: four double-precision divisions,
// and integer ones, that took one thread of every CTA 11 000 cycles while the others waited (a quarter of the
// kernel: 1024 images to 160x160 pixels 212 us, 168 this way).
struct alignas(16) ResizeItem {
    double inv_x, inv_y, sc_x, sc_y; // as in Scaling
    int32_t regime, isx, isy;
    int32_t window;      // output rows per band with a window of source pixels (0: without one)
    int32_t units;       // conversion units of a window row, and ceil(2^32 / units)
    uint32_t inv_units;
    int32_t lead;        // place of the crop's first pixel in its unit
    int32_t groups;      // runs of rows that a band is dealt out in
};
// Makes them, and the CTAs per image of the kernel below: as many as the image with the most bands has, at most enough of
// them for about four waves of the GPU (148 SMs x 4 resident CTAs) when all bands have windows, eight otherwise.  More waves cost
// the set-up its amortisation, fewer leave the last one emptier.  1024 images to 160x160 / 256x256, 256 to 192x192, alone
// (and all kernels as one of four in flight): 187 (369), 289 (506), 101 us (209) with eight, 183 (352), 281 (486), 103 (201)
// with four, 187 (347), 281 (482), 109 (199) with three; 64 to 384x384 without windows 268 with eight, 285 with five.  Worth a
// look at every box: a CTA without a band costs as much set-up as one with (512 images of 32x32 pixels to 24x24: 21 us,
// 36 with a CTA for every four rows; 256 of 192x192 to 96x96: 39 and 60).
class ResizeItems {
  public:
    ResizeItems(int n, int out_h, int out_w, int out_kind);
    // The image's crop box, inside the image (else: an empty item).  Packed pixels are read as such; fuse: from
    // planes (kFuseQuad: 4:2:0, kFusePlain: of one resolution) if a window of them pays, as item.window then says.
    enum Fuse { kPacked, kFuseQuad, kFusePlain };
    ResizeItem make(const int32_t *box, int img_h, int img_w, Fuse fuse);
    int bands() const { // (none made: without a window)
        const int bands = bands_ ? bands_ : (out_h_ + shape_.band - 1) / shape_.band;
        const int most = windowed_ && bands_ ? most_windowed_ : most_;
        return bands < most ? bands : most;
    }

    bool plain() const { return plain_; } // one of them is interpolated without a window

  private:
    int groups(int band, bool window);
    int out_h_, out_w_, bands_ = 0, most_, most_windowed_;
    bool windowed_ = true; // every band so far
    bool plain_ = false;
    size_t tile_row_;
    ResizeShape shape_;
    std::vector<uint8_t> groups_; // by rows of a band, 0: not worked out
    uint8_t plain_groups_ = 0;    // of bands without a window
};

// Fused crop + INTER_AREA resize + flip/translate/cutout + lookup-table normalise.  items (device): one per image
// (may be nullptr without `resize`).
void launch_resize_augment(const ResizeSource &src, int n, const int32_t *params, int n_params, const ResizeItem *items,
                           const OpList &ops, int resize, int out_h, int out_w, int out_kind, int bands, bool plain,
                           const void *lut, void *out, const int32_t *status, const SmallCopies &small, bool early, cudaStream_t stream);

// Colour jitter kinds (ffcv/transforms/color_jitter.py).
enum { kJitterBrightness = 0, kJitterContrast = 1, kJitterSaturation = 2 };

// A chain of them on a uint8 batch of n images, optionally followed by mixup.  All pointers are device
// pointers; apply and ratio hold n entries per operation, grey_sum too (zero at the start; used
// by contrasts); lam: n mixup factors, or nullptr.
constexpr int kMaxChainOps = 8;
struct PixelChain {
    int n, n_ops;
    int kind[kMaxChainOps];
    const uint8_t *apply;
    const double *ratio;
    unsigned long long *grey_sum;
    const double *lam;
};
// src [n, pixels, 3] uint8 through the chain into dst [n, pixels, 3] of out_size bytes per value: 1
// (dst may be src unless there is mixup), or 2 / 4 with the values of the 256 x 3 table `lut`.
void launch_pixel_chain(const uint8_t *src, void *dst, int pixels, const PixelChain &chain, int out_size, const void *lut,
                        cudaStream_t stream);

// The mixup alone on images of `count` values.
void launch_mixup_bytes(const uint8_t *src, uint8_t *dst, long long count, const PixelChain &chain, cudaStream_t stream);

// Soft one-hot rows [n, classes]: lam[i] at label[i], then 1 - lam[i] at label[i - 1].
void launch_onehot_mix(float *dst, int n, int classes, const int32_t *label, const float *lam, cudaStream_t stream);

// images[i] = clamp(images[i] * one_minus_alpha + mask) for the images with apply[i] != 0.
void launch_poison(uint8_t *images, int n, long long count, const uint8_t *apply, const double *one_minus_alpha,
                   const double *mask, float lo, float hi, cudaStream_t stream);

} // namespace ffcvb
