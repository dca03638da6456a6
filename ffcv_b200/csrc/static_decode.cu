// ffcvb_imdecode_static: JPEG -> RGB decode of one image that allocates nothing.
//
// Who needs it: code that already owns all of its GPU memory and is not allowed to ask the driver
// for more while it runs -- a serving process whose memory pool was carved up at start-up, a
// plugin running inside another framework's allocator, or a latency-critical loop where a
// cudaMalloc (which can synchronise the whole device) is unacceptable.  The regular entry points grow pinned and device buffers on demand; this one
// uses a fixed scratch area that is part of the library image instead, so every GPU that loads
// the library carries kScratchBytes of it until the process exits.
//
// The decode itself is the same chain of kernels as everywhere else (entropy decode, dequantise +
// IDCT, upsample + colour conversion); only the scratch comes from the static array.
#include <cuda_runtime.h>
#include <stdio.h>
#include <string.h>

#include <algorithm>
#include <mutex>

#include "../../include/ffcv_b200.h"
#include "jpeg_header.h"
#include "kernels.h"
#include "types.h"

using namespace ffcvb;

namespace {

// Limits of one call (stated in include/ffcv_b200.h).
constexpr size_t kMaxStreamBytes = FFCVB_STATIC_MAX_STREAM_BYTES;    // compressed size
constexpr size_t kMaxPaddedSamples = FFCVB_STATIC_MAX_PADDED_PIXELS; // per component, padded to MCUs

// Scratch layout inside the static array (all offsets multiples of 256).
constexpr uint32_t kSubseqTarget = 512;                              // one image: short subsequences spread it over the GPU
constexpr size_t kMaxSegments = kMaxStreamBytes / ((kSegSubs / 2) * kSubseqTarget / 8) + 2;
constexpr size_t kMaxBlocks = 3 * kMaxPaddedSamples / 64;
constexpr size_t kMaxTiles = kMaxBlocks / kBlockTile + 4;
constexpr size_t kMetaBytes = 96 * 1024;                             // descriptor, tables, lists, status
// unstuffed bit stream: every segment with its run-up and overlap, at most 1.58 times as much
constexpr size_t kCleanBytes = kMaxStreamBytes + kMaxStreamBytes * 5 / 8 + 8192;
constexpr size_t kSegBytes = (kMaxSegments * kSegScratch + 255) / 256 * 256;
constexpr size_t kIndexBytes = (kMaxBlocks * 6 + 255) / 256 * 256;   // position and DC value of every block
// blocks' places that a decode writes down, see record_room (without room for them it decodes twice)
constexpr size_t kMaxSubseqs = kMaxStreamBytes * 8 / kSubseqTarget + kSegSubs;
constexpr size_t kRecords = 4 * kMaxBlocks + 12 * kMaxSubseqs;
constexpr size_t kRecordBytes = (kRecords * sizeof(uint16_t) + 255) / 256 * 256;
constexpr size_t kPlaneBytes = 3 * kMaxPaddedSamples + 1024;         // each plane rounded up to 256
constexpr size_t kCleanOff = kMetaBytes;
constexpr size_t kSegOff = kCleanOff + kCleanBytes;
constexpr size_t kIndexOff = kSegOff + kSegBytes;
constexpr size_t kPlaneOff = kIndexOff + kIndexBytes;
constexpr size_t kRecordOff = kPlaneOff + (kPlaneBytes + 255) / 256 * 256;
constexpr size_t kScratchBytes = kRecordOff + kRecordBytes;

static __device__ __align__(256) unsigned char g_static_scratch[kScratchBytes];

// In host code `g_static_scratch` is only a handle for the runtime, not an address a kernel can
// use; the device address is looked up once per device and cached here.
constexpr int kMaxDevices = 64;
unsigned char *g_scratch_addr[kMaxDevices] = {};
std::mutex g_setup_mutex;

struct Meta {
    ImageDesc desc;
    int32_t list[4];
    int32_t status[4]; // [0] the image's status, [1] its counter of finished segments
    uint4 part;
    uint2 segs[kMaxSegments];
    uint2 tiles[kMaxTiles];
    alignas(16) HuffTable huff[6]; // read with 16-byte loads
    alignas(16) MultTable mult[3]; // read with 16-byte loads
};
static_assert(sizeof(Meta) <= kMetaBytes, "metadata must fit its scratch region");

int reject(int code, const char *why) {
    fprintf(stderr, "ffcvb_imdecode_static: %s\n", why);
    return code;
}

} // namespace

extern "C" int ffcvb_imdecode_static(const uint8_t *jpeg_host, uint64_t jpeg_size, const uint8_t *jpeg_dev,
                                     uint32_t height, uint32_t width, uint8_t *rgb_dev, void *stream) {
    if (!jpeg_host || !jpeg_dev || !rgb_dev || jpeg_size < 4) return reject(FFCVB_E_ARG, "null or empty argument");
    if (jpeg_size > kMaxStreamBytes) return reject(FFCVB_E_LIMIT, "JPEG stream larger than FFCVB_STATIC_MAX_STREAM_BYTES");
    int dev = -1;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices)
        return reject(FFCVB_E_NODEVICE, "no current CUDA device");

    // ---- set-up, once per device (the first call on a device; make it before any stream capture)
    unsigned char *scratch;
    {
        std::lock_guard<std::mutex> g(g_setup_mutex);
        if (!g_scratch_addr[dev]) {
            void *p = nullptr;
            cudaError_t e = cudaGetSymbolAddress(&p, g_static_scratch);
            if (e != cudaSuccess || !p) return reject(FFCVB_E_CUDA, cudaGetErrorString(e));
            g_scratch_addr[dev] = static_cast<unsigned char *>(p);
        }
        scratch = g_scratch_addr[dev];
    }

    // ---- headers on the host, limits
    JpegHeader h;
    int rc = parse_jpeg_header(jpeg_host, (size_t)jpeg_size, &h);
    if (rc != 0) return reject(FFCVB_E_DECODE, "not a baseline JPEG stream this library decodes");
    if ((uint32_t)h.width != width || (uint32_t)h.height != height)
        return reject(FFCVB_E_DECODE, "stream dimensions differ from the given height and width");
    if (height > 65535 || width > 65535) return reject(FFCVB_E_LIMIT, "image larger than FFCVB_STATIC_MAX_PADDED_PIXELS");
    Meta m;
    memset(&m, 0, sizeof(m));
    ImageDesc &d = m.desc;
    d.payload_size = (uint32_t)jpeg_size;
    d.height = d.dec_height = (uint16_t)height;
    d.width = d.dec_width = (uint16_t)width;
    d.bs_luma = d.bs_chroma = 8; // full scale
    d.rgb_pitch = (uint32_t)width * 3; // the caller's buffer is packed
    d.scan_off = (uint32_t)h.scan_off;
    d.scan_len = (uint32_t)h.scan_len;
    d.ncomp = (uint8_t)h.ncomp;
    d.hs = (uint8_t)h.hs[0];
    d.vs = (uint8_t)h.vs[0];
    d.bpm = (uint8_t)(h.ncomp == 1 ? 1 : h.hs[0] * h.vs[0] + 2);
    d.mcus_x = (uint16_t)((h.width + 8 * h.hs[0] - 1) / (8 * h.hs[0]));
    d.mcus_y = (uint16_t)((h.height + 8 * h.vs[0] - 1) / (8 * h.vs[0]));
    d.restart_interval = (uint16_t)h.restart_interval;
    d.mcu_rows = d.mcus_y;
    d.idct_row0 = d.idct_col0 = 0;
    d.idct_col1 = d.mcus_x;
    d.nblocks = (uint32_t)d.bpm * d.mcus_x * d.mcus_y;
    if (d.restart_interval) { // table of restart-interval starts behind the clean stream
        d.rst_off = ((size_t)d.scan_len + 96 + 15) & ~(size_t)15;
        const size_t mcus = (size_t)d.mcus_x * d.mcus_y;
        if (d.rst_off + 4 * ((mcus + d.restart_interval - 1) / d.restart_interval + 2) > kCleanBytes)
            return reject(FFCVB_E_LIMIT, "stream with restart markers too large for the static scratch");
    }
    const size_t luma_samples = (size_t)d.mcus_x * d.hs * 8 * d.mcus_y * d.vs * 8;
    if (luma_samples > kMaxPaddedSamples)
        return reject(FFCVB_E_LIMIT, "image larger than FFCVB_STATIC_MAX_PADDED_PIXELS");
    size_t plane = 0;
    d.fast_tables = 1;
    for (int c = 0; c < h.ncomp; c++) {
        // (chroma components nearly always share their tables)
        const int t = c == 2 && h.td[2] == h.td[1] && h.ta[2] == h.ta[1] ? 1 : c;
        if (t == c) {
            build_huff_table(h.dc[h.td[c]], true, &m.huff[2 * c]);
            build_huff_table(h.ac[h.ta[c]], false, &m.huff[2 * c + 1]);
            d.n_dc_tab = (uint8_t)(c + 1);
        }
        d.dc_tab[c] = (uint8_t)t;
        d.ac_tab[c] = (uint8_t)t; // + the number of DC tables, below
        if (!m.huff[2 * t].fast_ok || !m.huff[2 * t + 1].fast_ok) d.fast_tables = 0;
        build_mult_table(h.quant[h.tq[c]], &m.mult[c]);
        d.q_tab[c] = (uint8_t)c;
        d.plane_off[c] = plane;
        plane += ((size_t)d.mcus_x * (c == 0 ? d.hs : 1) * 8 * d.mcus_y * (c == 0 ? d.vs : 1) * 8 + 255) & ~(size_t)255;
    }

    int n_segs = 0;
    if (!d.restart_interval) {
        const ScanLayout l = layout_scan(d.scan_len, kSubseqTarget, d.bpm, true, false);
        d.subseq_bits = l.subseq_bits;
        d.seg_raw = l.seg_raw;
        d.seg_warm = l.seg_warm;
        d.seg_run_up = l.seg_run_up;
        d.seg_stride = l.seg_stride;
        d.seg_count = l.seg_count;
        d.seg_lanes = l.seg_lanes;
        n_segs = (int)l.seg_count;
        if (l.seg_count > kMaxSegments || (size_t)l.seg_count * l.seg_stride + 512 > kCleanBytes)
            return reject(FFCVB_E_LIMIT, "JPEG stream too large for the static scratch");
        for (uint32_t k = 0; k < l.seg_count; k++) m.segs[k] = make_uint2(0, k);
        m.part = repair_part(0, l.seg_count, 1, 0);
        d.rec_room = (uint32_t)std::min<size_t>(record_room(l.subseq_bits, d.scan_len, d.nblocks, true), kRecords / ((size_t)l.seg_count * l.seg_lanes) / 4 * 4);
    }
    const uint32_t n_tiles = block_tiles(d);
    if (n_tiles > kMaxTiles || d.nblocks > kMaxBlocks) return reject(FFCVB_E_LIMIT, "image larger than FFCVB_STATIC_MAX_PADDED_PIXELS");
    for (uint32_t k = 0; k < n_tiles; k++) m.tiles[k] = make_uint2(0, k);

    d.n_tab = (uint8_t)(2 * d.n_dc_tab);
    for (int t = 0; t < d.n_dc_tab; t++) {
        d.tab_id[t] = (uint8_t)(2 * t);
        d.tab_id[d.n_dc_tab + t] = (uint8_t)(2 * t + 1);
    }
    for (int c = 0; c < h.ncomp; c++) d.ac_tab[c] = (uint8_t)(d.ac_tab[c] + d.n_dc_tab);

    // ---- queue the work; everything the kernels need beyond input and output lives in `scratch`
    cudaStream_t st = (cudaStream_t)stream;
    Meta *meta_dev = reinterpret_cast<Meta *>(scratch);
    // `m` lives on this thread's stack (pageable memory): for such a source the runtime stages the
    // bytes before cudaMemcpyAsync returns, so `m` may go out of scope when this call does
    if (cudaMemcpyAsync(meta_dev, &m, sizeof(m), cudaMemcpyHostToDevice, st) != cudaSuccess)
        return reject(FFCVB_E_CUDA, "copy of the descriptor failed");
    const ImageDesc *desc_dev = &meta_dev->desc;
    const int32_t *list_dev = meta_dev->list; // {0}: the only image
    EntropyScratch es{};
    es.clean = scratch + kCleanOff;
    es.seg_dc = reinterpret_cast<int32_t *>(scratch + kSegOff);
    es.sub_info = reinterpret_cast<uint32_t *>(es.seg_dc + 4 * kMaxSegments);
    es.sub_exit = reinterpret_cast<uint16_t *>(es.sub_info + kSegSubs * kMaxSegments);
    es.meta = reinterpret_cast<SegMeta *>(es.sub_exit + kSegSubs * kMaxSegments);
    es.done = reinterpret_cast<uint32_t *>(&meta_dev->status[1]);
    es.pos = reinterpret_cast<uint32_t *>(scratch + kIndexOff);
    es.dc = reinterpret_cast<int16_t *>(es.pos + kMaxBlocks);
    if (d.rec_room > 0) es.records = reinterpret_cast<uint16_t *>(scratch + kRecordOff);
    EntropyWork work{};
    work.segs = meta_dev->segs;
    work.n_guess = n_segs;
    work.restart = list_dev;
    work.parts = &meta_dev->part;
    work.n_parts = n_segs > 0 ? 1 : 0;
    work.max_subseq_bits = d.subseq_bits;
    work.local_repair = true;
    work.n_restart = d.restart_interval ? 1 : 0;
    work.max_raw = d.seg_stride; // (run-up, own bytes and overlap)
    work.max_tables = 3 * d.n_dc_tab;
    launch_entropy_decode(desc_dev, work, jpeg_dev, meta_dev->huff, es, meta_dev->status, nullptr, nullptr, st);
    launch_blocks(desc_dev, meta_dev->tiles, (int)n_tiles, meta_dev->huff, meta_dev->mult, es, scratch + kPlaneOff, work.early(), st);
    const bool quad = d.ncomp == 3 && d.hs == 2 && d.vs == 2 && (width + 1) / 2 >= 3;
    const bool full = d.ncomp == 3 && d.hs == 1 && d.vs == 1;
    launch_color(desc_dev, list_dev, 1, quad ? 1 : 0, full ? 1 : 0, (quad || full) ? 0 : 1, (int)width, (int)height,
                 nullptr, 0, scratch + kPlaneOff, rgb_dev, nullptr, 0, ((reinterpret_cast<uintptr_t>(rgb_dev) | d.rgb_pitch) & 3) != 0, work.early(), st);
    if (cudaGetLastError() != cudaSuccess) return reject(FFCVB_E_CUDA, "kernel launch failed");
    return FFCVB_OK;
}
