// Structures shared by the host staging code and the CUDA kernels.  A staged batch is one
// contiguous blob, identical in pinned host memory and in HBM:
//   [BatchHeader][ImageDesc x n][HuffTable x n_huff][MultTable x n_mult][params int32][payloads]
// so one host->device copy moves everything a batch needs.
#pragma once
#include <stdint.h>

namespace ffcvb {

constexpr int kMaxComponents = 3;
constexpr int kPayloadAlign = 16;

// A scan is entropy-decoded in segments of up to kSegSubs subsequences, a thread each.  kSegOverlap raw
// bytes behind a segment are unstuffed with it, so that a block that begins inside can be read to
// its end (63 symbols of at most 26 bits = 205 bytes, twice that when every second byte is stuffing).
constexpr int kSegSubs = 128;
constexpr int kSegOverlap = 512;
constexpr int kMaxSubseqBits = 2560; // longest subsequence: bounds a segment's shared memory
static_assert(kSegSubs * kMaxSubseqBits + 8 * kSegOverlap + 4096 < 1 << 24, "a position inside a segment has 24 bits");
// Few scans are decoded from every possible block slot at once (scan_slots_kernel): segments of up to
// kSlotSubs subsequences of kSlotBits bits, each with up to kSlotStates entry states; the last place is kept
// for a state that was not found in time.
constexpr int kSlotSubs = 64, kSlotBits = 512, kSlotStates = 16, kSlotRounds = 4;
constexpr uint32_t kSlotMiss = 255;

struct alignas(8) SlotMap {
    uint32_t from, to; // state before (kNoState: none), state behind | blocks << 16
};
struct SlotTables {                         // of one segment
    uint32_t info[kSlotSubs][kSlotStates];  // entry state of a subsequence | blocks completed in it << 16
    uint8_t next[kSlotSubs][kSlotStates];   // which state of the next subsequence it leads to
    SlotMap map[kSlotStates];               // per state of the first subsequence
};
constexpr uint32_t kNoState = 0xFFFFFFFFu;

// Per-sample work descriptor.
struct ImageDesc {
    uint64_t payload_off;  // byte offset of the staged payload inside the blob (16-byte aligned)
    uint32_t payload_size; // staged bytes
    uint16_t mode;         // 0 jpg, 1 raw (ffcv/fields/rgb_image.py:21-23)
    int16_t host_status;   // 0, or a negative code: the host parser rejected the stream, or its bytes did not arrive
    uint16_t height, width;
    uint16_t row0, rows;   // raw: first image row present in the staged payload, number of rows
    uint16_t col0, cols;   // raw: first image column present, number of columns
    union {
        uint32_t raw_pitch; // raw: bytes between staged rows (>= cols * 3)
        uint32_t rgb_pitch; // JPEG: bytes between rows of the decoded RGB image (>= dec_width * 3; a multiple
                            // of 16 in the batch scratch so that the colour kernels store whole words)
    };
    // ---- JPEG only ----
    uint32_t scan_off;     // entropy-coded segment, relative to payload_off
    uint32_t scan_len;
    uint8_t ncomp, hs, vs, bpm; // luma sampling factors; blocks per MCU
    uint16_t mcus_x, mcus_y;
    uint16_t restart_interval;
    uint8_t fast_tables;             // every Huffman table is HuffTable::fast_ok
    uint8_t n_tab, n_dc_tab;         // distinct Huffman tables of this image (the DC tables first):
    uint8_t tab_id[6];               // their indices into the batch's HuffTable array,
    uint8_t dc_tab[kMaxComponents];  // and which of them each component's
    uint8_t ac_tab[kMaxComponents];  // DC and AC symbols use
    uint8_t q_tab[kMaxComponents];   // indices into the batch's MultTable array
    uint8_t raw_skew;      // raw, gathered row by row: row r of the staged payload starts
                           // (src_addr + r * width * 3) & 15 bytes into its raw_pitch-wide slot
    // Decoding at reduced scale (1 / 2^scale_shift, JPEG only): every block of a component is
    // inverted straight to bs x bs samples (8 at full scale), and the decoded image has
    // dec_height x dec_width = ceil(height / 2^s) x ceil(width / 2^s) pixels.  With 2x2 chroma
    // subsampling the chroma blocks use twice the luma's bs (at most 8), so all planes of a scaled
    // image have the same resolution.  dec_* equal height / width for unscaled and raw samples.
    uint8_t scale_shift, bs_luma, bs_chroma;
    uint16_t dec_height, dec_width;
    // Entropy decode in segments (scans without restart markers): length in bits of the
    // subsequences (multiple of 32); raw bytes of a segment; subsequences of run-up before every
    // segment but the first; bits of run-up before every subsequence (a multiple of 32); bytes of a segment's place in the unstuffed stream; and which of the
    // batch's segments are this image's; and how many subsequences of its own a segment has at most.
    uint32_t subseq_bits, seg_raw, seg_warm, seg_run_up, seg_stride, seg_first, seg_count, seg_lanes;
    uint32_t rec_first, rec_room; // room for what its subsequences write down, see record_room: the first one's place / 4, and of each
    uint32_t slots;        // decoded from every slot at once: 1 + the first of the image's SlotTables (0: not)
    uint32_t index_use;    // place in the decode index: 0 none, bit 0 the entry may be read, bit 1 and is written
    uint64_t index_off;    // byte offset of the entry in the context's index pool
    // The crop box decides how much of the image is needed: the entropy decoder stops after
    // `mcu_rows` rows of MCUs and the inverse transform runs only on the MCUs of the box below
    // (the crop box grown by the reach of the chroma filter).  Whole image when there is no crop.
    uint16_t mcu_rows;                           // MCU rows to entropy-decode (<= mcus_y)
    uint16_t idct_row0, idct_col0, idct_col1;    // MCU box to transform: rows [idct_row0, mcu_rows), cols [idct_col0, idct_col1)
    uint32_t nblocks;      // 8x8 blocks to decode: bpm * mcus_x * mcu_rows
    uint32_t block_base;   // first block of this image in the batch's block index
    uint64_t clean_off;    // byte offset of the unstuffed scan in the bitstream scratch (16-aligned)
    uint64_t rst_off;      // streams with restart markers: byte offset, in the same scratch, of a table of
                           // ceil(MCUs / restart_interval) + 1 uint32 interval starts (4-aligned)
    uint64_t plane_off[kMaxComponents]; // byte offsets of the Y/Cb/Cr planes in the plane scratch
    uint64_t rgb_off;      // byte offset of the decoded h*w*3 image in the RGB scratch
    uint16_t fuse_rows;    // the resize kernel converts the planes itself, for this many output rows at a time (0: the
                           // colour kernels leave an image in the RGB scratch)
    uint64_t src_addr;     // device-visible address of the payload in pinned host memory (0: staged copy)
};

// Canonical Huffman code (ITU-T T.81 Annex C) prepared for table-driven decoding.
constexpr int kHuffBits = 10;     // bits the first level resolves: 99 % of the symbols of photographs
constexpr int kHuffSubTables = 8; // the standard tables need 5; others fall back to the code-length walk
constexpr int kHuffExtra = 512;
constexpr int kHuffFast = 65536 / 64 + kHuffExtra - kHuffExtra / 64;
static_assert(kHuffBits == 10, "the fast tables count on it");
constexpr int kPairAdvance = 4;
struct HuffTable {
    // Table entries describe what a code does to the decoder rather than what it is (see
    // huff_entry): bits 0-4 the bits the symbol consumes (code + magnitude bits), bits 5-8 the
    // number of magnitude bits, bits 9-14 the zig-zag positions it advances (DC: 1; AC: run + 1,
    // 16 for a run of zeros, 63 for an end of block, which always reaches the block's end).
    // First level, indexed by the next kHuffBits bits: such an entry for codes that fit;
    // kHuffLong | k when the code is longer and continues in sub[k]; all ones when it is longer
    // and no sub-table was left (walk maxcode/valoff instead).  A prefix that is no code holds
    // huff_invalid.
    uint16_t look[1 << kHuffBits];
    // Second level, indexed by the bits of the code behind those, up to the 16th: an entry as above.
    uint16_t sub[kHuffSubTables][1 << (16 - kHuffBits)];
    // For the entropy decoder's inner loop, which may not branch: the low byte of an entry is the number
    // of bits consumed, the high byte the positions advanced.  With v the next 16 bits, the index is
    // max(v / 64, v - 65536 + kHuffFast): the first kHuffBits bits, except for the last kHuffExtra values
    // of v, which have an entry each.  Codes are assigned in order of their length, so the long ones
    // are the last; whether all codes of more than kHuffBits bits lie there (those of the standard
    // tables begin 320 before the end) is `fast_ok`.
    uint16_t fast[kHuffFast];
    // The same for AC symbols, but two at a time where the second one's bits are among the first
    // kHuffBits as well and the first one advances at most kPairAdvance positions: with less than 64 -
    // kPairAdvance positions behind it a block cannot end between the two.
    uint16_t pair[kHuffFast];
    int32_t maxcode[18]; // largest code of each length, -1 if none
    int32_t valoff[17];  // index of the first symbol of each length minus its first code
    int32_t is_dc, fast_ok, pad[3];
    uint8_t vals[256];
};
constexpr uint32_t kHuffLong = 0x8000u;
static_assert(sizeof(HuffTable) % 16 == 0, "tables are copied in vectors");

#if defined(__CUDACC__)
#define FFCVB_HD __host__ __device__
#else
#define FFCVB_HD
#endif
// Entry of a code of `len` bits for symbol `sym` (run << 4 | magnitude bits).  An AC symbol without
// magnitude bits is a run of 16 zeros when its run field is 15 and ends the block otherwise.
FFCVB_HD inline uint16_t huff_entry(int len, int sym, bool dc) {
    const int s = sym & 15, r = sym >> 4;
    const int dz = dc ? 1 : (s != 0 ? r + 1 : (r == 15 ? 16 : 63));
    return (uint16_t)((len + s) | (s << 5) | (dz << 9));
}
// A bit pattern that is no code: 16 bits without a value that end the block (an AC symbol), so that a
// decoder on garbage makes progress.
FFCVB_HD inline uint16_t huff_invalid(bool dc) { return (uint16_t)(16 | ((dc ? 1 : 63) << 9)); }

// Dequantisation multipliers of the fast integer IDCT in zig-zag order: quantiser step x AAN scale, 2
// fraction bits; and, in natural order, the plain quantiser steps, which the reduced-size transforms
// of a scaled decode use.
struct MultTable {
    int16_t m[64];
    uint16_t q[64];
};

// Segment of a scan as scan_guess_kernel leaves it.  Bits count from the start of the segment's
// place in the unstuffed stream.
struct alignas(16) SegMeta {
    uint32_t own_bit, own_end; // the segment's own bits (behind its run-up, before its overlap)
    uint32_t bytes;            // unstuffed bytes, overlap included
    uint32_t blocks;           // blocks completed in the segment
    uint32_t entry;            // SlotTables: which state of the first subsequence is the real one
    uint32_t pad[3];
    uint32_t doubt[kSegSubs / 32]; // a bit per subsequence that may not begin in the state the one before it ends in
};

// Positions of its blocks that the decode of a subsequence writes down as it goes: room for so many, the last place
// spare.  A quarter of a subsequence's bits are as many as the standard tables allow, four times the scan's own bytes.
// Where that is too much (`all` is false: kAllRecordsBits), twice as many as it has on average, at least one for
// every 20 bits.  Segments with a subsequence that has more are decoded once more, a whole walk later than the others: with
// twice the average alone the photographs' overexposed parts cost 1024 images of 145 kbit 25 us of 207; 1024 images whose upper half
// is of one colour take 265 us with room for all, 318 with less, 336 with 127 blocks.
constexpr uint64_t kAllRecordsBits = 160u << 20; // of a batch's scans, at most: 80 MB
FFCVB_HD inline uint32_t record_room(uint32_t subseq_bits, uint32_t scan_len, uint32_t blocks, bool all) {
    const uint64_t mean = scan_len ? (uint64_t)blocks * subseq_bits / (8 * (uint64_t)scan_len) : 0, least = subseq_bits / 20, most = subseq_bits / 4 + 2;
    const uint64_t room = 2 * mean + 8 > least ? 2 * mean + 8 : least;
    return (uint32_t)((all || room > most ? most : room) + 15) / 16 * 16;
}

constexpr uint32_t kNoBlock = 0xFFFFFFFFu; // position of a block that the scan does not hold

// Decode index: what a finished decode of a stream knows and the next decode of the same stream can
// start from -- the exact decoder state at the start of every subsequence and the number of blocks
// completed in it.  With it no guess has to be repaired.  An entry lives in device memory:
//   [DecodeIndexHeader][per segment: uint32 sub_info x ImageDesc::seg_lanes]
// and is valid when `magic` is set (written last) and the other fields match.  Which batch writes it and which
// may read it is settled on the host (DecodeIndex).
struct DecodeIndexHeader {
    uint32_t magic, scan_len, subseq_bits, segments;
};
constexpr uint32_t kDecodeIndexMagic = 0x58444947u;
FFCVB_HD inline size_t decode_index_bytes(uint32_t segments, uint32_t lanes) {
    return (sizeof(DecodeIndexHeader) + (size_t)segments * lanes * 4 + 15) / 16 * 16;
}

struct BatchHeader {
    uint32_t n, n_huff, n_mult, n_params; // n_params = int32 per sample
    uint64_t desc_off, huff_off, mult_off, params_off, payload_off, total_bytes;
};

// Augmentation list + output description handed to the fused kernel by value.
struct OpList {
    int32_t n_ops;
    int32_t type[8];
    int32_t arg[8];
    uint8_t fill[8][4];
};

enum : int { kErrFormat = -1, kErrUnsupported = -2, kErrDims = -3, kErrData = -4 };

} // namespace ffcvb
