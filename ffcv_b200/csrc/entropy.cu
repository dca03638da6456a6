// Batched baseline-JPEG entropy decode (ITU-T T.81 F.2) for sm_100a: from a scan to the place of
// every 8x8 block in it.
//
// The scan has no restart markers in FFCV-written files (ffcv/fields/rgb_image.py:26-34 passes only
// the quality to cv2.imencode), so parallelism inside an image comes from the self-synchronising
// property of Huffman codes.  What these kernels produce is not coefficients but an index: for every
// block the bit position of its first AC symbol in the unstuffed stream, and its DC value.  With it
// the inverse transform (idct.cu) decodes any block on its own, in parallel and only where the crop
// needs it, and no coefficient ever travels through global memory.
//
//   scan_guess_kernel   one thread per subsequence, up to 128 of them a segment, whose bytes lie in shared memory without
//                       their stuffing: decodes a run-up before the subsequence from a guessed state, then the
//                       subsequence itself, writing down where its blocks begin.  A decoder that starts
//                       mid-stream falls in step after 0.9 kbit on average (4:2:0, quality 90), dominated by
//                       the block's slot inside the MCU: after 1.9 kbit nine in ten have.
//   scan_repair_kernel  decodes the others again, from the state the subsequence before them really ends in,
//                       until every one begins where the one before it ends.
//   scan_slots_kernel, scan_chain_kernel   instead of the two above while a batch's scans leave most of the
//                       GPU idle: every subsequence from all block slots at once, see there.
//   scan_index_kernel   positions and DC values of the blocks, out of what was written down (with
//                       scan_slots_kernel: by decoding once more from the exact states); the last CTA of an
//                       image integrates the DC differences.
//
// Integer work bound by instruction issue at large batches and by the chain look-up -> shift ->
// look-up at small ones: about 25 instructions per symbol and lane, tables and stream in shared memory.
#include "huffman.h"
#include "kernels.h"

#include <algorithm>

namespace ffcvb {

namespace {

constexpr int kThreads = kSegSubs;          // one thread per subsequence: a team of four warps per segment
constexpr int kFastBytes = 2 * kHuffFast;   // a Huffman table in shared memory

// The threads that work on one segment.  A CTA holds one team, or several that share the Huffman
// tables in shared memory and meet at barriers of their own.  Every team's first warp is another one of the
// SM's quarters', because segments often need only the first two (130 us instead of 94 when they were the same ones').
template <int TEAMS, int SIZE = kThreads>
struct Team {
    static constexpr int size = SIZE;
    int index, tid;
    __device__ __forceinline__ Team() : index(TEAMS == 1 ? 0 : threadIdx.x / SIZE), tid(TEAMS == 1 ? threadIdx.x : (threadIdx.x + 32 * index) % SIZE) {}
    __device__ __forceinline__ void sync() const {
        if (TEAMS == 1)
            __syncthreads();
        else
            asm volatile("bar.sync %0, %1;" ::"r"(index + 1), "n"(SIZE) : "memory");
    }
};

// Exclusive prefix sum over `warps` warps that meet at `sync`; `total` receives the sum.
template <class Sync>
__device__ __forceinline__ int scan_exclusive(int v, int tid, int warps, int *s_warp, int &total, Sync &&sync) {
    const int lane = tid & 31, warp = tid >> 5;
    int inc = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        int t = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += t;
    }
    if (lane == 31) s_warp[warp] = inc;
    sync();
    int before = 0, all = 0;
#pragma unroll
    for (int k = 0; k < warps; k++) {
        const int w = s_warp[k];
        before += k < warp ? w : 0;
        all += w;
    }
    sync();
    total = all;
    return before + inc - v;
}
template <class AnyTeam>
__device__ __forceinline__ int team_scan(const AnyTeam &team, int v, int *s_warp, int &total) {
    return scan_exclusive(v, team.tid, AnyTeam::size / 32, s_warp, total, [&] { team.sync(); });
}

__device__ __forceinline__ uint32_t shared_address(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ uint32_t load_shared(uint32_t a) {
    uint32_t v;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(a));
    return v;
}

// Global to shared memory without passing through registers; copies_wait: this thread's have landed.
__device__ __forceinline__ void copy16_async(void *dst, const void *src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(shared_address(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void copies_wait() {
    asm volatile("cp.async.commit_group;" ::: "memory");
    asm volatile("cp.async.wait_group 0;" ::: "memory");
}

// Tables of an image in shared memory: for every block slot of an MCU where its Huffman tables are
// and which slot follows, then HuffTable::fast of the image's distinct tables (DC, then AC), then
// HuffTable::pair of the AC tables.
struct Slot {
    uint32_t tables; // shared-memory address of the DC table | of the AC table << 16
    uint32_t next;   // shared-memory address of the slot that follows
};
struct Tables {
    Slot slot[6];
    uint32_t bpm, luma, pairs, pad; // blocks of an MCU, luma blocks among them; from an AC table to its pair table
    uint16_t fast[8];               // (the first vector of the tables)
};
constexpr size_t kTablesHead = offsetof(Tables, fast);
static_assert(kSegSubs == 128, "SegMeta::doubt is read as four words");
static_assert(kTablesHead % 16 == 0 && kFastBytes % 16 == 0 && offsetof(HuffTable, fast) % 16 == 0 && offsetof(HuffTable, pair) % 16 == 0,
              "tables are copied in vectors");
__host__ __device__ constexpr size_t tables_bytes(int n_tables) { return kTablesHead + (size_t)n_tables * kFastBytes; }

// Starts the copies of the tables; copies_wait and a barrier of the whole CTA complete them.
__device__ __forceinline__ void load_tables(Tables *s, const ImageDesc &d, const HuffTable *__restrict__ huff) {
    const int luma = d.hs * d.vs, n = d.n_tab, n_dc = d.n_dc_tab, tid = threadIdx.x;
    const uint32_t fast = shared_address(s->fast);
    if (d.fast_tables)
        for (int u = 0; u < 2 * n - n_dc; u++) {
            const HuffTable &t = huff[d.tab_id[u < n ? u : u - (n - n_dc)]];
            const uint4 *src = reinterpret_cast<const uint4 *>(u < n ? t.fast : t.pair);
            uint4 *dst = reinterpret_cast<uint4 *>(s->fast) + u * (kFastBytes / 16);
            for (int i = tid; i < kFastBytes / 16; i += blockDim.x) copy16_async(dst + i, src + i);
        }
    if (tid < d.bpm) {
        const int comp = (d.ncomp == 1 || tid < luma) ? 0 : tid - luma + 1;
        s->slot[tid].tables = (fast + d.dc_tab[comp] * (uint32_t)kFastBytes) | (fast + d.ac_tab[comp] * (uint32_t)kFastBytes) << 16;
        s->slot[tid].next = shared_address(&s->slot[tid + 1 == d.bpm ? 0 : tid + 1]);
    }
    if (tid == 0) {
        s->bpm = d.bpm;
        s->luma = d.ncomp == 1 ? 1 : luma;
        s->pairs = (uint32_t)((n - n_dc) * kFastBytes);
    }
}

// Decoder state between two symbols: bit position, block slot inside the MCU, next zig-zag index
// (0: DC expected).
struct Cursor {
    uint32_t p;
    int c, z;
};
// Packed into 16 bits relative to a position `from` that the cursor has reached by less than 32 bits.
__device__ __forceinline__ uint32_t pack(const Cursor &s, uint32_t from) { return (s.p - from) | (uint32_t)s.c << 5 | (uint32_t)s.z << 8; }
__device__ __forceinline__ Cursor unpack(uint32_t v, uint32_t from) { return Cursor{from + (v & 31), (int)((v >> 5) & 7), (int)((v >> 8) & 63)}; }

// What a walk writes down: nothing, positions of blocks, or the records of a subsequence.
enum { kNothing, kPositions, kRecord };

// The walk below in plain code: for tables that are not fast_ok, and for the few walks on a stream in
// global memory.  One symbol at a time, tables where they are.
template <int RECORD>
__device__ __noinline__ uint32_t walk_plain(const uint32_t *words, Cursor &cur, uint32_t end, const ImageDesc &d,
                                            const HuffTable *__restrict__ huff, uint32_t *pos, uint32_t blk, uint32_t limit, uint16_t *rec) {
    const int luma = d.ncomp == 1 ? 1 : d.hs * d.vs;
    uint32_t done = 0, n = 0;
    while (cur.p < end) {
        if (RECORD == kPositions && cur.z == 0) {
            if (blk < limit) pos[blk] = cur.p;
            blk++;
        }
        if (RECORD == kRecord && cur.z == 0) {
            if (n < limit - 1) rec[n] = (uint16_t)(cur.p + blk);
            n++;
        }
        const uint32_t w = __funnelshift_l(words[(cur.p >> 5) + 1], words[cur.p >> 5], cur.p);
        const int comp = cur.c < luma ? 0 : cur.c - luma + 1;
        const HuffTable *t = huff + d.tab_id[cur.z ? d.ac_tab[comp] : d.dc_tab[comp]];
        uint32_t e = t->look[w >> (32 - kHuffBits)];
        if (e & kHuffLong) e = huff_long(t, e, w);
        cur.p += e & 31;
        cur.z += (int)(e >> 9);
        if (cur.z >= 64) {
            cur.z = 0;
            cur.c = cur.c + 1 == d.bpm ? 0 : cur.c + 1;
            done++;
        }
    }
    return done;
}

// Decodes symbols from `cur` until its position reaches `end`; returns the number of blocks
// completed.  `buf`: the segment's stream (words most significant bit first) in shared memory, or, with GLOBAL, in
// global memory.  With kPositions every block that begins before `end` gets its position written to pos[blk], pos[blk + 1],
// ... below pos[limit]; `blk` is the first of them.  With kRecord the low 16 bits of the positions, plus blk, go to
// rec[0], rec[1], ... as far as rec[limit - 2]; what lies behind the last one, up to rec[limit - 1], may be overwritten.
//
// The 32 lanes of a warp walk unrelated places, so nothing in the loops branches: position (bits 0-23)
// and zig-zag index (bits 24-30) share one word that an entry is simply added to; a 96-bit window over
// the stream stays in registers (hi holds the word the position lies in, lo and nx the two behind it)
// and is moved on by predicated instructions; so are the table switches and the slot at the end of a
// block; codes too long for the first level are reached by the index's maximum.  As long as `end` is
// more than kHuffBits away an entry may stand for two symbols (1.46 on average), so that the walk's
// last position is the same whatever state it came from.
constexpr uint32_t kPosMask = 0xffffff;
constexpr int kLongest = 31; // bits of a symbol, at most
template <int RECORD, bool GLOBAL = false>
__device__ __forceinline__ uint32_t walk(const unsigned char *buf, Cursor &cur, uint32_t end, const Tables *s, const ImageDesc &d,
                                         const HuffTable *__restrict__ huff, uint32_t *pos = nullptr, uint32_t blk = 0, uint32_t limit = 0,
                                         uint16_t *rec = nullptr) {
    if (cur.p >= end) return 0;
    if (!d.fast_tables) return walk_plain<RECORD>(reinterpret_cast<const uint32_t *>(buf), cur, end, d, huff, pos, blk, limit, rec);
    const uint32_t pairs = s->pairs;
    uint32_t st = cur.p | (uint32_t)cur.z << 24, done = 0;
    const Slot here = s->slot[cur.c];
    uint32_t ac = here.tables >> 16, tab = cur.z ? ac : here.tables & 0xffff;
    uint32_t ahead = load_shared(here.next), after = load_shared(here.next + 4); // the slot that follows
    uint32_t wa = 0, hi, lo, nx;
    const uint32_t *ga = reinterpret_cast<const uint32_t *>(buf) + (cur.p >> 5);
    if (GLOBAL) {
        for (uint32_t k = 0; k < (end - cur.p) / 8; k += 128) { // every line once, so that the words come from the cache below
            uint32_t touched;
            asm volatile("ld.global.u32 %0, [%1];" : "=r"(touched) : "l"(ga + k / 4));
        }
        hi = ga[0], lo = ga[1], nx = ga[2];
        ga += 3;
    } else {
        wa = shared_address(buf) + (cur.p >> 5) * 4;
        hi = load_shared(wa), lo = load_shared(wa + 4), nx = load_shared(wa + 8);
        wa += 12;
    }
    if (RECORD == kPositions && cur.z == 0) {
        if (blk < limit) pos[blk] = cur.p;
        blk++;
    }
    if (RECORD == kRecord && cur.z == 0) *rec++ = (uint16_t)(cur.p + blk);
    uint32_t p = cur.p;
    auto symbol = [&](bool paired) {
        const uint32_t w = __funnelshift_l(lo, hi, st);
        const uint32_t index = (uint32_t)__viaddmax_s32((int)(w >> 16), kHuffFast - 65536, (int)(w >> 22));
        uint32_t e;
        asm volatile("{\n\t"
                     ".reg .u16 h;\n\t"
                     "ld.shared.u16 h, [%1];\n\t"
                     "cvt.u32.u16 %0, h;\n\t"
                     "}"
                     : "=r"(e)
                     : "r"(tab + index * 2));
        e = __byte_perm(e, 0, 0x1440); // bits consumed to bits 0-7, positions advanced to bits 24-31
        const uint32_t before = st;
        st += e;
        if (GLOBAL)
            asm volatile("{\n\t"
                         ".reg .pred q;\n\t"
                         ".reg .b32 t;\n\t"
                         "xor.b32 t, %4, %5;\n\t"
                         "and.b32 t, t, 32;\n\t"
                         "setp.ne.u32 q, t, 0;\n\t"
                         "@q mov.b32 %0, %1;\n\t"
                         "@q mov.b32 %1, %2;\n\t"
                         "@q ld.global.u32 %2, [%3];\n\t"
                         "@q add.u64 %3, %3, 4;\n\t"
                         "}"
                         : "+r"(hi), "+r"(lo), "+r"(nx), "+l"(ga)
                         : "r"(before), "r"(st));
        else
            asm volatile("{\n\t"
                         ".reg .pred q;\n\t"
                         ".reg .b32 t;\n\t"
                         "xor.b32 t, %4, %5;\n\t"
                         "and.b32 t, t, 32;\n\t"
                         "setp.ne.u32 q, t, 0;\n\t"
                         "@q mov.b32 %0, %1;\n\t"
                         "@q mov.b32 %1, %2;\n\t"
                         "@q ld.shared.u32 %2, [%3];\n\t"
                         "@q add.u32 %3, %3, 4;\n\t"
                         "}"
                         : "+r"(hi), "+r"(lo), "+r"(nx), "+r"(wa)
                         : "r"(before), "r"(st));
        // (closer to the block's end a pair might reach beyond it with its first symbol)
        tab = ac + (paired && st < (uint32_t)(64 - kPairAdvance) << 24 ? pairs : 0);
        const bool eob = st >= 0x40000000u;
        asm volatile("{\n\t"
                     ".reg .pred q;\n\t"
                     "setp.ge.u32 q, %0, 0x40000000;\n\t"
                     "@q and.b32 %0, %0, 0xffffff;\n\t"
                     "@q add.u32 %1, %1, 1;\n\t"
                     "@q and.b32 %2, %4, 0xffff;\n\t"
                     "@q shr.u32 %3, %4, 16;\n\t"
                     "@q ld.shared.v2.u32 {%4, %5}, [%5];\n\t"
                     "}"
                     : "+r"(st), "+r"(done), "+r"(tab), "+r"(ac), "+r"(ahead), "+r"(after));
        p = st & kPosMask;
        if (RECORD == kPositions) {
            if (eob && p < end && blk < limit) pos[blk] = p;
            blk += eob ? 1 : 0;
        }
        if (RECORD == kRecord && eob && done < limit) rec[done - 1] = (uint16_t)(st + blk);
    };
    const int pairs_end = (int)end - kHuffBits; // the first symbol of a pair that begins up to here ends before `end`
    if ((int)p <= pairs_end) {
        while ((int)p <= pairs_end - kLongest) { // (so does one behind it)
            symbol(true);
            symbol(true);
        }
        while ((int)p <= pairs_end) symbol(true);
        if (st >> 24) tab = ac; // (at 0 it is the DC table)
    }
    while (p < end) symbol(false);
    cur.p = p;
    cur.z = (int)(st >> 24);
    cur.c = (int)((cur.c + done) % s->bpm);
    return done;
}

// ---- byte stuffing -------------------------------------------------------------------------
// Bytes of y (little-endian word x of the scan, prev: the byte before it) that are to be dropped: a
// 00 behind an FF.  Bit 8k + 7 is set for byte k.
__device__ __forceinline__ uint32_t stuffing_of(uint32_t x, uint32_t prev_word) {
    const uint32_t y = x | ~__funnelshift_l(prev_word, x, 8); // a byte is 0 where x is 00 and its predecessor FF
    return ~(((y & 0x7f7f7f7fu) + 0x7f7f7f7fu) | y | 0x7f7f7f7fu);
}
// The first k bytes of a word (as the flags above); k <= 0: none, k >= 4: all.
__device__ __forceinline__ uint32_t first_bytes(int k) {
    return k <= 0 ? 0u : (k >= 4 ? 0x80808080u : 0x80808080u >> (8 * (4 - k)));
}

// Unstuffs `len` raw bytes at `src` into `buf` (shared memory; room for len + 64 bytes and a word), most
// significant byte of every word first, followed by 64 zero bytes.  `first`: nothing precedes the
// bytes.  s_mark[k] receives how many kept bytes lie before raw offset at[k].  Returns the number of
// bytes kept.  A thread takes 32 aligned bytes per pass; nearly all words lose nothing and leave as
// one shifted word, single bytes are stored only where two threads' bytes share a word.
template <class AnyTeam>
__device__ __forceinline__ uint32_t unstuff(const AnyTeam &team, unsigned char *buf, const uint8_t *__restrict__ src, uint32_t len,
                                            bool first, const uint32_t (&at)[2], int *s_warp, uint32_t *s_mark) {
    constexpr int kWords = 8;
    const int tid = team.tid;
    const uint32_t lead = (uint32_t)(reinterpret_cast<uintptr_t>(src) & 15);
    const uint8_t *aligned = src - lead;
    const uint32_t nwords = ((lead + len + 15) >> 4) * 4;
    uint32_t *words = reinterpret_cast<uint32_t *>(buf);
    uint32_t kept = 0;
    uint4 v[2];
    auto fetch = [&](uint32_t w) {
#pragma unroll
        for (int k = 0; k < 2; k++) v[k] = w + 4 * k < nwords ? reinterpret_cast<const uint4 *>(aligned)[(w >> 2) + k] : make_uint4(0, 0, 0, 0);
    };
    fetch(tid * kWords);
    for (uint32_t tile = 0; tile < nwords; tile += AnyTeam::size * kWords) {
        const uint32_t w0 = tile + tid * kWords;
        uint32_t x[kWords] = {v[0].x, v[0].y, v[0].z, v[0].w, v[1].x, v[1].y, v[1].z, v[1].w};
        fetch(w0 + AnyTeam::size * kWords); // the next pass's bytes arrive during this one
        const int off = (int)(w0 * 4) - (int)lead; // raw offset of the first of these bytes
        const bool edge = off < 0 || off + kWords * 4 > (int)len;
        if (first && off < 0) // what lies in front of the scan is no predecessor
#pragma unroll
            for (int k = 0; k < 4; k++) x[k] &= ~((first_bytes(-(off + 4 * k)) >> 7) * 255u);
        uint32_t prev = __shfl_up_sync(0xffffffffu, x[kWords - 1], 1);
        if ((tid & 31) == 0) prev = w0 < nwords && (w0 > 0 || (lead == 0 && !first)) ? (uint32_t)aligned[(int)(w0 * 4) - 1] << 24 : 0;
        uint32_t keep[kWords];
        int cnt = 0;
#pragma unroll
        for (int k = 0; k < kWords; k++) {
            keep[k] = ~stuffing_of(x[k], k == 0 ? prev : x[k - 1]) & 0x80808080u;
            if (edge) keep[k] &= ~first_bytes(-(off + 4 * k)) & first_bytes((int)len - (off + 4 * k));
            cnt += __popc(keep[k]);
        }
        int total;
        const uint32_t o = kept + (uint32_t)team_scan(team, cnt, s_warp, total);
#pragma unroll
        for (int m = 0; m < 2; m++) {
            const int a = (int)at[m] - off;
            if (a >= 0 && a < kWords * 4) { // raw offset at[m] is one of these bytes
                uint32_t n = o;
#pragma unroll
                for (int k = 0; k < kWords; k++) n += __popc(keep[k] & first_bytes(a - 4 * k));
                s_mark[m] = n;
            }
        }
        // `acc` holds the bytes of word wi this thread has so far, ph bits of the word are taken (by it
        // or by the thread before it)
        uint32_t ph = (o & 3) * 8, acc = 0, wi = o >> 2, mine = o & 3; // bytes below `mine` are another thread's
        auto store = [&](uint32_t upto) {
            if (mine == 0 && upto == 4)
                words[wi] = acc;
            else
                for (uint32_t q = mine; q < upto; q++) buf[(wi * 4 + q) ^ 3u] = (uint8_t)(acc >> (24 - 8 * q));
            mine = 0;
            wi++;
        };
#pragma unroll
        for (int k = 0; k < kWords; k++) {
            uint32_t b = __byte_perm(x[k], 0, 0x0123), bits = 32;
            if (keep[k] != 0x80808080u) { // close the gaps, last byte first
                bits = 8 * __popc(keep[k]);
#pragma unroll 1
                for (uint32_t gone = ~keep[k] & 0x80808080u; gone != 0; gone &= gone - 1) {
                    // the dropped byte with the lowest address not yet dealt with is the one nearest the top
                    const uint32_t q = (__ffs(gone) - 1) & ~7u, shift = q - (8 * __popc(~keep[k] & 0x80808080u & ((gone & (0u - gone)) - 1)));
                    const uint32_t top = shift ? 0xffffffffu << (32 - shift) : 0;
                    b = (b & top) | ((b << 8) & ~top);
                }
            }
            acc |= b >> ph;
            ph += bits;
            if (ph >= 32) {
                store(4);
                ph -= 32;
                acc = __funnelshift_lc(0u, b, bits - ph); // the ph bits that did not fit
            }
        }
        store(ph / 8);
        kept += (uint32_t)total;
    }
    if (tid < 64) buf[(kept + tid) ^ 3u] = 0;
    team.sync();
    return kept;
}

// ---- kernels -------------------------------------------------------------------------------

struct GuessShared {
    uint16_t exit[kThreads];
    int warp[kThreads / 32];
    uint32_t mark[2];
    alignas(16) uint32_t differ[2][kThreads / 32];
};
// Shared memory of a team's stream: the aligned vectors that hold max_raw bytes, and the zero bytes behind.
__host__ __device__ constexpr size_t stream_bytes(uint32_t max_raw) { return ((size_t)max_raw + 16 + 64 + 31) / 16 * 16; }

__device__ __forceinline__ bool index_entry_valid(const DecodeIndexHeader *entry, const ImageDesc &d) {
    const volatile DecodeIndexHeader *h = entry; // written by an earlier launch
    return h->magic == kDecodeIndexMagic && h->scan_len == d.scan_len && h->subseq_bits == d.subseq_bits && h->segments == d.seg_count;
}

// What subsequence t of segment j writes down.
__device__ __forceinline__ uint16_t *records_of(const EntropyScratch &scratch, const ImageDesc &d, uint32_t j, uint32_t t) {
    return scratch.records + 4 * (size_t)d.rec_first + ((size_t)j * d.seg_lanes + t) * d.rec_room;
}

// Every thread decodes one subsequence, beginning a run-up before it in a guessed state: a block, slot 0, begins there.  Most
// have fallen in step with the real state where the subsequence begins.  Of the others each is noticed by its neighbour's
// exit, once: SegMeta::doubt, for scan_repair_kernel.  With `local` the CTA repeats them itself, in rounds, until every
// subsequence begins where the one before it ends, and only a segment's first one is left in doubt; only then have segments
// subsequences that lead up to them (negative t, which a decode index, never used with `local`, has no words for).
template <int TEAMS>
__global__ void __launch_bounds__(kThreads * TEAMS, TEAMS == 4 ? 2 : 1)
scan_guess_kernel(const ImageDesc *__restrict__ descs, const uint2 *__restrict__ segs, int n_segs, const uint8_t *__restrict__ blob,
                  const HuffTable *__restrict__ huff, EntropyScratch scratch, const uint8_t *__restrict__ index_pool,
                  unsigned long long *__restrict__ index_stats, int table_slots, uint32_t buf_bytes, bool local) {
    const bool local_repair = TEAMS == 1 && local; // (segments that share tables never are)
    extern __shared__ __align__(16) unsigned char s_dyn[];
    __shared__ GuessShared s_teams[TEAMS];
    next_may_begin();
    const Team<TEAMS> team;
    const int tid = team.tid;
    GuessShared &sh = s_teams[team.index];
    Tables *tables = reinterpret_cast<Tables *>(s_dyn);
    unsigned char *buf = s_dyn + tables_bytes(table_slots) + team.index * buf_bytes;
    const int mine = blockIdx.x * TEAMS + team.index;
    const uint2 which = segs[min(mine, n_segs - 1)];
    const uint32_t j = which.y;
    const ImageDesc &d = descs[which.x];
    const uint32_t S = d.subseq_bits, R = d.seg_raw, run_up = d.seg_run_up, lead = TEAMS > 1 || j == 0 ? 0 : d.seg_warm;
    load_tables(tables, d, huff); // (the same whichever team's sample they are taken from)
    if (TEAMS > 1) {
        copies_wait();
        __syncthreads();
        if (mine >= n_segs) return;
    }

    // ---- the segment's raw bytes: run-up, own part, and what follows it to the end of a block
    const uint32_t scan_len = d.scan_len, own0 = j * R, own1 = min(own0 + R, scan_len);
    const uint32_t raw0 = own0 - min(own0, (run_up + lead * S) >> 3), raw1 = min(own1 + kSegOverlap, scan_len);
    const uint32_t at[2] = {own0 - raw0, own1 - raw0};
    const uint32_t kept = unstuff(team, buf, blob + d.payload_off + d.scan_off + raw0, raw1 - raw0, raw0 == 0, at, sh.warp, sh.mark);
    const uint32_t own_bit = at[0] == 0 ? 0 : sh.mark[0] * 8, own_end = own1 == raw1 ? kept * 8 : sh.mark[1] * 8;
    {
        uint4 *dst = reinterpret_cast<uint4 *>(scratch.clean + d.clean_off + (size_t)j * d.seg_stride);
        const uint4 *src = reinterpret_cast<const uint4 *>(buf);
        for (uint32_t k = tid; k < (kept + 64 + 15) / 16; k += kThreads) dst[k] = src[k];
    }
    // thread `lead` has the segment's first subsequence, those before it have some that lead up to it
    const int t = tid - (int)lead, n_own = (int)((own_end - own_bit + S - 1) / S);
    const size_t seg = (size_t)d.seg_first + j, sub = seg * kSegSubs + max(t, 0);

    if (TEAMS == 1) {
        copies_wait();
        team.sync();
    }

    // ---- decode index: the states an earlier decode of this very stream left behind (the answer is uniform: a
    // batch is only given an entry that no launch beside it writes)
    const uint32_t *known = nullptr;
    if (index_pool != nullptr && d.index_use != 0) {
        const DecodeIndexHeader *h = reinterpret_cast<const DecodeIndexHeader *>(index_pool + d.index_off);
        if (index_entry_valid(h, d)) {
            known = reinterpret_cast<const uint32_t *>(h + 1) + (size_t)j * d.seg_lanes;
            if (tid == 0 && j == 0 && index_stats) atomicAdd(index_stats, 1ull);
        }
    }

    const int begin = (int)own_bit + t * (int)S;
    const bool live = t < n_own && (t >= 0 ? true : begin >= 0);
    const uint32_t start = (uint32_t)max(begin, 0), end = min(start + S, own_end);
    uint32_t done = 0, entry = 0;
    if (live) {
        Cursor cur{start - min(start, run_up), 0, 0}; // (the scan's first one begins in this state)
        if (known)
            cur = unpack(__ldcg(known + t) & 0xffff, start);
        else
            walk<kNothing>(buf, cur, start, tables, d, huff);
        entry = pack(cur, start);
    }
    // With local_repair subsequences are decoded again until each begins where the one before it ends.
    const bool chained = live && tid > 0 && begin >= (int)S;
    bool again = live;
    uint32_t differ;
    for (int round = 0;; round++) {
        if (again) {
            Cursor cur = unpack(entry, start);
            done = scratch.records && t >= 0 ? walk<kRecord>(buf, cur, end, tables, d, huff, nullptr, 0, d.rec_room, records_of(scratch, d, j, (uint32_t)t))
                                             : walk<kNothing>(buf, cur, end, tables, d, huff);
            sh.exit[tid] = (uint16_t)pack(cur, end);
        }
        team.sync();
        const uint32_t before = chained ? sh.exit[tid - 1] : entry;
        again = before != entry;
        differ = __ballot_sync(0xffffffffu, again);
        if ((tid & 31) == 0) sh.differ[round & 1][tid >> 5] = differ;
        team.sync();
        const uint4 all = *reinterpret_cast<const uint4 *>(sh.differ[round & 1]);
        if (!local_repair || round >= kThreads || (all.x | all.y | all.z | all.w) == 0) break;
        if (again) entry = before;
    }
    const bool own = live && t >= 0;
    if (own) {
        scratch.sub_info[sub] = entry | done << 16;
        scratch.sub_exit[sub] = sh.exit[tid];
    }
    int total;
    team_scan(team, own ? (int)done : 0, sh.warp, total);
    // (whether a segment's first one begins where the segment before ends is not known here, unless its entry says so)
    if ((tid & 31) == 0) {
        // (with local_repair none is left; otherwise lead is 0)
        scratch.meta[seg].doubt[tid >> 5] = (local_repair ? 0 : differ) | (tid == 0 && j > 0 && n_own > 0 && !known ? 1 : 0);
    }
    if (tid == 0) {
        SegMeta &m = scratch.meta[seg];
        m.own_bit = own_bit, m.own_end = own_end, m.bytes = kept, m.blocks = (uint32_t)total, m.entry = 0;
    }
}

// Makes every subsequence begin in the state the one before it ends in, a CTA for `group` parts of scans (of the same
// tables, unless it is one).  The first one of a part stays as it is, in doubt if anything is before it.  In a round all subsequences in doubt of which that is not so are decoded again from that state; the
// ones behind them are in doubt in the next round.  A part's first such subsequence is right after the round, so the rounds
// end.  The subsequences of all parts share the warps, because there are few of them: bound by the chain of look-ups, some
// 350 a round in the longest ones.
constexpr size_t kRepairStreams = 26 * 1024; // shared memory for streams (60 KB: 1 % faster alone, 2 % slower in flight)
constexpr int kRepairThreads = 256, kRepairWarps = kRepairThreads / 32, kRepairList = 1024;
__global__ void __launch_bounds__(kRepairThreads)
scan_repair_kernel(const ImageDesc *__restrict__ descs, const uint4 *__restrict__ list, int n_parts, int group,
                   const HuffTable *__restrict__ huff, EntropyScratch scratch, int table_slots, int stream_vectors, int at_once) {
    extern __shared__ __align__(16) unsigned char s_dyn[];
    __shared__ uint32_t s_item[kRepairList]; // subsequence of its scan | part of the group << 28
    __shared__ uint16_t s_state[kRepairList];
    __shared__ int s_warp[kRepairWarps], s_most;
    next_may_begin();
    Tables *tables = reinterpret_cast<Tables *>(s_dyn);
    unsigned char *streams = s_dyn + tables_bytes(table_slots);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int first = blockIdx.x * group, here = min(group, n_parts - first);
    bool loaded = false; // the tables
    // the warps share the parts' segments out, a segment per lane
    const int parts = kRepairWarps / group, part = warp / group, g = warp % group;
    const uint4 mine = list[first + min(g, here - 1)];
    const ImageDesc &d = descs[mine.x];
    const int n_seg = g < here ? (int)mine.z : 0;
    SegMeta *meta = scratch.meta + d.seg_first;
    const uint32_t *info = scratch.sub_info + (size_t)d.seg_first * kSegSubs;
    const uint16_t *exits = scratch.sub_exit + (size_t)d.seg_first * kSegSubs;
    if (tid == 0) s_most = 0;
    await_previous();
    __syncthreads();
    if (lane == 0) atomicMax(&s_most, n_seg);
    __syncthreads();
    const int most = s_most;
    auto own = [](const SegMeta &m, uint32_t S) -> uint32_t { return (m.own_end - m.own_bit + S - 1) / S; };
    for (int round = 0; round <= most * group * kSegSubs; round++) {
        int listed = 0;
        for (int base = 0; base < most; base += parts * 32) {
            const int in_part = base + part * 32 + lane, k = (int)mine.y + in_part;
            uint32_t differ[4] = {0, 0, 0, 0}, kept = 0;
            if (in_part < n_seg) { // (bits are set by atomic operations, hence not out of the first-level cache)
                const uint4 doubt = __ldcg(reinterpret_cast<const uint4 *>(meta[k].doubt));
                const uint32_t words[4] = {doubt.x, doubt.y, doubt.z, doubt.w};
#pragma unroll
                for (int q = 0; q < 4; q++)
                    for (uint32_t left = words[q]; left; left &= left - 1) {
                        const int bit = __ffs(left) - 1, i = k * kSegSubs + 32 * q + bit;
                        if ((q | bit) == 0 || ((info[i] ^ exits[i - 1]) & 0xffff) != 0) differ[q] |= 1u << bit;
                    }
            }
            if (in_part == 0 && k > 0) kept = differ[0] & 1;
            differ[0] &= ~kept;
            // (a segment's first one: behind the last of the segment before, which is never empty: an empty one, out of a
            // scan that ends in stuffing, has none behind it)
            int before = 0;
            if (differ[0] & 1) {
                before = (k - 1) * kSegSubs + (int)own(meta[k - 1], d.subseq_bits) - 1;
                if (((info[k * kSegSubs] ^ exits[before]) & 0xffff) == 0) differ[0] &= ~1u;
            }
            int total;
            int at = listed + scan_exclusive(__popc(differ[0]) + __popc(differ[1]) + __popc(differ[2]) + __popc(differ[3]), tid, kRepairWarps, s_warp, total,
                                             [] { __syncthreads(); });
            // in the order of the segments, so that the first of some part is always among them
#pragma unroll
            for (int q = 0; q < 4; q++)
                for (; differ[q] && at < kRepairList; differ[q] &= differ[q] - 1, at++) {
                    const int bit = __ffs(differ[q]) - 1, i = k * kSegSubs + 32 * q + bit;
                    s_item[at] = (uint32_t)i | (uint32_t)g << 28;
                    s_state[at] = exits[(q | bit) == 0 ? before : i - 1];
                }
            if (in_part < n_seg) // the others, for which the list has no room
                *reinterpret_cast<uint4 *>(meta[k].doubt) = make_uint4(differ[0] | kept, differ[1], differ[2], differ[3]);
            listed += total;
        }
        if (listed == 0) break;
        if (!loaded) load_tables(tables, descs[list[first].x], huff);
        loaded = true;
        const int count = min(listed, kRepairList);
        for (int begin = 0; begin < count; begin += at_once) {
            // their streams first: words that come from global memory one by one would keep a warp waiting
            const int items = min(at_once, count - begin);
            __syncthreads();
            for (int v = tid; v < items * stream_vectors; v += kRepairThreads) {
                const int n = v / stream_vectors;
                const uint32_t item = s_item[begin + n], i = item & 0xfffffff, k = i / kSegSubs;
                const ImageDesc &e = descs[list[first + (item >> 28)].x];
                const uint32_t start = scratch.meta[e.seg_first + k].own_bit + (i - k * kSegSubs) * e.subseq_bits;
                copy16_async(streams + (size_t)v * 16, reinterpret_cast<const uint4 *>(scratch.clean + e.clean_off + (size_t)k * e.seg_stride) + (start >> 7) + v - n * stream_vectors);
            }
            copies_wait();
            __syncthreads();
            if (tid < items) {
                const uint32_t item = s_item[begin + tid], i = item & 0xfffffff, k = i / kSegSubs, t = i - k * kSegSubs, state = s_state[begin + tid];
                const uint4 its = list[first + (item >> 28)];
                const ImageDesc &e = descs[its.x];
                const size_t seg = (size_t)e.seg_first + k, sub = (size_t)e.seg_first * kSegSubs + i;
                const uint32_t S = e.subseq_bits, start = scratch.meta[seg].own_bit + t * S, end = min(start + S, scratch.meta[seg].own_end);
                const uint32_t skip = start & ~127u; // position of the copied stream's bit 0
                const unsigned char *stream = streams + (size_t)tid * stream_vectors * 16;
                Cursor cur = unpack(state, start - skip);
                const uint32_t done = scratch.records ? walk<kRecord>(stream, cur, end - skip, tables, e, huff, nullptr, skip, e.rec_room, records_of(scratch, e, k, t))
                                                      : walk<kNothing>(stream, cur, end - skip, tables, e, huff);
                const uint32_t was = scratch.sub_info[sub] >> 16;
                scratch.sub_info[sub] = state | done << 16;
                scratch.sub_exit[sub] = (uint16_t)pack(cur, end - skip);
                if (done != was) atomicAdd(&scratch.meta[seg].blocks, done - was);
                if (t + 1 < own(scratch.meta[seg], S))
                    atomicOr(&scratch.meta[seg].doubt[(t + 1) >> 5], 1u << ((t + 1) & 31));
                else if (k + 1 < its.y + its.z && scratch.meta[seg + 1].own_bit < scratch.meta[seg + 1].own_end)
                    atomicOr(&scratch.meta[seg + 1].doubt[0], 1u);
            }
        }
        __syncthreads();
    }
}

// ---- few scans: every slot at once --------------------------------------------------------
// What keeps a decoder that starts mid-stream out of step is the block's slot inside the MCU.  With the GPU
// mostly idle every subsequence is therefore decoded from all slots in parallel, then from the exit states of
// the subsequence before it that were not among those, and so on for kSlotRounds rounds; the real state is
// among the known ones by then.  Three times the work of one guess, but a chain of 4 x 512 bits instead of the
// 6 to 10 kbit that the slowest of a few hundred guesses takes to fall in step: a 224x256 photograph's
// scan takes 33 + 7 us instead of 61 + 5, one of 1213x1617 pixels 36 + 15 instead of 105 + 15.
constexpr int kSlotRunUp = kSlotRounds, kSlotThreads = ((kSlotSubs + kSlotRunUp) * 6 + 31) / 32 * 32;

struct SlotShared {
    uint16_t state[kSlotSubs + kSlotRunUp + 1][kSlotStates]; // entry states, relative to the subsequence's start
    uint16_t exit[kSlotSubs + kSlotRunUp][kSlotStates];      // ... and what they lead to
    uint16_t blocks[kSlotSubs + kSlotRunUp][kSlotStates];
    uint8_t next[kSlotSubs + kSlotRunUp][kSlotStates];       // place of `exit` among the next subsequence's states, or kSlotMiss
    int count[kSlotSubs + kSlotRunUp + 1];
    uint16_t list[kSlotThreads]; // (subsequence << 4 | state) to decode
    int n_list;
    int warp[kSlotThreads / 32];
    uint32_t mark[2];
};

// Place of state e among the first n of `states` (two per word), or kSlotMiss.
__device__ __forceinline__ uint32_t find_state(const uint16_t *states, int n, uint32_t e) {
    const uint32_t *pairs = reinterpret_cast<const uint32_t *>(states);
    uint32_t found = kSlotMiss;
#pragma unroll
    for (int k = kSlotStates / 2 - 1; k >= 0; k--) {
        const uint32_t p = pairs[k];
        if ((p >> 16) == e && 2 * k + 1 < n) found = 2 * k + 1;
        if ((p & 0xffff) == e && 2 * k < n) found = 2 * k;
    }
    return found;
}

// One CTA per segment, at first one thread per (subsequence, slot).  Bound by the chain of look-ups, at one or
// two CTAs per SM.
__global__ void __launch_bounds__(kSlotThreads)
scan_slots_kernel(const ImageDesc *__restrict__ descs, const uint2 *__restrict__ segs, const uint8_t *__restrict__ blob,
                  const HuffTable *__restrict__ huff, EntropyScratch scratch, int table_slots) {
    extern __shared__ __align__(16) unsigned char s_dyn[];
    __shared__ __align__(16) SlotShared sh;
    next_may_begin();
    await_previous();
    const Team<1, kSlotThreads> team;
    const int tid = team.tid;
    Tables *tables = reinterpret_cast<Tables *>(s_dyn);
    unsigned char *buf = s_dyn + tables_bytes(table_slots);
    const uint2 which = segs[blockIdx.x];
    const uint32_t j = which.y;
    const ImageDesc &d = descs[which.x];
    const uint32_t S = d.subseq_bits, R = d.seg_raw, warm = j == 0 ? 0 : d.seg_warm;
    const int bpm = d.bpm;
    load_tables(tables, d, huff);
    const uint32_t scan_len = d.scan_len, own0 = j * R, own1 = min(own0 + R, scan_len);
    const uint32_t raw0 = own0 - min(own0, warm * (S >> 3)), raw1 = min(own1 + kSegOverlap, scan_len);
    const uint32_t at[2] = {own0 - raw0, own1 - raw0};
    const uint32_t kept = unstuff(team, buf, blob + d.payload_off + d.scan_off + raw0, raw1 - raw0, raw0 == 0, at, sh.warp, sh.mark);
    const uint32_t own_bit = at[0] == 0 ? 0 : sh.mark[0] * 8, own_end = own1 == raw1 ? kept * 8 : sh.mark[1] * 8;
    {
        uint4 *dst = reinterpret_cast<uint4 *>(scratch.clean + d.clean_off + (size_t)j * d.seg_stride);
        for (uint32_t k = tid; k < (kept + 64 + 15) / 16; k += kSlotThreads) dst[k] = reinterpret_cast<const uint4 *>(buf)[k];
    }
    const size_t seg = (size_t)d.seg_first + j;
    const int n_own = (int)((own_end - own_bit + S - 1) / S), n_subs = (int)warm + n_own;
    auto start_of = [&](int t) -> int { return (int)own_bit + (t - (int)warm) * (int)S; };
    // ---- the guesses: every slot (the scan itself begins with slot 0)
    for (int k = tid; k < (n_subs + 1) * kSlotStates; k += kSlotThreads) {
        const int c = k % kSlotStates;
        sh.state[k / kSlotStates][c] = (uint16_t)pack(Cursor{0, c < bpm ? c : 0, 0}, 0);
        if (k / kSlotStates < n_subs) sh.next[k / kSlotStates][c] = kSlotMiss;
    }
    for (int t = tid; t <= n_subs; t += kSlotThreads) sh.count[t] = j == 0 && t == 0 ? 1 : (t == n_subs ? 0 : bpm);
    copies_wait();
    __syncthreads();
    auto decode = [&](int t, int i) {
        // (the run-up lacks the bytes that its stuffing took: its first subsequence is shorter)
        const uint32_t start = (uint32_t)max(start_of(t), 0), end = (uint32_t)max(min(start_of(t + 1), (int)own_end), 0);
        Cursor cur = unpack(sh.state[t][i], start);
        sh.blocks[t][i] = (uint16_t)walk<kNothing>(buf, cur, end, tables, d, huff);
        sh.exit[t][i] = (uint16_t)pack(cur, end);
    };
    int lo = 0; // states of this thread's subsequence that were decoded in the last round: [lo, hi)
    for (int round = 0; round < kSlotRounds; round++) {
        int sub = tid / bpm, which_state = tid - sub * bpm;
        bool live = sub < n_subs && which_state < sh.count[min(sub, n_subs)];
        if (round > 0) {
            live = tid < sh.n_list;
            sub = live ? sh.list[tid] >> 4 : 0;
            which_state = live ? sh.list[tid] & (kSlotStates - 1) : 0;
        }
        if (live) decode(sub, which_state);
        __syncthreads();
        if (tid == 0) sh.n_list = 0;
        __syncthreads();
        // thread t looks its subsequence's new exits up among the next one's states; the unknown ones join them
        const int t = tid;
        int first_new = 0, n_new = 0;
        if (t < n_subs) {
            const int hi = sh.count[t];
            // (count[t] may grow below, by the thread before this one: a barrier lies between)
            int n = sh.count[t + 1];
            first_new = n;
            for (int i = lo; i < hi; i++) {
                const uint32_t e = sh.exit[t][i];
                uint32_t at_ = find_state(sh.state[t + 1], n, e);
                if (at_ == kSlotMiss && n < kSlotStates - 1 && round + 1 < kSlotRounds && t + 1 < n_subs) {
                    at_ = n;
                    sh.state[t + 1][n++] = (uint16_t)e;
                }
                sh.next[t][i] = (uint8_t)at_;
            }
            lo = hi;
            n_new = n - first_new;
        }
        __syncthreads();
        if (n_new > 0) {
            sh.count[t + 1] = first_new + n_new;
            const int base = atomicAdd(&sh.n_list, n_new); // (at most one per state decoded in this round, hence per thread)
            for (int k = 0; k < n_new; k++) sh.list[base + k] = (uint16_t)((t + 1) << 4 | (first_new + k));
        }
        __syncthreads();
        if (sh.n_list == 0) break;
    }
    // ---- what the segment makes of every state its first own subsequence may begin in
    SlotTables *out = scratch.slots + (d.slots - 1) + j;
    if (tid < 32) {
        SlotMap map{kNoState, 0};
        const bool wanted = n_own > 0 && tid < min(sh.count[warm], kSlotStates);
        auto follow = [&](int i, bool repair) {
            const int entry = i;
            uint32_t total = 0;
            int t = (int)warm;
            for (; t + 1 < n_subs; t++) {
                total += sh.blocks[t][i];
                int to = sh.next[t][i];
                if (to == kSlotMiss && repair && sh.count[t + 1] < kSlotStates - 1) {
                    to = sh.count[t + 1]++;
                    sh.state[t + 1][to] = sh.exit[t][i];
                    decode(t + 1, to);
                    sh.next[t + 1][to] = t + 2 < n_subs ? (uint8_t)find_state(sh.state[t + 2], sh.count[t + 2], sh.exit[t + 1][to]) : (uint8_t)kSlotMiss;
                    sh.next[t][i] = (uint8_t)to;
                }
                if (to == kSlotMiss) return;
                i = to;
            }
            map = SlotMap{sh.state[warm][entry], sh.exit[t][i] | (total + sh.blocks[t][i]) << 16};
        };
        if (wanted) follow(tid, false);
        // Which of them the run-up's guesses lead to: the real one is nearly always among these few, so where
        // one of these meets an unknown state a thread decodes on until it is in step.
        int i = tid;
        bool reached = tid < sh.count[0];
        for (int t = 0; t < (int)warm && reached; t++) {
            i = sh.next[t][i];
            reached = i != kSlotMiss;
        }
        const uint32_t unresolved = __ballot_sync(0xffffffffu, wanted && map.from == kNoState);
        for (uint32_t left = unresolved & __reduce_or_sync(0xffffffffu, reached ? 1u << i : 0u); left; left &= left - 1) {
            if (tid == __ffs(left) - 1) follow(tid, true);
            __syncwarp();
        }
        if (tid < kSlotStates) out->map[tid] = map;
    }
    __syncthreads();
    for (int k = tid; k < n_own * kSlotStates; k += kSlotThreads) {
        const int t = k / kSlotStates, i = k % kSlotStates;
        out->info[t][i] = i < sh.count[t + warm] ? sh.state[t + warm][i] | (uint32_t)sh.blocks[t + warm][i] << 16 : kNoState;
        out->next[t][i] = sh.next[t + warm][i];
    }
    if (tid == 0) scratch.meta[seg] = SegMeta{own_bit, own_end, kept, 0, 0};
}

// One CTA per image: follows the real state from segment to segment through their maps.  Many segments are
// shared out: every warp composes the maps of a run of them for all 16 states, the first warp chains
// the runs, then every warp follows the real state through its own run.  Where the real state is not
// among a segment's (one in several thousand), one thread decodes that segment.
constexpr int kChainThreads = 1024;
__global__ void __launch_bounds__(kChainThreads)
scan_chain_kernel(const ImageDesc *__restrict__ descs, const int32_t *__restrict__ list, const HuffTable *__restrict__ huff,
                  EntropyScratch scratch, int map_slots) {
    extern __shared__ __align__(16) SlotMap s_maps[]; // [segment][state]
    __shared__ uint32_t s_entry[kChainThreads / 32 + 1];
    __shared__ SlotMap s_run[kChainThreads / 32][kSlotStates]; // (state, or kNoState; state behind the run)
    __shared__ uint8_t s_done[kChainThreads / 32];
    next_may_begin();
    await_previous();
    const ImageDesc &d = descs[list[blockIdx.x]];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, n_seg = (int)d.seg_count;
    SlotTables *tabs = scratch.slots + (d.slots - 1);
    SegMeta *meta = scratch.meta + d.seg_first;
    const uint32_t S = d.subseq_bits;
    const bool staged = n_seg <= map_slots;
    if (staged)
        for (int k = tid; k < n_seg * kSlotStates; k += blockDim.x) s_maps[k] = tabs[k / kSlotStates].map[k % kSlotStates];
    __syncthreads();
    auto map_of = [&](int k, int i) -> SlotMap { return staged ? s_maps[k * kSlotStates + i] : tabs[k].map[i]; };
    // The real state `state` through segment k, by a whole warp: which of its states it is, and what is behind it.
    auto follow = [&](int k, uint32_t state) -> uint32_t {
        const SlotMap m = map_of(k, lane & (kSlotStates - 1));
        const uint32_t who = __ballot_sync(0xffffffffu, m.from == state) & ((1u << kSlotStates) - 1);
        uint32_t behind;
        if (who != 0) {
            const int src = __ffs(who) - 1;
            behind = __shfl_sync(0xffffffffu, m.to, src);
            if (lane == 0) {
                meta[k].entry = src;
                meta[k].blocks = behind >> 16;
            }
        } else {
            if (lane == 0) { // subsequence by subsequence; those with an unknown state are decoded here, into the last place
                const SegMeta sm = meta[k];
                SlotTables &tab = tabs[k];
                const uint32_t *words = reinterpret_cast<const uint32_t *>(scratch.clean + d.clean_off + (size_t)k * d.seg_stride);
                const int n_own = (int)((sm.own_end - sm.own_bit + S - 1) / S);
                uint32_t at = state, blocks = 0, from = kSlotMiss;
                uint32_t i = kSlotMiss; // place of `at` among the states of subsequence t
                for (int t = 0; t < n_own; t++) {
                    const uint32_t start = sm.own_bit + (uint32_t)t * S, end = min(start + S, sm.own_end);
                    if (i == kSlotMiss)
                        for (uint32_t c = 0; c < kSlotStates - 1 && i == kSlotMiss; c++)
                            if ((tab.info[t][c] & 0xffff) == at) i = c;
                    const bool known = i != kSlotMiss;
                    if (!known) i = kSlotStates - 1;
                    if (t == 0) meta[k].entry = i;
                    else tab.next[t - 1][from] = (uint8_t)i;
                    uint32_t to = known && t + 1 < n_own ? tab.next[t][i] : kSlotMiss;
                    if (to == kSlotMiss) {
                        Cursor cur = unpack(at, start);
                        const uint32_t done = walk_plain<kNothing>(words, cur, end, d, huff, nullptr, 0, 0, nullptr);
                        tab.info[t][i] = at | done << 16;
                        at = pack(cur, end);
                        blocks += done;
                    } else {
                        blocks += tab.info[t][i] >> 16;
                        at = tab.info[t + 1][to] & 0xffff;
                    }
                    from = i;
                    i = to;
                }
                if (n_own == 0) meta[k].entry = 0;
                meta[k].blocks = blocks;
                behind = at;
            }
            behind = __shfl_sync(0xffffffffu, behind, 0);
        }
        return behind & 0xffff;
    };
    const int warps = blockDim.x / 32, run = (n_seg + warps - 1) / warps, first = warp * run, last = min(first + run, n_seg);
    if (warps == 1) {
        uint32_t state = 0;
        for (int k = 0; k < n_seg; k++) state = follow(k, state);
        return;
    }
    if (first < last && lane < kSlotStates) {
        const SlotMap m = map_of(first, lane);
        uint32_t at = m.from == kNoState ? kNoState : m.to & 0xffff;
        for (int k = first + 1; k < last; k++) {
            uint32_t to = kNoState;
            for (int i = 0; i < kSlotStates; i++) {
                const SlotMap o = map_of(k, i);
                if (o.from == at && at != kNoState) to = o.to & 0xffff;
            }
            at = to;
        }
        s_run[warp][lane] = SlotMap{at == kNoState ? kNoState : m.from, at};
    }
    if (lane == 0) s_done[warp] = 0;
    __syncthreads();
    if (warp == 0) {
        uint32_t state = 0;
        for (int w = 0; w < warps && w * run < n_seg; w++) {
            if (lane == 0) s_entry[w] = state;
            const SlotMap m = s_run[w][lane & (kSlotStates - 1)];
            const uint32_t who = __ballot_sync(0xffffffffu, m.from == state) & ((1u << kSlotStates) - 1);
            if (who != 0) {
                state = __shfl_sync(0xffffffffu, m.to, __ffs(who) - 1);
            } else { // the run cannot be skipped
                for (int k = w * run; k < min((w + 1) * run, n_seg); k++) state = follow(k, state);
                if (lane == 0) s_done[w] = 1;
            }
        }
    }
    __syncthreads();
    if (first < last && !s_done[warp]) {
        uint32_t state = s_entry[warp];
        for (int k = first; k < last; k++) state = follow(k, state);
    }
}

// Where the blocks of a segment are, and their DC values.  SLOTS: of the samples decoded from every slot, by
// walking every subsequence once more from its real state, its stream in shared memory.  Otherwise the records
// say it already, unless a subsequence has more blocks than they hold (or there are none): the segments of
// such a CTA are walked in global memory.  (Only the warps', or the subsequences themselves: the CTA takes no less time then, see
// record_room.)
template <bool SLOTS>
constexpr int kIndexTeam = SLOTS ? kSlotSubs : kSegSubs;
template <int TEAMS, bool SLOTS>
__global__ void __launch_bounds__(kIndexTeam<SLOTS> * TEAMS, TEAMS == 4 ? 2 : 1)
scan_index_kernel(const ImageDesc *__restrict__ descs, const uint2 *__restrict__ segs, int n_segs, const HuffTable *__restrict__ huff,
                  EntropyScratch scratch, int32_t *__restrict__ status, uint8_t *__restrict__ index_pool,
                  unsigned long long *__restrict__ index_stats, int table_slots, uint32_t buf_bytes) {
    constexpr int kThreads = kIndexTeam<SLOTS>;
    extern __shared__ __align__(16) unsigned char s_dyn[];
    __shared__ int s_warps[TEAMS][kThreads / 32];
    __shared__ uint32_t s_lasts[TEAMS];
    __shared__ __align__(16) uint16_t s_dc[kMaxComponents][1 << kHuffBits]; // first level of the DC tables
    next_may_begin();
    const Team<TEAMS, kThreads> team;
    const int tid = team.tid;
    int *s_warp = s_warps[team.index];
    uint32_t &s_last = s_lasts[team.index];
    Tables *tables = reinterpret_cast<Tables *>(s_dyn);
    unsigned char *buf = s_dyn + tables_bytes(table_slots) + team.index * buf_bytes;
    const int mine = blockIdx.x * TEAMS + team.index;
    const uint2 which = segs[min(mine, n_segs - 1)];
    const int img = (int)which.x;
    const uint32_t j = which.y;
    const ImageDesc &d = descs[img];
    const size_t seg = (size_t)d.seg_first + j;
    if (SLOTS) load_tables(tables, d, huff);
    for (int t = 0; t < d.n_dc_tab; t++) { // (the same whichever team's sample they are taken from)
        const uint4 *src = reinterpret_cast<const uint4 *>(huff[d.tab_id[t]].look);
        for (int k = threadIdx.x; k < (1 << kHuffBits) / 8; k += blockDim.x) reinterpret_cast<uint4 *>(s_dc[t])[k] = src[k];
    }
    await_previous();
    const SegMeta m = scratch.meta[seg];
    const uint32_t S = d.subseq_bits, nblocks = d.nblocks;
    const int n_own = (int)((m.own_end - m.own_bit + S - 1) / S);
    uint32_t info = 0, n_rec = 0;
    bool walks = SLOTS;
    if (!SLOTS) {
        if (tid < n_own) {
            info = scratch.sub_info[seg * kSegSubs + tid];
            n_rec = (info >> 16) + (scratch.sub_exit[seg * kSegSubs + tid] >> 8 ? 1 : 0) - ((info >> 8 & 63) ? 1 : 0);
        }
        walks = __syncthreads_or(tid < n_own && (!scratch.records || n_rec >= d.rec_room)) != 0;
        if (walks) load_tables(tables, d, huff);
    }
    copies_wait();
    __syncthreads();
    if (TEAMS > 1 && mine >= n_segs) return;
    uint32_t *pos = scratch.pos + d.block_base;
    int16_t *dc = scratch.dc + d.block_base;

    uint32_t base = 0; // blocks before this segment
    if (j > 0) {
        int before = 0, all;
        for (uint32_t k = tid; k < j; k += kThreads) before += (int)scratch.meta[d.seg_first + k].blocks;
        team_scan(team, before, s_warp, all);
        base = (uint32_t)all;
    }
    if (SLOTS) { // one thread follows the real state from subsequence to subsequence
        const SlotTables *t = scratch.slots + (d.slots - 1) + j;
        uint8_t *next = buf, *path = buf + sizeof(t->next); // (the buffer is free until the stream arrives)
        for (int k = tid; k < (int)(sizeof(t->next) / 16); k += kThreads) reinterpret_cast<uint4 *>(next)[k] = reinterpret_cast<const uint4 *>(t->next)[k];
        team.sync();
        if (tid == 0)
            for (int k = 0, i = (int)m.entry; k < n_own; k++) {
                path[k] = (uint8_t)i;
                i = next[k * kSlotStates + i] & (kSlotStates - 1);
            }
        team.sync();
        if (tid < n_own) info = t->info[tid][path[tid]];
        team.sync();
    }
    int sums[3] = {0, 0, 0};
    if (base < nblocks) { // (uniform) otherwise the crop needs nothing of this segment
        const unsigned char *stream = scratch.clean + d.clean_off + (size_t)j * d.seg_stride;
        const uint32_t skip = SLOTS ? m.own_bit >> 7 : 0; // vectors of the run-up
        if (SLOTS) {
            for (uint32_t k = skip + tid; k < (m.bytes + 64 + 15) / 16; k += kThreads)
                copy16_async(buf + (size_t)(k - skip) * 16, reinterpret_cast<const uint4 *>(stream) + k);
            stream = buf;
        }
        if (SLOTS) copies_wait();
        int in_segment;
        const uint32_t first = base + (uint32_t)team_scan(team, (int)(info >> 16), s_warp, in_segment); // (and a barrier for the copies)
        const uint32_t bias = j * d.seg_stride * 8 + skip * 128; // position of the walked stream's bit 0
        const uint32_t start = m.own_bit - skip * 128 + (uint32_t)tid * S;
        const uint32_t end = min(start + S, m.own_end - skip * 128);
        Cursor cur = unpack(info & 0xffff, start);
        const uint32_t b0 = first + (cur.z != 0 ? 1 : 0); // the block in progress belongs to the subsequence it began in
        uint32_t b1 = b0;
        int sum[3] = {0, 0, 0};
        const uint32_t luma = d.ncomp == 1 ? 1 : d.hs * d.vs, bpm = d.bpm;
        const uint32_t tab = d.dc_tab[0] | (uint32_t)d.dc_tab[1] << 8 | (uint32_t)d.dc_tab[2] << 16;
        if (tid < n_own && first < nblocks && cur.p < end) {
            const uint16_t *rec = SLOTS ? nullptr : records_of(scratch, d, j, (uint32_t)tid);
            if (walks) {
                const uint32_t done = walk<kPositions, !SLOTS>(stream, cur, end, tables, d, huff, pos, b0, nblocks);
                n_rec = done + (cur.z != 0 ? 1 : 0) - (b0 - first);
            }
            b1 = min(b0 + n_rec, nblocks);
            // the DC symbols of the blocks found: positions move on to the first AC symbol, values count
            // from the thread's first block.  Four blocks' words are fetched at a time.
            uint32_t slot = b0 % bpm;
            for (uint32_t b = b0; b < b1; b += 4) {
                uint32_t p[4], w[4];
                if (walks) {
#pragma unroll
                    for (int k = 0; k < 4; k++) p[k] = b + k < b1 ? pos[b + k] : start;
                } else {
                    const uint2 r = *reinterpret_cast<const uint2 *>(rec + (b - b0));
                    const uint32_t low[4] = {r.x & 0xffff, r.x >> 16, r.y & 0xffff, r.y >> 16};
#pragma unroll
                    for (int k = 0; k < 4; k++) p[k] = b + k < b1 ? start + ((low[k] - start) & 0xffff) : start;
                }
#pragma unroll
                for (int k = 0; k < 4; k++) {
                    const uint32_t *at = reinterpret_cast<const uint32_t *>(stream) + (p[k] >> 5);
                    w[k] = __funnelshift_l(at[1], at[0], p[k]);
                }
#pragma unroll
                for (int k = 0; k < 4; k++) {
                    if (b + k >= b1) break;
                    const int comp = slot < luma ? 0 : (int)(slot - luma) + 1, t = tab >> 8 * comp & 255;
                    uint32_t e = s_dc[t][w[k] >> (32 - kHuffBits)];
                    if (e & kHuffLong) e = huff_long(huff + d.tab_id[t], e, w[k]);
                    const uint32_t n = e & 31, size = (e >> 5) & 15;
                    const int v = size ? huff_value(w[k], n, size) : 0;
                    sum[0] += comp == 0 ? v : 0;
                    sum[1] += comp == 1 ? v : 0;
                    sum[2] += comp == 2 ? v : 0;
                    pos[b + k] = bias + p[k] + n;
                    dc[b + k] = (int16_t)(comp == 0 ? sum[0] : (comp == 1 ? sum[1] : sum[2]));
                    slot = slot + 1 == bpm ? 0 : slot + 1;
                }
            }
        }
        // what the segment holds before the thread's first block
        int before[3];
#pragma unroll
        for (int c = 0; c < 3; c++) before[c] = c < d.ncomp ? team_scan(team, sum[c], s_warp, sums[c]) : 0;
        uint32_t slot = b0 % bpm;
        for (uint32_t b = b0; b < b1; b += 4) {
            int v[4];
#pragma unroll
            for (int k = 0; k < 4; k++) v[k] = b + k < b1 ? dc[b + k] : 0;
#pragma unroll
            for (int k = 0; k < 4; k++) {
                if (b + k < b1) dc[b + k] = (int16_t)(v[k] + (slot < luma ? before[0] : (slot == luma ? before[1] : before[2])));
                slot = slot + 1 == bpm ? 0 : slot + 1;
            }
        }
    }
    if (tid == 0) {
        int32_t *o = scratch.seg_dc + seg * 4;
        o[0] = sums[0];
        o[1] = sums[1];
        o[2] = sums[2];
    }
    const bool record = index_pool != nullptr && (d.index_use & 2) != 0 && d.host_status == 0 &&
                        !index_entry_valid(reinterpret_cast<const DecodeIndexHeader *>(index_pool + d.index_off), d);
    if (record) {
        uint32_t *dst = reinterpret_cast<uint32_t *>(index_pool + d.index_off + sizeof(DecodeIndexHeader)) + (size_t)j * d.seg_lanes;
        if (tid < (int)d.seg_lanes) dst[tid] = info;
    }
    // ---- the CTA that finishes an image last turns the segments' DC sums into sums before them
    __threadfence();
    team.sync();
    if (tid == 0) s_last = atomicInc(&scratch.done[img], d.seg_count - 1) == d.seg_count - 1 ? 1 : 0; // wraps back to 0
    team.sync();
    if (!s_last) return;
    __threadfence();
    int carry[3] = {0, 0, 0}, blocks = 0;
    for (uint32_t k0 = 0; k0 < d.seg_count; k0 += kThreads) {
        const uint32_t k = k0 + tid;
        int32_t *o = scratch.seg_dc + ((size_t)d.seg_first + k) * 4;
        int n;
        team_scan(team, k < d.seg_count ? (int)__ldcg(&scratch.meta[d.seg_first + k].blocks) : 0, s_warp, n);
        blocks += n;
#pragma unroll
        for (int c = 0; c < 3; c++) {
            int all;
            const int e = team_scan(team, k < d.seg_count ? __ldcg(o + c) : 0, s_warp, all);
            if (k < d.seg_count) o[c] = carry[c] + e;
            carry[c] += all;
        }
    }
    const bool complete = (uint32_t)blocks >= nblocks;
    for (uint32_t b = (uint32_t)blocks + tid; b < nblocks; b += kThreads) { // a scan that ended early
        pos[b] = kNoBlock;
        dc[b] = 0;
    }
    if (tid == 0) {
        status[img] = d.host_status != 0 ? (int)d.host_status : (complete ? 0 : (int)kErrData);
        if (record) {
            DecodeIndexHeader *h = reinterpret_cast<DecodeIndexHeader *>(index_pool + d.index_off);
            h->scan_len = d.scan_len;
            h->subseq_bits = d.subseq_bits;
            h->segments = d.seg_count;
            __threadfence();
            h->magic = kDecodeIndexMagic;
            if (index_stats) atomicAdd(index_stats + 1, 1ull);
        }
    }
}

// ------------------------------------------------------------------------------------------
// Streams with restart markers (DRI != 0): every restart interval is an independent piece of the
// stream (byte aligned, DC predictors reset, T.81 F.2.1.3.1 / E.2.4), so no speculation is
// needed: the unstuffing pass also removes the RSTn markers and records where each interval
// starts, then one thread walks one interval and records its blocks with their final DC values.
// One CTA per image.
constexpr int kRestartThreads = 256;
__global__ void __launch_bounds__(kRestartThreads)
scan_restart_kernel(const ImageDesc *__restrict__ descs, const int32_t *__restrict__ list, const uint8_t *__restrict__ blob,
                    const HuffTable *__restrict__ huff, EntropyScratch scratch, int32_t *__restrict__ status) {
    __shared__ int s_warp[kRestartThreads / 32];
    __shared__ int s_bad;
    const int img = list[blockIdx.x];
    const ImageDesc &d = descs[img];
    const int tid = threadIdx.x, bpm = d.bpm, luma = d.ncomp == 1 ? 1 : d.hs * d.vs;
    if (tid == 0) s_bad = 0;

    // ---- remove byte stuffing and restart markers; note where every interval starts
    const uint32_t scan_len = d.scan_len;
    const uint8_t *scan = blob + d.payload_off + d.scan_off;
    uint8_t *cl = scratch.clean + d.clean_off;
    uint32_t *starts = reinterpret_cast<uint32_t *>(scratch.clean + d.rst_off); // byte offsets in the clean stream
    const int nmcu_all = d.mcus_x * d.mcus_y, ri = d.restart_interval;
    const uint32_t cap = (uint32_t)((nmcu_all + ri - 1) / ri) + 1; // entries the table holds
    if (tid == 0) starts[0] = 0;
    uint32_t clean_len = 0, n_mark = 0;
    for (uint32_t base = 0; base < scan_len; base += kRestartThreads * 16) {
        const uint32_t my = base + tid * 16;
        uint8_t b[17];
        uint32_t keep = 0, marks = 0;
        int prev = (my > 0 && my <= scan_len) ? scan[my - 1] : 0;
#pragma unroll
        for (int i = 0; i < 17; i++) b[i] = my + i < scan_len ? scan[my + i] : 0;
#pragma unroll
        for (int i = 0; i < 16; i++) {
            const uint32_t at = my + i;
            const bool rst_ff = b[i] == 0xFF && (b[i + 1] & 0xF8) == 0xD0;
            const bool rst_code = prev == 0xFF && (b[i] & 0xF8) == 0xD0;
            const bool stuffing = b[i] == 0 && prev == 0xFF;
            if (at < scan_len && !rst_ff && !rst_code && !stuffing) keep |= 1u << i;
            if (at < scan_len && rst_code) marks |= 1u << i;
            prev = b[i];
        }
        int total, mtotal;
        auto sync = [] { __syncthreads(); };
        const int off = scan_exclusive(__popc(keep), tid, kRestartThreads / 32, s_warp, total, sync);
        const int moff = scan_exclusive(__popc(marks), tid, kRestartThreads / 32, s_warp, mtotal, sync);
        uint32_t o = clean_len + off, m = n_mark + moff;
#pragma unroll
        for (int i = 0; i < 16; i++) {
            if (keep & (1u << i)) cl[(o++) ^ 3u] = b[i];
            if (marks & (1u << i)) {
                m++;
                if (m < cap) starts[m] = o; // interval m begins with the next byte kept
            }
        }
        clean_len += total;
        n_mark += mtotal;
    }
    if (tid < 64) cl[(clean_len + tid) ^ 3u] = 0;

    // ---- one thread per restart interval
    uint32_t *pos = scratch.pos + d.block_base;
    int16_t *dc = scratch.dc + d.block_base;
    for (uint32_t k = tid; k < d.nblocks; k += kRestartThreads) {
        pos[k] = kNoBlock;
        dc[k] = 0;
    }
    __syncthreads();
    const uint32_t *words = reinterpret_cast<const uint32_t *>(cl);
    const int nmcu = d.mcus_x * d.mcu_rows; // the crop may need only the upper rows
    const uint32_t needed = (uint32_t)((nmcu + ri - 1) / ri);
    const uint32_t found = n_mark + 1 < cap ? n_mark + 1 : cap;
    if (found < needed && tid == 0) s_bad = 1; // fewer intervals than the frame needs
    for (uint32_t k = tid; k < needed && k < found; k += kRestartThreads) {
        const int first = (int)k * ri, count = nmcu - first < ri ? nmcu - first : ri;
        const uint32_t limit = (k + 1 < found ? starts[k + 1] : clean_len) * 8;
        uint32_t blk = (uint32_t)(first * bpm);
        const uint32_t end_blk = blk + (uint32_t)(count * bpm);
        int pred[3] = {0, 0, 0}, z = 0;
        int c = 0;
        uint32_t p = starts[k] * 8;
        while (blk < end_blk) {
            if (p >= limit) { // the interval's bits ran out
                s_bad = 1;
                break;
            }
            const uint32_t w = __funnelshift_l(words[(p >> 5) + 1], words[p >> 5], p);
            const int comp = c < luma ? 0 : c - luma + 1;
            const HuffTable *table = huff + d.tab_id[z ? d.ac_tab[comp] : d.dc_tab[comp]];
            uint32_t e = table->look[w >> (32 - kHuffBits)];
            if (e & kHuffLong) e = huff_long(table, e, w);
            if (z == 0) {
                const uint32_t n = e & 31, size = (e >> 5) & 15;
                const int v = size ? huff_value(w, n, size) : 0;
                pred[0] += comp == 0 ? v : 0;
                pred[1] += comp == 1 ? v : 0;
                pred[2] += comp == 2 ? v : 0;
                pos[blk] = p + n;
                dc[blk] = (int16_t)(comp == 0 ? pred[0] : (comp == 1 ? pred[1] : pred[2]));
            }
            p += e & 31;
            z += (int)(e >> 9);
            if (z >= 64) {
                z = 0;
                blk++;
                c = c + 1 == bpm ? 0 : c + 1;
            }
        }
    }
    __syncthreads();
    if (tid == 0) status[img] = d.host_status != 0 ? (int)d.host_status : (s_bad ? (int)kErrData : 0);
}

} // namespace

// Run-up before a subsequence, in bits.  Shorter ones leave more to repair: 1600 / 800 bits 244 us instead of 229 alone and
// 370 instead of 368 as one of four in flight (1024 photographs), 1280 / 640 270 and 372.
constexpr uint32_t kRunUp = 1920, kRunUpFewSlots = 960;

uint32_t subseq_target(uint64_t total_bits) {
    // A subsequence costs a run-up on top of its own length, so long ones are less work; short ones are a shorter chain,
    // which decides while few bits leave the GPU mostly idle.  Batches of 80 Mbit, alone / as one of four in flight, all
    // kernels: 352 / 211 us with 200 subsequences per SM, 355 / 208 with 320, 390 / 226 with 480.  Below some 32 Mbit, where the
    // run-up is longer than they are, fewer do better: 18 Mbit 196 / 93 with 256 and 202 / 106 with 320, 27 Mbit 214 / 119 and
    // 241 / 134, 30 Mbit 247 / 120 and 239 / 130, but 44 Mbit 280 / 189 and 278 / 190, 53 Mbit of 4:4:4 222 / 123 and 216 / 123.
    const uint64_t t = total_bits / (148 * (total_bits <= (32u << 20) ? 256 : 320));
    return (uint32_t)(t < 256 ? 256 : (t > kMaxSubseqBits ? kMaxSubseqBits : (t + 31) / 32 * 32));
}

ScanLayout layout_scan(uint32_t scan_len, uint32_t target_bits, int bpm, bool local_repair, bool indexed) {
    ScanLayout l{};
    const uint64_t bits = (uint64_t)scan_len * 8, target = target_bits;
    auto up = [](uint64_t a, uint64_t b) { return (a + b - 1) / b; };
    l.seg_run_up = bpm > 3 ? kRunUp : kRunUpFewSlots;
    l.seg_count = 1;
    uint64_t own = kSegSubs; // subsequences of a segment
    if (local_repair) {
        if (bits > own * target) {
            // (8 kbit before a segment: all but one in 10^4 of its first subsequences begin in the real state then)
            l.seg_warm = (uint32_t)up(8192 - l.seg_run_up, target);
            own -= l.seg_warm;
            l.seg_count = (uint32_t)up(bits, own * target);
        }
    } else { // two warps at most (128 of them share the SM's memory out worse: 64 images of 14 Mbit 696 us instead of 653)
        own = indexed ? kSegSubs : 64;
        // (with a decode index a scan that one segment of somewhat longer subsequences takes is not cut in two: 1024 photographs of
        // 145 kbit from their entries 118 us in one segment each, 128 in two of 96 subsequences)
        l.seg_count = indexed && bits <= own * std::min<uint64_t>(target + target / 4, kMaxSubseqBits) ? 1 : (uint32_t)up(bits, own * target);
        if (l.seg_count < 1) l.seg_count = 1;
        const uint64_t lanes = 32 * up(bits, 32 * target * l.seg_count);
        own = lanes < 32 ? 32 : (lanes > own ? own : lanes);
    }
    l.subseq_bits = (uint32_t)up(up(bits, own * l.seg_count), 32) * 32;
    if (l.subseq_bits < 128) l.subseq_bits = 128;
    l.seg_raw = (uint32_t)own * l.subseq_bits / 8;
    l.seg_lanes = (uint32_t)own;
    l.seg_count = scan_len ? (scan_len + l.seg_raw - 1) / l.seg_raw : 1;
    l.seg_stride = (((uint32_t)own + l.seg_warm) * l.subseq_bits + l.seg_run_up) / 8 + kSegOverlap + 64 + 31;
    l.seg_stride = l.seg_stride / 16 * 16;
    return l;
}

ScanLayout layout_scan_slots(uint32_t scan_len) {
    ScanLayout l{};
    const uint64_t bits = (uint64_t)scan_len * 8, own = (uint64_t)kSlotSubs * kSlotBits;
    l.seg_count = (uint32_t)((bits + own - 1) / own);
    if (l.seg_count < 1) l.seg_count = 1;
    l.subseq_bits = (uint32_t)((bits + kSlotSubs * l.seg_count - 1) / (kSlotSubs * l.seg_count) + 31) / 32 * 32;
    // (shorter ones leave real states unknown after the last round, which one thread then decodes one by one:
    // eight images of 64x64 pixels 133 us with 288 bits, 69 with 384)
    if (l.subseq_bits < 384) l.subseq_bits = 384;
    l.seg_warm = kSlotRunUp;
    l.seg_raw = kSlotSubs * l.subseq_bits / 8;
    l.seg_lanes = kSlotSubs;
    l.seg_count = scan_len ? (scan_len + l.seg_raw - 1) / l.seg_raw : 1;
    l.seg_stride = ((kSlotSubs + kSlotRunUp) * l.subseq_bits / 8 + kSegOverlap + 64 + 31) / 16 * 16;
    return l;
}

void launch_entropy_decode(const ImageDesc *descs, const EntropyWork &work, const uint8_t *blob, const HuffTable *huff,
                           const EntropyScratch &scratch, int32_t *status, uint8_t *index_pool, unsigned long long *index_stats,
                           cudaStream_t stream) {
    const int n_segs = work.n_guess + work.n_slots;
    if (n_segs > 0) {
        const uint32_t buf = (uint32_t)stream_bytes(work.max_raw);
        const int tables = work.max_tables;
        const bool early = work.early();
        auto allow = [](auto kernel, size_t smem) { cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem); };
        // With enough segments to fill every SM four teams share a set of tables: eight segments of up to
        // 22 KB fit an SM then, instead of five.  (Segments that are repaired on the spot keep to themselves; in slot mode it is the
        // index kernel's: 1024 images of 40x46 pixels 132 us instead of 135 to 137, 3000 of 24x30 286 instead of 288 to 292.)
        const int slot_teams = work.alike && n_segs >= 148 * 5 ? 4 : 1, teams = work.local_repair ? 1 : slot_teams;
        const size_t smem = tables_bytes(tables) + (size_t)teams * buf;
        if (work.n_guess > 0) {
            const int grid = (work.n_guess + teams - 1) / teams;
            auto run = [&](auto kernel) {
                allow(kernel, smem);
                kernel<<<grid, kThreads * teams, smem, stream>>>(descs, work.segs, work.n_guess, blob, huff, scratch, index_pool, index_stats, tables, buf,
                                                                 work.local_repair);
            };
            if (teams == 4) run(scan_guess_kernel<4>); else run(scan_guess_kernel<1>);
            int group = 1;
            while (work.alike && group < kRepairWarps && work.n_parts >= 256 * group) group *= 2;
            // (a subsequence may begin behind its first vector's start, and 64 bytes beyond)
            const int vectors = (int)(work.max_subseq_bits / 128 + 5);
            const int at_once = (int)std::min<size_t>(kRepairThreads, kRepairStreams / (16 * vectors));
            const size_t repair = tables_bytes(tables) + (size_t)at_once * vectors * 16;
            allow(scan_repair_kernel, repair);
            launch(early, (work.n_parts + group - 1) / group, kRepairThreads, repair, stream, scan_repair_kernel, descs, work.parts, work.n_parts, group, huff,
                   scratch, tables, vectors, at_once);
            if (work.n_whole > 0)
                launch(early, work.n_whole, kRepairThreads, repair, stream, scan_repair_kernel, descs, work.parts + work.n_parts, work.n_whole, 1, huff, scratch,
                       tables, vectors, at_once);
        }
        if (work.n_slots > 0) {
            const size_t one = tables_bytes(tables) + buf;
            allow(scan_slots_kernel, one);
            launch(early && work.n_guess > 0, work.n_slots, kSlotThreads, one, stream, scan_slots_kernel, descs, work.segs + work.n_guess, blob, huff, scratch, tables);
            // As many runs as segments in each: both are followed one after the other.  The maps fit
            // shared memory up to 1500 segments (6 MB of scan).
            int warps = 1;
            if (work.max_slot_segs > 12)
                while (warps * warps < work.max_slot_segs && warps < kChainThreads / 32) warps++;
            const int slots = work.max_slot_segs < 1500 ? work.max_slot_segs : 1500;
            const size_t maps = (size_t)slots * kSlotStates * sizeof(SlotMap);
            allow(scan_chain_kernel, maps);
            launch(early, work.n_slot_images, warps * 32, maps, stream, scan_chain_kernel, descs, work.slot_images, huff, scratch, slots);
        }
        auto index = [&](auto kernel, const uint2 *segs, int n, int of, int team, size_t bytes) {
            allow(kernel, bytes);
            launch(early, (n + of - 1) / of, team * of, bytes, stream, kernel, descs, segs, n, huff, scratch, status, index_pool, index_stats, tables,
                   buf);
        };
        if (work.n_guess > 0)
            index(teams == 4 ? scan_index_kernel<4, false> : scan_index_kernel<1, false>, work.segs, work.n_guess, teams, kIndexTeam<false>, tables_bytes(tables));
        if (work.n_slots > 0)
            index(slot_teams == 4 ? scan_index_kernel<4, true> : scan_index_kernel<1, true>, work.segs + work.n_guess, work.n_slots, slot_teams, kIndexTeam<true>,
                  tables_bytes(tables) + (size_t)slot_teams * buf);
    }
    if (work.n_restart > 0)
        scan_restart_kernel<<<work.n_restart, kRestartThreads, 0, stream>>>(descs, work.restart, blob, huff, scratch, status);
}

} // namespace ffcvb
