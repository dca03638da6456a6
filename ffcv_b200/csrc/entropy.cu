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
//   scan_sync_kernel    one CTA per segment of a scan (about 128 subsequences): removes the byte
//                       stuffing, decodes every subsequence from a guessed state and repairs the
//                       guesses by re-decoding from the left neighbour's exit state until nothing
//                       changes.  A decoder that starts mid-stream falls in step after 0.9 kbit on
//                       average (4:2:0, quality 90; 99 % within 4 kbit), dominated by the block's
//                       slot inside the MCU, so two passes and a few stragglers settle a segment.
//                       Segments behind the first decode the last 8 kbit before them as a run-up.
//   scan_stitch_kernel  scans of several segments: where a run-up was too short, walks
//                       on from the exact state until it meets the recorded one.
//   scan_slots_kernel, scan_chain_kernel   instead of the two above while a batch's scans leave most of the
//                       GPU idle: every subsequence from all block slots at once, see there.
//   scan_index_kernel   every subsequence once more from its exact state: records the blocks; the
//                       last CTA of an image integrates the DC differences.
//
// Integer work bound by instruction issue at large batches and by the chain look-up -> shift ->
// look-up at small ones: about 25 instructions per symbol and lane, tables and stream in shared memory.
#include "huffman.h"
#include "kernels.h"

namespace ffcvb {

namespace {

constexpr int kThreads = kSegSubs;          // one thread per subsequence: a team of four warps per segment
constexpr int kFastBytes = 2 * kHuffFast;   // a Huffman table in shared memory

// The threads that work on one segment.  A CTA holds one team, or several that share the Huffman
// tables in shared memory and meet at barriers of their own.
template <int TEAMS, int SIZE = kThreads>
struct Team {
    static constexpr int size = SIZE;
    int index, tid;
    __device__ __forceinline__ Team() : index(TEAMS == 1 ? 0 : threadIdx.x / SIZE), tid(TEAMS == 1 ? threadIdx.x : threadIdx.x % SIZE) {}
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

// The walk below in plain code: for tables that are not fast_ok, and for the few walks on a stream in
// global memory.  One symbol at a time, tables where they are.
template <bool RECORD>
__device__ __noinline__ uint32_t walk_plain(const uint32_t *words, Cursor &cur, uint32_t end, const ImageDesc &d,
                                            const HuffTable *__restrict__ huff, uint32_t *pos, uint32_t blk, uint32_t limit) {
    const int luma = d.ncomp == 1 ? 1 : d.hs * d.vs;
    uint32_t done = 0;
    while (cur.p < end) {
        if (RECORD && cur.z == 0) {
            if (blk < limit) pos[blk] = cur.p;
            blk++;
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
// completed.  `buf`: the segment's stream in shared memory (words most significant bit first).  With
// RECORD every block that begins before `end` gets its position written to pos[blk], pos[blk + 1],
// ... below pos[limit]; `blk` is the first of them.
//
// The 32 lanes of a warp walk unrelated places, so nothing in the loops branches: position (bits 0-17)
// and zig-zag index (bits 24-30) share one word that an entry is simply added to; a 96-bit window over
// the stream stays in registers (hi holds the word the position lies in, lo and nx the two behind it)
// and is moved on by predicated instructions; so are the table switches and the slot at the end of a
// block; codes too long for the first level are reached by the index's maximum.  As long as `end` is
// more than kHuffBits away an entry may stand for two symbols (1.46 on average), so that the walk's
// last position is the same whatever state it came from.
constexpr uint32_t kPosMask = 0x3ffff;
template <bool RECORD>
__device__ __forceinline__ uint32_t walk(const unsigned char *buf, Cursor &cur, uint32_t end, const Tables *s, const ImageDesc &d,
                                         const HuffTable *__restrict__ huff, uint32_t *pos = nullptr, uint32_t blk = 0, uint32_t limit = 0) {
    if (cur.p >= end) return 0;
    if (!d.fast_tables) return walk_plain<RECORD>(reinterpret_cast<const uint32_t *>(buf), cur, end, d, huff, pos, blk, limit);
    const uint32_t pairs = s->pairs;
    uint32_t st = cur.p | (uint32_t)cur.z << 24, done = 0;
    const Slot here = s->slot[cur.c];
    uint32_t ac = here.tables >> 16, tab = cur.z ? ac : here.tables & 0xffff;
    uint32_t ahead = load_shared(here.next), after = load_shared(here.next + 4); // the slot that follows
    uint32_t wa = shared_address(buf) + (cur.p >> 5) * 4;
    uint32_t hi = load_shared(wa), lo = load_shared(wa + 4), nx = load_shared(wa + 8);
    wa += 12;
    if (RECORD && cur.z == 0) {
        if (blk < limit) pos[blk] = cur.p;
        blk++;
    }
    uint32_t p = cur.p;
    auto symbol = [&](bool live, bool paired) { // (not live: nothing moves)
        const uint32_t w = __funnelshift_l(lo, hi, st);
        const uint32_t index = (uint32_t)__viaddmax_s32((int)(w >> 16), kHuffFast - 65536, (int)(w >> 22));
        uint32_t e = 0;
        asm volatile("{\n\t"
                     ".reg .pred q;\n\t"
                     "setp.ne.u32 q, %2, 0;\n\t"
                     "@q ld.shared.u16 %0, [%1];\n\t"
                     "}"
                     : "+r"(e)
                     : "r"(tab + index * 2), "r"((uint32_t)live));
        e = __byte_perm(e, 0, 0x1440); // bits consumed to bits 0-7, positions advanced to bits 24-31
        const uint32_t before = st;
        st += e;
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
        const uint32_t to = ac + (paired && st < (uint32_t)(64 - kPairAdvance) << 24 ? pairs : 0);
        tab = live ? to : tab;
        const bool eob = st >= 0x40000000u;
        asm volatile("{\n\t"
                     ".reg .pred q;\n\t"
                     "setp.ge.u32 q, %0, 0x40000000;\n\t"
                     "@q and.b32 %0, %0, 0x3ffff;\n\t"
                     "@q add.u32 %1, %1, 1;\n\t"
                     "@q and.b32 %2, %4, 0xffff;\n\t"
                     "@q shr.u32 %3, %4, 16;\n\t"
                     "@q ld.shared.v2.u32 {%4, %5}, [%5];\n\t"
                     "}"
                     : "+r"(st), "+r"(done), "+r"(tab), "+r"(ac), "+r"(ahead), "+r"(after));
        p = st & kPosMask;
        if (RECORD) {
            if (eob && p < end && blk < limit) pos[blk] = p;
            blk += eob ? 1 : 0;
        }
    };
    const int pairs_end = (int)end - kHuffBits; // the first symbol of a pair that begins up to here ends before `end`
    if ((int)p <= pairs_end) {
        do {
            symbol(true, true);
            symbol((int)p <= pairs_end, true);
        } while ((int)p <= pairs_end);
        if (st >> 24) tab = ac; // (at 0 it is the DC table)
    }
    while (p < end) symbol(true, false);
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

struct SyncShared {
    uint16_t entry[kThreads + 2]; // state at the start of every subsequence, relative to it
    uint16_t blocks[kThreads];    // blocks completed inside it
    uint8_t list[2][kThreads];    // subsequences to decode (again)
    int count[2];
    int warp[kThreads / 32];
    uint32_t mark[2];
};
// Shared memory of a team's stream: the aligned vectors that hold max_raw bytes, and the zero bytes behind.
__host__ __device__ constexpr size_t stream_bytes(uint32_t max_raw) { return ((size_t)max_raw + 16 + 64 + 31) / 16 * 16; }

__device__ __forceinline__ bool index_entry_valid(const DecodeIndexHeader *entry, const ImageDesc &d) {
    const volatile DecodeIndexHeader *h = entry; // written by an earlier launch
    return h->magic == kDecodeIndexMagic && h->scan_len == d.scan_len && h->subseq_bits == d.subseq_bits && h->segments == d.seg_count;
}

template <int TEAMS>
__global__ void __launch_bounds__(kThreads * TEAMS)
scan_sync_kernel(const ImageDesc *__restrict__ descs, const uint2 *__restrict__ segs, int n_segs, const uint8_t *__restrict__ blob,
                 const HuffTable *__restrict__ huff, EntropyScratch scratch, const uint8_t *__restrict__ index_pool,
                 unsigned long long *__restrict__ index_stats, int table_slots, uint32_t buf_bytes) {
    extern __shared__ __align__(16) unsigned char s_dyn[];
    __shared__ SyncShared s_teams[TEAMS];
    next_may_begin();
    const Team<TEAMS> team;
    const int tid = team.tid;
    SyncShared &sh = s_teams[team.index];
    Tables *tables = reinterpret_cast<Tables *>(s_dyn);
    unsigned char *buf = s_dyn + tables_bytes(table_slots) + team.index * buf_bytes;
    const int mine = blockIdx.x * TEAMS + team.index;
    const uint2 which = segs[min(mine, n_segs - 1)];
    const uint32_t j = which.y;
    const ImageDesc &d = descs[which.x];
    const uint32_t S = d.subseq_bits, R = d.seg_raw, warm = j == 0 ? 0 : d.seg_warm;
    load_tables(tables, d, huff); // (the same whichever team's sample they are taken from)
    if (TEAMS > 1) {
        copies_wait();
        __syncthreads();
        if (mine >= n_segs) return;
    }

    // ---- the segment's raw bytes: run-up, own part, and what follows it to the end of a block
    const uint32_t scan_len = d.scan_len, own0 = j * R, own1 = min(own0 + R, scan_len);
    const uint32_t raw0 = own0 - min(own0, warm * (S >> 3)), raw1 = min(own1 + kSegOverlap, scan_len);
    const uint32_t at[2] = {own0 - raw0, own1 - raw0};
    const uint32_t kept = unstuff(team, buf, blob + d.payload_off + d.scan_off + raw0, raw1 - raw0, raw0 == 0, at, sh.warp, sh.mark);
    const uint32_t own_bit = at[0] == 0 ? 0 : sh.mark[0] * 8, own_end = own1 == raw1 ? kept * 8 : sh.mark[1] * 8;
    {
        uint4 *dst = reinterpret_cast<uint4 *>(scratch.clean + d.clean_off + (size_t)j * d.seg_stride);
        const uint4 *src = reinterpret_cast<const uint4 *>(buf);
        for (uint32_t k = tid; k < (kept + 64 + 15) / 16; k += kThreads) dst[k] = src[k];
    }
    const size_t seg = (size_t)d.seg_first + j;
    const int n_own = (int)((own_end - own_bit + S - 1) / S), n_subs = (int)warm + n_own;

    if (TEAMS == 1) copies_wait();

    // ---- decode index: the states an earlier decode of this very stream left behind (the answer is uniform: a
    // batch is only given an entry that no launch beside it writes)
    if (index_pool != nullptr && d.index_use != 0) {
        const DecodeIndexHeader *h = reinterpret_cast<const DecodeIndexHeader *>(index_pool + d.index_off);
        if (index_entry_valid(h, d)) {
            const uint32_t *src = reinterpret_cast<const uint32_t *>(h + 1) + (size_t)j * (kSegSubs + 2);
            scratch.sub_info[seg * kSegSubs + tid] = __ldcg(src + tid);
            if (tid == 0) {
                scratch.meta[seg] = SegMeta{own_bit, own_end, kept, __ldcg(src + kSegSubs), __ldcg(src + kSegSubs + 1), 0};
                if (j == 0 && index_stats) atomicAdd(index_stats, 1ull);
            }
            return;
        }
    }

    // ---- guess and repair.  Subsequences t < warm lie in the run-up.
    auto start_of = [&](int t) -> int { return (int)own_bit + (t - (int)warm) * (int)S; };
    sh.entry[tid] = 0; // guess: a block, slot 0, begins here (exact for the scan's first subsequence)
    sh.blocks[tid] = 0;
    if (tid == 0) {
        sh.entry[kThreads] = 0;
        sh.count[0] = sh.count[1] = 0;
    }
    team.sync();
    int n_list = n_subs;
    for (int round = 0; round <= n_subs && n_list > 0; round++) {
        int t = -1;
        uint32_t in = 0;
        if (tid < n_list) {
            t = round == 0 ? (start_of(tid) >= 0 ? tid : -1) : sh.list[round & 1][tid];
            if (t >= 0) in = sh.entry[t];
        }
        team.sync(); // every entry state is read before any exit state is written
        if (tid == 0) sh.count[round & 1] = 0; // filled again from the next round's second half on
        bool changed = false;
        if (t >= 0) {
            const uint32_t start = (uint32_t)start_of(t), end = min(start + S, own_end);
            Cursor cur = unpack(in, start);
            sh.blocks[t] = (uint16_t)walk<false>(buf, cur, end, tables, d, huff);
            const uint32_t out = pack(cur, end);
            changed = sh.entry[t + 1] != out;
            if (changed) sh.entry[t + 1] = (uint16_t)out; // only this thread writes entry t + 1 in this round
            changed = changed && t + 1 < n_subs;
        }
        __syncwarp();
        const uint32_t who = __ballot_sync(0xffffffffu, changed);
        if (who != 0) { // one place in the next list per warp, then per lane
            int base = 0;
            if ((tid & 31) == 0) base = atomicAdd(&sh.count[(round + 1) & 1], __popc(who));
            base = __shfl_sync(0xffffffffu, base, 0);
            if (changed) sh.list[(round + 1) & 1][base + __popc(who & ((1u << (tid & 31)) - 1))] = (uint8_t)(t + 1);
        }
        team.sync();
        n_list = sh.count[(round + 1) & 1];
    }

    // ---- own subsequences: entry state and completed blocks
    const uint32_t done = tid < n_own ? sh.blocks[tid + warm] : 0;
    if (tid < n_own) scratch.sub_info[seg * kSegSubs + tid] = sh.entry[tid + warm] | done << 16;
    int total;
    team_scan(team, (int)done, sh.warp, total);
    if (tid == 0) scratch.meta[seg] = SegMeta{own_bit, own_end, kept, sh.entry[n_subs], (uint32_t)total, 0};
}

// Scans of several segments, one CTA each: the exit state of every segment has to be the entry state
// the next one worked out from its run-up.  Where it is not, one thread walks on from the exact
// state, subsequence by subsequence, until it meets the recorded ones; a walk that crosses a whole
// segment makes the boundary behind it the next round's.
__global__ void __launch_bounds__(kThreads)
scan_stitch_kernel(const ImageDesc *__restrict__ descs, const int32_t *__restrict__ list, const HuffTable *__restrict__ huff,
                   EntropyScratch scratch) {
    next_may_begin();
    await_previous();
    const ImageDesc &d = descs[list[blockIdx.x]];
    const int tid = threadIdx.x, n_seg = (int)d.seg_count;
    const uint32_t S = d.subseq_bits;
    SegMeta *meta = scratch.meta + d.seg_first;
    uint32_t *info = scratch.sub_info + (size_t)d.seg_first * kSegSubs;
    for (int round = 0; round < n_seg; round++) {
        bool any = false;
        for (int k0 = 1; k0 < n_seg; k0 += kThreads) { // (a round looks at all boundaries, kThreads at a time)
            const int k = k0 + tid;
            uint32_t exact = 0;
            bool differs = false;
            if (k < n_seg) {
                exact = meta[k - 1].exit;
                // an empty segment (its scan ended in stuffing) hands the state on
                differs = meta[k].own_bit < meta[k].own_end ? exact != (info[(size_t)k * kSegSubs] & 0xffff) : exact != meta[k].exit;
            }
            if (!__syncthreads_or(differs)) continue;
            any = true;
            if (differs) {
                const SegMeta m = meta[k];
                const uint32_t *words = reinterpret_cast<const uint32_t *>(scratch.clean + d.clean_off + (size_t)k * d.seg_stride);
                uint32_t *mine = info + (size_t)k * kSegSubs;
                const int n_own = (int)((m.own_end - m.own_bit + S - 1) / S);
                uint32_t state = exact, blocks = m.blocks;
                int t = 0;
                for (; t < n_own && (mine[t] & 0xffff) != state; t++) {
                    const uint32_t start = m.own_bit + (uint32_t)t * S, end = min(start + S, m.own_end);
                    Cursor cur = unpack(state, start);
                    const uint32_t done = walk_plain<false>(words, cur, end, d, huff, nullptr, 0, 0);
                    blocks += done - (mine[t] >> 16);
                    mine[t] = state | done << 16;
                    state = pack(cur, end);
                }
                meta[k].blocks = blocks;
                if (t == n_own) meta[k].exit = state;
            }
            __syncthreads();
        }
        if (!any) break;
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
        sh.blocks[t][i] = (uint16_t)walk<false>(buf, cur, end, tables, d, huff);
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
    if (tid == 0) scratch.meta[seg] = SegMeta{own_bit, own_end, kept, 0, 0, 0};
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
                meta[k].exit = behind & 0xffff;
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
                        const uint32_t done = walk_plain<false>(words, cur, end, d, huff, nullptr, 0, 0);
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
                meta[k].exit = at;
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

template <int TEAMS>
__global__ void __launch_bounds__(kThreads * TEAMS)
scan_index_kernel(const ImageDesc *__restrict__ descs, const uint2 *__restrict__ segs, int n_segs, const HuffTable *__restrict__ huff,
                  EntropyScratch scratch, int32_t *__restrict__ status, uint8_t *__restrict__ index_pool,
                  unsigned long long *__restrict__ index_stats, int table_slots, uint32_t buf_bytes) {
    extern __shared__ __align__(16) unsigned char s_dyn[];
    __shared__ int s_warps[TEAMS][kThreads / 32];
    __shared__ uint32_t s_lasts[TEAMS];
    next_may_begin();
    const Team<TEAMS> team;
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
    load_tables(tables, d, huff);
    await_previous();
    if (TEAMS > 1) {
        copies_wait();
        __syncthreads();
        if (mine >= n_segs) return;
    }
    const size_t seg = (size_t)d.seg_first + j;
    const SegMeta m = scratch.meta[seg];
    const uint32_t S = d.subseq_bits, nblocks = d.nblocks;
    uint32_t *pos = scratch.pos + d.block_base;
    int16_t *dc = scratch.dc + d.block_base;

    uint32_t base = 0; // blocks before this segment
    if (j > 0) {
        int before = 0, all;
        for (uint32_t k = tid; k < j; k += kThreads) before += (int)scratch.meta[d.seg_first + k].blocks;
        team_scan(team, before, s_warp, all);
        base = (uint32_t)all;
    }
    const int n_own = (int)((m.own_end - m.own_bit + S - 1) / S);
    uint32_t info = 0;
    if (d.slots == 0) {
        if (tid < n_own) info = scratch.sub_info[seg * kSegSubs + tid];
    } else { // one thread follows the real state from subsequence to subsequence
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
        const uint32_t skip = m.own_bit >> 7; // vectors of the run-up
        const uint4 *src = reinterpret_cast<const uint4 *>(scratch.clean + d.clean_off + (size_t)j * d.seg_stride);
        for (uint32_t k = skip + tid; k < (m.bytes + 64 + 15) / 16; k += kThreads) copy16_async(buf + (size_t)(k - skip) * 16, src + k);
        copies_wait();
        int in_segment;
        const uint32_t first = base + (uint32_t)team_scan(team, (int)(info >> 16), s_warp, in_segment); // (and a barrier for the copies)
        const uint32_t bias = j * d.seg_stride * 8 + skip * 128; // stream position of the buffer's bit 0
        const uint32_t start = m.own_bit - skip * 128 + (uint32_t)tid * S;
        const uint32_t end = min(start + S, m.own_end - skip * 128);
        Cursor cur = unpack(info & 0xffff, start);
        const uint32_t b0 = first + (cur.z != 0 ? 1 : 0); // the block in progress belongs to the subsequence it began in
        uint32_t b1 = b0;
        int sum[3] = {0, 0, 0};
        if (tid < n_own && first < nblocks && cur.p < end) {
            const uint32_t stream = shared_address(buf), luma = tables->luma, bpm = tables->bpm;
            const uint32_t done = walk<true>(buf, cur, end, tables, d, huff, pos, b0, nblocks);
            b1 = min(first + done + (cur.z != 0 ? 1 : 0), nblocks);
            // the DC symbols of the blocks found: positions move on to the first AC symbol, values count
            // from the thread's first block
            uint32_t slot = b0 % bpm, next_pos = b0 < b1 ? pos[b0] : 0;
            for (uint32_t b = b0; b < b1; b++) {
                const uint32_t p = next_pos, wa = stream + (p >> 5) * 4;
                if (b + 1 < b1) next_pos = pos[b + 1];
                const uint32_t w = __funnelshift_l(load_shared(wa + 4), load_shared(wa), p);
                const int comp = slot < luma ? 0 : (int)(slot - luma) + 1;
                const HuffTable *table = huff + d.tab_id[d.dc_tab[comp]];
                uint32_t e = table->look[w >> (32 - kHuffBits)];
                if (e & kHuffLong) e = huff_long(table, e, w);
                const uint32_t n = e & 31, size = (e >> 5) & 15;
                const int v = size ? huff_value(w, n, size) : 0;
                sum[0] += comp == 0 ? v : 0;
                sum[1] += comp == 1 ? v : 0;
                sum[2] += comp == 2 ? v : 0;
                pos[b] = bias + p + n;
                dc[b] = (int16_t)(comp == 0 ? sum[0] : (comp == 1 ? sum[1] : sum[2]));
                slot = slot + 1 == bpm ? 0 : slot + 1;
            }
        }
        // what the segment holds before the thread's first block
        int before[3];
#pragma unroll
        for (int c = 0; c < 3; c++) before[c] = c < d.ncomp ? team_scan(team, sum[c], s_warp, sums[c]) : 0;
        uint32_t slot = b0 % tables->bpm;
        for (uint32_t b = b0; b < b1; b++) {
            dc[b] = (int16_t)(dc[b] + (slot < tables->luma ? before[0] : (slot == tables->luma ? before[1] : before[2])));
            slot = slot + 1 == tables->bpm ? 0 : slot + 1;
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
        uint32_t *dst = reinterpret_cast<uint32_t *>(index_pool + d.index_off + sizeof(DecodeIndexHeader)) + (size_t)j * (kSegSubs + 2);
        dst[tid] = info;
        if (tid == 0) {
            dst[kSegSubs] = m.exit;
            dst[kSegSubs + 1] = m.blocks;
        }
    }
    // ---- the CTA that finishes an image last turns the segments' DC sums into sums before them
    if (TEAMS == 1) copies_wait(); // (nothing may be under way when the CTA ends)
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

uint32_t subseq_target(uint64_t total_bits) {
    // A subsequence costs a re-synchronisation (0.9 kbit, 0.35 without subsampling) on top of its own length, so
    // long ones are less work; short ones are a shorter chain, which decides while few bits leave the GPU
    // mostly idle.  256 subsequences per SM are enough of them: batches of 80 Mbit, alone / four in flight, take
    // 473 / 335 us at 512 bits, 424 / 274 at 1024, 388 / 255 at 1280; a 4:4:4 scan of 24 Mbit 554 us at 256 bits,
    // 505 at 512, 499 at 768, 509 at 1024.
    const uint64_t t = total_bits / (148 * 256);
    return (uint32_t)(t < 256 ? 256 : (t > kMaxSubseqBits ? kMaxSubseqBits : (t + 31) / 32 * 32));
}

ScanLayout layout_scan(uint32_t scan_len, uint32_t target_bits) {
    ScanLayout l{};
    const uint64_t bits = (uint64_t)scan_len * 8;
    const uint32_t warm = (8192 + target_bits - 1) / target_bits; // all but one in 10^4 run-ups are long enough
    if (bits <= (uint64_t)kSegSubs * target_bits || (target_bits > 512 && bits <= (uint64_t)kSegSubs * kMaxSubseqBits)) {
        l.seg_count = 1;
        l.subseq_bits = (uint32_t)((bits + kSegSubs - 1) / kSegSubs + 31) / 32 * 32;
        if (l.subseq_bits < 128) l.subseq_bits = 128;
        l.seg_raw = kSegSubs * l.subseq_bits / 8;
    } else {
        const uint64_t own = kSegSubs - warm;
        l.seg_count = (uint32_t)((bits + own * target_bits - 1) / (own * target_bits));
        l.subseq_bits = (uint32_t)((bits + own * l.seg_count - 1) / (own * l.seg_count) + 31) / 32 * 32;
        l.seg_warm = warm;
        l.seg_raw = (uint32_t)own * l.subseq_bits / 8;
        l.seg_count = (scan_len + l.seg_raw - 1) / l.seg_raw;
    }
    l.seg_stride = (kSegSubs * l.subseq_bits / 8 + kSegOverlap + 64 + 31) / 16 * 16;
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
        // 22 KB fit an SM then, instead of five.
        const int teams = work.alike && n_segs >= 148 * 5 ? 4 : 1;
        const size_t smem = tables_bytes(tables) + (size_t)teams * buf;
        if (work.n_guess > 0) {
            const int grid = (work.n_guess + teams - 1) / teams;
            auto run = [&](auto kernel) {
                allow(kernel, smem);
                kernel<<<grid, kThreads * teams, smem, stream>>>(descs, work.segs, work.n_guess, blob, huff, scratch, index_pool, index_stats, tables, buf);
            };
            if (teams == 4) run(scan_sync_kernel<4>); else run(scan_sync_kernel<1>);
            if (work.n_multi > 0) launch(early, work.n_multi, kThreads, 0, stream, scan_stitch_kernel, descs, work.multi, huff, scratch);
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
        auto run = [&](auto kernel) {
            allow(kernel, smem);
            launch(early, (n_segs + teams - 1) / teams, kThreads * teams, smem, stream, kernel, descs, work.segs, n_segs, huff, scratch, status, index_pool,
                   index_stats, tables, buf);
        };
        if (teams == 4) run(scan_index_kernel<4>); else run(scan_index_kernel<1>);
    }
    if (work.n_restart > 0)
        scan_restart_kernel<<<work.n_restart, kRestartThreads, 0, stream>>>(descs, work.restart, blob, huff, scratch, status);
}

} // namespace ffcvb
