// Host side of libffcv_b200.so: contexts, batch slots, the staging thread pool and the C ABI
// declared in include/ffcv_b200.h.
#include <cuda_runtime.h>
#include <emmintrin.h>
#include <errno.h>
#include <fcntl.h>
#include <stdarg.h>
#include <stddef.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>
#include <sys/vfs.h>
#include <unistd.h>

#include <array>
#include <atomic>
#include <condition_variable>
#include <functional>
#include <mutex>
#include <string>
#include <memory>
#include <thread>
#include <unordered_map>
#include <chrono>
#include <vector>

#include "../../include/ffcv_b200.h"
#include "decode_index.h"
#include "jpeg_header.h"
#include "kernels.h"
#include "table_store.h"
#include "types.h"

using namespace ffcvb;

namespace {

// ------------------------------------------------------------------ staging thread pool
// Worker threads with two job lanes.  The synchronous lane (parallel_for) serves the header
// parse of the batch being staged; the asynchronous lane carries the payload copy of the batch
// staged before it, which keeps running while the caller goes on.  Workers drain the synchronous
// lane first, so a parse never queues behind a copy.  Items are handed out under the mutex,
// `grain` at a time.
class Pool {
  public:
    enum Lane { kSync = 0, kAsync = 1 };
    explicit Pool(int n) {
        for (int i = 0; i < n; i++) workers_.emplace_back([this] { loop(); });
    }
    ~Pool() {
        {
            std::lock_guard<std::mutex> g(m_);
            stop_ = true;
        }
        cv_.notify_all();
        for (auto &t : workers_) t.join();
    }
    // Runs fn(i) for i in [0, n) on the pool and the calling thread; returns when all are done.
    void parallel_for(int n, int grain, std::function<void(int)> fn) {
        post(kSync, n, grain, std::move(fn), nullptr);
        wait(kSync);
    }
    // Hands fn(i), i in [0, n), to the workers and returns.  `done` runs once after the last item
    // (under the pool's mutex: it must be short and must not call the pool).  The lane must be idle.
    // At most `max_threads` threads work on the job at a time (0 = no limit).
    void post(Lane lane, int n, int grain, std::function<void(int)> fn, std::function<void()> done,
              int max_threads = 0) {
        wait(lane);
        if (n <= 0) {
            if (done) done();
            return;
        }
        {
            std::lock_guard<std::mutex> g(m_);
            Job &j = jobs_[lane];
            j.fn = std::move(fn);
            j.done = std::move(done);
            j.n = n;
            j.next = 0;
            j.grain = grain < 1 ? 1 : grain;
            j.inflight = 0;
            j.limit = max_threads > 0 ? max_threads : 1 << 30;
            j.active = true;
        }
        const int chunks = (n + (grain < 1 ? 1 : grain) - 1) / (grain < 1 ? 1 : grain);
        if (workers_.empty())
            wait(lane); // nobody else would run it
        else if (chunks >= (int)workers_.size())
            cv_.notify_all();
        else
            for (int k = 0; k < chunks; k++) cv_.notify_one();
    }
    // Lends the calling thread to the lane's job, then waits until the job is complete.
    void wait(Lane lane) {
        std::unique_lock<std::mutex> g(m_);
        Job &j = jobs_[lane];
        while (j.active) {
            if (j.next < j.n)
                run_some(j, g);
            else
                done_cv_.wait(g, [&] { return !j.active; });
        }
    }
    void wait_all() {
        wait(kSync);
        wait(kAsync);
    }
    int size() const { return (int)workers_.size() + 1; }

  private:
    struct Job {
        std::function<void(int)> fn;
        std::function<void()> done;
        int n = 0, next = 0, grain = 1, inflight = 0, limit = 1 << 30;
        bool active = false;
    };
    // Called with the mutex held and items left; returns with it held.
    void run_some(Job &j, std::unique_lock<std::mutex> &g) {
        const int lo = j.next;
        const int hi = lo + j.grain < j.n ? lo + j.grain : j.n;
        j.next = hi;
        j.inflight++;
        g.unlock();
        for (int i = lo; i < hi; i++) j.fn(i);
        g.lock();
        j.inflight--;
        if (j.next >= j.n && j.inflight == 0) {
            if (j.done) j.done();
            j.done = nullptr;
            j.active = false;
            done_cv_.notify_all();
        }
    }
    Job *pending() {
        for (Job &j : jobs_)
            if (j.active && j.next < j.n && j.inflight < j.limit) return &j;
        return nullptr;
    }
    void loop() {
        std::unique_lock<std::mutex> g(m_);
        for (;;) {
            cv_.wait(g, [&] { return stop_ || pending() != nullptr; });
            if (stop_) return;
            while (Job *j = pending()) run_some(*j, g);
        }
    }
    std::vector<std::thread> workers_;
    std::mutex m_;
    std::condition_variable cv_, done_cv_;
    bool stop_ = false;
    Job jobs_[2];
};

size_t align_up(size_t v, size_t a) { return (v + a - 1) / a * a; }

// Multiplicative hash over a table's bytes, eight at a time: lets the (serial) table
// deduplication of a batch compare 8 bytes per table instead of the tables themselves; the hashes
// are computed by the parallel header parse.
uint64_t hash_bytes(const void *p, size_t n) {
    const uint8_t *b = static_cast<const uint8_t *>(p);
    uint64_t h = 0x9E3779B97F4A7C15ull ^ n;
    size_t i = 0;
    for (; i + 8 <= n; i += 8) {
        uint64_t w;
        memcpy(&w, b + i, 8);
        h = (h ^ w) * 0xFF51AFD7ED558CCDull;
        h ^= h >> 29;
    }
    uint64_t w = 0;
    if (i < n) memcpy(&w, b + i, n - i);
    h = (h ^ w) * 0xC4CEB9FE1A85EC53ull;
    return h ^ (h >> 32);
}

// Copy into the pinned staging buffer with non-temporal stores: the destination is read next by
// the DMA engine, not by the CPU, so it should not displace the cache or cost a read-for-ownership.
// dst is 16-byte aligned (payload offsets are).
void stream_copy(uint8_t *dst, const uint8_t *src, size_t n) {
    if ((reinterpret_cast<uintptr_t>(dst) & 15) != 0 || n < 4096) {
        memcpy(dst, src, n);
        return;
    }
    size_t k = 0;
    for (; k + 64 <= n; k += 64) {
        __m128i a = _mm_loadu_si128(reinterpret_cast<const __m128i *>(src + k));
        __m128i b = _mm_loadu_si128(reinterpret_cast<const __m128i *>(src + k + 16));
        __m128i c = _mm_loadu_si128(reinterpret_cast<const __m128i *>(src + k + 32));
        __m128i d = _mm_loadu_si128(reinterpret_cast<const __m128i *>(src + k + 48));
        _mm_stream_si128(reinterpret_cast<__m128i *>(dst + k), a);
        _mm_stream_si128(reinterpret_cast<__m128i *>(dst + k + 16), b);
        _mm_stream_si128(reinterpret_cast<__m128i *>(dst + k + 32), c);
        _mm_stream_si128(reinterpret_cast<__m128i *>(dst + k + 48), d);
    }
    if (k < n) memcpy(dst + k, src + k, n - k);
}

// The same to any address, in whole cache lines but for the ends.  What several threads write for one transfer has
// to leave their caches this way: the transfer otherwise waits for lines that lie dirty in cores which
// have gone to sleep meanwhile (4.3 MB: 650-900 us instead of 90).
void stream_copy_lines(uint8_t *dst, const uint8_t *src, size_t n) {
    const size_t head = (size_t)(-reinterpret_cast<uintptr_t>(dst) & 63);
    if (n < head + 64) {
        memcpy(dst, src, n);
        return;
    }
    memcpy(dst, src, head);
    size_t k = head;
    for (; k + 64 <= n; k += 64) {
        __m128i v[4];
        for (int q = 0; q < 4; q++) v[q] = _mm_loadu_si128(reinterpret_cast<const __m128i *>(src + k) + q);
        for (int q = 0; q < 4; q++) _mm_stream_si128(reinterpret_cast<__m128i *>(dst + k) + q, v[q]);
    }
    memcpy(dst + k, src + k, n - k);
}

// What the marker segments of a JPEG stream said, as far as staging needs it.
struct StreamHeader {
    uint64_t size; // of the whole stream
    uint32_t scan_off, scan_len, table_set;
    uint16_t restart_interval, width, height;
    int16_t status; // 0 or why the stream was rejected
    uint8_t ncomp, hs, vs;
};

// StreamHeaders by the stream's offset in its file: open addressing, never shrinks.
class HeaderCache {
  public:
    const StreamHeader *find(uint64_t key) const {
        if (slots_.empty()) return nullptr;
        for (size_t k = place(key);; k = (k + 1) & (slots_.size() - 1)) {
            if (slots_[k].key == key) return &slots_[k].header;
            if (slots_[k].key == kFree) return nullptr;
        }
    }
    void insert(uint64_t key, const StreamHeader &h) {
        if (2 * (count_ + 1) > slots_.size()) {
            std::vector<Entry> old(slots_.empty() ? 1024 : slots_.size() * 2, Entry{kFree, {}});
            old.swap(slots_);
            count_ = 0;
            for (const Entry &e : old)
                if (e.key != kFree) insert(e.key, e.header);
        }
        size_t k = place(key);
        while (slots_[k].key != kFree && slots_[k].key != key) k = (k + 1) & (slots_.size() - 1);
        count_ += slots_[k].key == kFree;
        slots_[k] = Entry{key, h};
    }
    size_t size() const { return count_; }
    void clear() {
        slots_.clear();
        count_ = 0;
    }

  private:
    static constexpr uint64_t kFree = ~0ull;
    struct Entry {
        uint64_t key;
        StreamHeader header;
    };
    size_t place(uint64_t key) const { return (size_t)((key * 0x9E3779B97F4A7C15ull) >> 20) & (slots_.size() - 1); }
    std::vector<Entry> slots_;
    size_t count_ = 0;
};

struct DevBuf {
    void *p = nullptr;
    size_t cap = 0;
};

struct Slot {
    uint8_t *host = nullptr; // pinned
    size_t host_cap = 0;
    DevBuf blob, clean, segs, records, slot_tables, index, planes, rgb; // segs: per-segment scratch; index: per-block positions and DC values
    BatchHeader hdr{};
    ffcvb_plan plan{};
    int n = 0, n_jpeg = 0;
    EntropyWork work{}; // (the lists' addresses are filled in when the batch runs)
    int n_quad = 0, n_444 = 0, n_other = 0, max_w = 0, max_h = 0;
    uint64_t jpeg_list_off = 0, segs_off = 0, parts_off = 0, slot_images_off = 0, restart_off = 0, block_tiles_off = 0, quad_tiles_off = 0;
    uint64_t status_off = 0; // status word and counter of finished segments of every sample
    uint64_t items_off = 0;  // ResizeItem of every sample
    uint64_t gather_off = 0; // gather_ranges, for so many CTAs (0: nothing is gathered)
    int gather_ctas = 0;
    int n_block_tiles = 0, n_quad_tiles = 0, bands = 1;
    bool plain = false; // see ResizeItems
    uint32_t total_blocks = 0;
    bool keep_records = false; // `records` has room for the staged batch
    size_t clean_bytes = 0, plane_bytes = 0, rgb_bytes = 0, scan_bytes = 0, raw_bytes = 0, jpeg_bytes = 0;
    bool staged = false;
    bool packed = false; // single-image calls: the decoded rows are the result, without padding
    bool direct = false; // payloads are gathered by the GPU from pinned host memory
    const uint8_t *range_src = nullptr; // the payloads lie in one piece of pinned memory: copied as such
    size_t range_len = 0;
    size_t staged_end = 0; // blob bytes [0, staged_end) come from the pinned staging buffer
    bool copy_done = true; // the staging threads have finished this slot's payload copy (guarded by ctx->copy_m)
    std::vector<ImageDesc> descs;
    std::vector<uint64_t> src_ptrs;
    // values of the sample's other fields that travel in the head of this batch's blob
    struct Rider {
        std::vector<uint8_t> inline_bytes; // n * item_bytes, or empty when gathered from the file
        std::vector<uint64_t> ptrs;        // file offsets of the n items (gathered riders)
        uint64_t item_bytes = 0;
        void *dst_dev = nullptr;
        uint64_t off = 0, bytes = 0;       // place in the blob (set by ffcvb_stage_batch)
    };
    struct Copy { // a piece of a sample's payload that a staging thread copies
        int sample;
        size_t from, bytes;
    };
    std::vector<Copy> copies;
    std::vector<Rider> pending_riders, riders; // set for the next staging / staged with the current batch
    double stage_ms[4] = {0, 0, 0, 0}; // header parse, layout, payload copy, total
    // working lists of the staging call, kept for their memory
    std::vector<StreamHeader> headers;
    std::vector<int> to_parse;
    std::vector<JpegHeader> parsed;
    std::vector<std::array<uint64_t, 9>> hashes; // of a parsed header's (DC, AC, quantisation) tables x 3 components
    std::vector<ResizeItem> items;
    std::vector<int32_t> jpeg_list, slot_images, restart;
    std::vector<uint4> parts, wholes;
    std::vector<uint2> slot_segs;  // those of slot_images, behind
    std::vector<uint2> seg_list;   // (sample, segment) of the entropy decoder's CTAs
    std::vector<uint2> blk_tiles;  // (sample, k) of the block decoder's CTAs
    std::vector<uint2> quad_tiles; // (sample, tile x | tile y << 16) of the 4:2:0 colour kernel's CTAs
    cudaEvent_t ev[6] = {nullptr, nullptr, nullptr, nullptr, nullptr, nullptr};
    cudaEvent_t ev_begin = nullptr, ev_gather_start = nullptr, ev_gathered = nullptr;
    // recorded behind the copies of the slot's last batch: staging the slot again waits for it, so a
    // caller that forgets to fence the ring gets a stall instead of a batch that is overwritten under
    // its copies (on the device the slot's stream keeps its batches in order)
    cudaEvent_t ev_copied = nullptr;
    bool in_flight = false;
    cudaStream_t last_stream = nullptr; // the stream that batch was queued on
    cudaEvent_t ev_done = nullptr;      // behind all of its work
    bool gather_timed = false; // ev_gather_start .. ev_gathered bracket the last gather of this slot
    bool timed = false; // events of the last run are valid
    uint64_t index_life = 0; // of the decode index that the staged batch has places in
};

constexpr double kMaxAdaptiveShare = 0.5; // of a pinned batch's bytes that the threads may be left to copy

struct AuxBuf {
    DevBuf dev;
    uint8_t *host = nullptr;
    size_t host_cap = 0;
    cudaEvent_t ev = nullptr;
    bool used = false;
};

} // namespace

struct WaitArg {
    ffcvb_ctx *ctx;
    int slot;
};

struct ffcvb_ctx {
    int device = 0;
    std::vector<Slot> slots;
    std::vector<WaitArg> wait_args; // one per slot, for the stream callback that waits for its copy
    std::mutex copy_m;
    std::condition_variable copy_cv;
    std::atomic<bool> copy_timeout{false};
    std::atomic<bool> direct_broken{false}; // an O_DIRECT read was refused: buffered reads from now on
    Pool *pool = nullptr;
    std::string err;
    AuxBuf aux[16];
    int aux_next = 0;
    std::mutex aux_m; // held from stage_aux to the recording of the buffer's event: several threads may share a context
    bool profile = false;
    bool async_staging = false;
    int cpu_share_permille = 0; // pinned source: share of the payload bytes the staging threads copy
    bool adaptive_split = false; // ... adjusted from batch to batch so that both sides take equally long
    double share = 0.0;          // the adjusted share, 0..1
    double batch_interval = 0.0; // ms between two staging calls, smoothed
    std::chrono::steady_clock::time_point last_staged;
    int split_copy_threads = 4; // ... and how many of them copy at a time (more only crowd the gather out)
    // Tuning overrides, read from the environment once when the context is created (0 = none):
    // FFCV_B200_COPY_THREADS, FFCV_B200_SUBSEQ_BITS, FFCV_B200_GATHER_CTAS.
    int tune_copy_threads = 0, tune_subseq_bits = 0, gather_ctas = 0;
    size_t records_limit = SIZE_MAX; // most device memory a slot asks for to write down blocks' places (FFCV_B200_RECORDS_MB)
    // Transfers of a page-locked source run on one stream of their own, in the order of the batches: two
    // batches that share the link would both arrive late, and the first one's kernels would have nothing
    // to overlap with.  High priority, so that a gather's few CTAs are placed ahead of the large grids
    // that are queued.
    cudaStream_t copy_stream = nullptr;
    int32_t *gather_failed = nullptr; // page-locked: set by a gather whose wait for the link ran out
    uint64_t gather_limit_ns = 2000000000ull; // of such a wait (FFCV_B200_GATHER_LIMIT_MS)
    // single-image entry points: their stream, device buffers, pinned result and events of its pieces
    DevBuf one_src, one_dst;
    uint8_t *one_host = nullptr, *one_in = nullptr;
    size_t one_host_cap = 0, one_in_cap = 0;
    cudaStream_t one_stream = nullptr;
    cudaEvent_t one_ev[16] = {};
    // Header cache: what the marker segments of a JPEG sample said, kept per sample (key: its
    // offset in the file) so that from the second epoch on staging a sample is a table look-up
    // instead of a parse; the few distinct tables of a file live in a store of their own.
    bool cache_headers = false; // ffcvb_set_header_cache: sample offsets identify samples (one file per context)
    HeaderCache header_cache;
    TableStore tables;
    // Decode index (ffcvb_set_decode_index): a pool of device memory that keeps, per JPEG stream seen,
    // the decoder states a finished decode left behind; entries are handed out in order and never
    // moved.  Keyed by the sample's offset in the file: the context then serves one file.
    DevBuf index_pool, index_stats;
    DecodeIndex index;
    uint64_t index_life = 0; // counts the calls that set the index up: places of an earlier one mean nothing
};

namespace {

int fail(ffcvb_ctx *c, int code, const char *fmt, ...) {
    char buf[512];
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(buf, sizeof(buf), fmt, ap);
    va_end(ap);
    if (c) c->err = buf;
    return code;
}

#define CU(call)                                                                                   \
    do {                                                                                           \
        cudaError_t e_ = (call);                                                                   \
        if (e_ != cudaSuccess)                                                                     \
            return fail(ctx, e_ == cudaErrorMemoryAllocation ? FFCVB_E_NOMEM : FFCVB_E_CUDA,       \
                        "%s: %s", #call, cudaGetErrorString(e_));                                  \
    } while (0)

int grow_dev(ffcvb_ctx *ctx, DevBuf &b, size_t need) {
    if (need <= b.cap) return 0;
    size_t cap = align_up(need + need / 4, 1 << 20);
    if (b.p) {
        CU(cudaDeviceSynchronize());
        CU(cudaFree(b.p));
        b.p = nullptr;
        b.cap = 0;
    }
    CU(cudaMalloc(&b.p, cap));
    b.cap = cap;
    return 0;
}

// A buffer that a batch cannot do without.  What was written down of blocks' places it can: where memory runs out
// that goes, of all slots.
int grow_needed(ffcvb_ctx *ctx, DevBuf &b, size_t need) {
    const std::string err = ctx->err;
    int rc = grow_dev(ctx, b, need);
    if (rc != FFCVB_E_NOMEM) return rc;
    cudaGetLastError();
    bool freed = false;
    for (auto &s : ctx->slots) {
        if (!s.records.p) continue;
        if (!freed) CU(cudaDeviceSynchronize());
        CU(cudaFree(s.records.p));
        s.records = DevBuf{};
        freed = true;
    }
    if (!freed) return rc;
    ctx->records_limit = 0;
    if ((rc = grow_dev(ctx, b, need)) == FFCVB_OK) ctx->err = err; // (no call has failed)
    return rc;
}

// Room for what the slot's batch writes down of blocks' places (EntropyScratch::records); without it the index
// kernel decodes once more.  A context that has run short of memory does not ask again.
bool grow_records(ffcvb_ctx *ctx, Slot &s, size_t need) {
    if (need <= s.records.cap) return true;
    if (need > ctx->records_limit) return false;
    const std::string err = ctx->err;
    if (grow_dev(ctx, s.records, need) == FFCVB_OK) return true;
    cudaGetLastError();
    ctx->err = err; // (no call has failed)
    ctx->records_limit = 0;
    return false;
}

int grow_host(ffcvb_ctx *ctx, uint8_t *&p, size_t &cap_io, size_t need) {
    if (need <= cap_io) return 0;
    size_t cap = align_up(need + need / 4, 1 << 20);
    if (p) {
        CU(cudaDeviceSynchronize());
        CU(cudaFreeHost(p));
        p = nullptr;
        cap_io = 0;
    }
    CU(cudaHostAlloc((void **)&p, cap, cudaHostAllocDefault));
    cap_io = cap;
    return 0;
}

// The same for a buffer whose first `used` bytes have to stay.
int grow_host_keeping(ffcvb_ctx *ctx, uint8_t *&p, size_t &cap_io, size_t need, size_t used) {
    if (need <= cap_io) return 0;
    uint8_t *larger = nullptr;
    size_t cap = 0;
    const int rc = grow_host(ctx, larger, cap, need);
    if (rc) return rc;
    if (p) {
        memcpy(larger, p, used);
        CU(cudaDeviceSynchronize());
        CU(cudaFreeHost(p));
    }
    p = larger;
    cap_io = cap;
    return 0;
}

bool valid_plan(const ffcvb_plan *p) {
    if (!p || p->out_h <= 0 || p->out_w <= 0 || p->n_ops < 0 || p->n_ops > FFCVB_MAX_OPS) return false;
    if (p->out_kind < FFCVB_OUT_U8_NHWC || p->out_kind > FFCVB_OUT_F32_NCHW) return false;
    if (p->out_kind != FFCVB_OUT_U8_NHWC && !p->lut_dev) return false;
    for (int k = 0; k < p->n_ops; k++) {
        int t = p->ops[k].type;
        if (t != FFCVB_OP_FLIP && t != FFCVB_OP_TRANSLATE && t != FFCVB_OP_CUTOUT) return false;
        if (t != FFCVB_OP_FLIP && p->ops[k].arg < 0) return false;
    }
    if (p->dct_scale < -1 || p->dct_scale > 3 || (p->dct_scale < 0 && !p->resize)) return false;
    return true;
}

// The box of a sample decoded at reduced scale that covers its crop box.
void scaled_box(const ImageDesc &d, int32_t *p) {
    const int sh = d.scale_shift, r0 = p[0] >> sh, c0 = p[1] >> sh;
    int r1 = (p[0] + p[2] + (1 << sh) - 1) >> sh, c1 = (p[1] + p[3] + (1 << sh) - 1) >> sh;
    if (r1 > (int)d.dec_height) r1 = d.dec_height;
    if (c1 > (int)d.dec_width) c1 = d.dec_width;
    p[0] = r0;
    p[1] = c0;
    p[2] = r1 - r0;
    p[3] = c1 - c0;
}

OpList make_oplist(const ffcvb_plan &p) {
    OpList o{};
    o.n_ops = p.n_ops;
    for (int k = 0; k < p.n_ops; k++) {
        o.type[k] = p.ops[k].type;
        o.arg[k] = p.ops[k].arg;
        memcpy(o.fill[k], p.ops[k].fill, 4);
    }
    return o;
}

} // namespace

extern "C" {

int ffcvb_create(int device, int n_slots, int n_threads, ffcvb_ctx **out) {
    if (!out || n_slots < 1 || n_slots > 64) return FFCVB_E_ARG;
    *out = nullptr;
    int count = 0;
    if (cudaGetDeviceCount(&count) != cudaSuccess || count <= 0 || device < 0 || device >= count)
        return FFCVB_E_NODEVICE;
    if (cudaSetDevice(device) != cudaSuccess) return FFCVB_E_CUDA;
    if (n_threads <= 0) {
        long cores = sysconf(_SC_NPROCESSORS_ONLN);
        n_threads = (int)(cores < 1 ? 1 : (cores > 32 ? 32 : cores));
    }
    ffcvb_ctx *c = new ffcvb_ctx();
    c->device = device;
    c->slots.resize(n_slots);
    for (int i = 0; i < n_slots; i++) c->wait_args.push_back(WaitArg{c, i});
    c->pool = new Pool(n_threads - 1);
    auto env_int = [](const char *name, int lo, int hi) {
        const char *e = getenv(name);
        const int v = e ? atoi(e) : 0;
        return v >= lo && v <= hi ? v : 0;
    };
    c->tune_copy_threads = env_int("FFCV_B200_COPY_THREADS", 1, 256);
    c->tune_subseq_bits = env_int("FFCV_B200_SUBSEQ_BITS", 128, kMaxSubseqBits) / 32 * 32;
    c->gather_ctas = env_int("FFCV_B200_GATHER_CTAS", 1, 1024);
    if (const char *e = getenv("FFCV_B200_GATHER_LIMIT_MS"))
        if (*e >= '0' && *e <= '9') c->gather_limit_ns = (uint64_t)env_int("FFCV_B200_GATHER_LIMIT_MS", 0, 600000) * 1000000;
    if (const char *e = getenv("FFCV_B200_RECORDS_MB"))
        if (*e >= '0' && *e <= '9') c->records_limit = (size_t)env_int("FFCV_B200_RECORDS_MB", 0, 1 << 20) << 20;
    *out = c;
    return FFCVB_OK;
}

void ffcvb_destroy(ffcvb_ctx *ctx) {
    if (!ctx) return;
    ctx->pool->wait_all();
    cudaSetDevice(ctx->device);
    cudaDeviceSynchronize();
    for (auto &s : ctx->slots) {
        if (s.host) cudaFreeHost(s.host);
        for (DevBuf *b : {&s.blob, &s.clean, &s.segs, &s.records, &s.slot_tables, &s.index, &s.planes, &s.rgb})
            if (b->p) cudaFree(b->p);
        for (auto &e : s.ev)
            if (e) cudaEventDestroy(e);
        if (s.ev_begin) cudaEventDestroy(s.ev_begin);
        if (s.ev_done) cudaEventDestroy(s.ev_done);
        if (s.ev_copied) cudaEventDestroy(s.ev_copied);
        if (s.ev_gathered) cudaEventDestroy(s.ev_gathered);
        if (s.ev_gather_start) cudaEventDestroy(s.ev_gather_start);
    }
    for (auto &a : ctx->aux) {
        if (a.dev.p) cudaFree(a.dev.p);
        if (a.host) cudaFreeHost(a.host);
        if (a.ev) cudaEventDestroy(a.ev);
    }
    if (ctx->index_pool.p) cudaFree(ctx->index_pool.p);
    if (ctx->index_stats.p) cudaFree(ctx->index_stats.p);
    if (ctx->gather_failed) cudaFreeHost(ctx->gather_failed);
    if (ctx->copy_stream) cudaStreamDestroy(ctx->copy_stream);
    if (ctx->one_src.p) cudaFree(ctx->one_src.p);
    if (ctx->one_dst.p) cudaFree(ctx->one_dst.p);
    if (ctx->one_host) cudaFreeHost(ctx->one_host);
    if (ctx->one_in) cudaFreeHost(ctx->one_in);
    if (ctx->one_stream) cudaStreamDestroy(ctx->one_stream);
    for (auto &e : ctx->one_ev)
        if (e) cudaEventDestroy(e);
    delete ctx->pool;
    delete ctx;
}

const char *ffcvb_last_error(const ffcvb_ctx *ctx) { return ctx ? ctx->err.c_str() : "null context"; }

} // extern "C"

namespace {

// Where a batch's stored bytes come from: a mapping of the file (`base`), or file descriptors the
// staging threads read from straight into the slot's pinned buffer (`fd` buffered, `fd_direct`
// opened with O_DIRECT or -1).
struct Source {
    const uint8_t *base = nullptr;
    int fd = -1, fd_direct = -1;
    bool in_memory = false; // the file lies on a memory file system: every read is a copy by a core
    bool from_fd() const { return base == nullptr; }
};

// Reads [lo, lo + len) of the file into dst.  With O_DIRECT (offset, length and address are
// multiples of 4096 then) the bytes never enter the page cache; a file system that refuses it at
// read time is served through the buffered descriptor, whose pages are handed back afterwards so
// that resident memory stays bounded by the slot ring.  Returns the bytes read (short at EOF).
// What a core copies out of memory goes through a buffer of the thread's and past its caches: lines that lie dirty in
// the caches of cores which have gone to sleep make the transfer that fetches them many times as long (8.3 MB
// read by 8 threads: 518 us, 158 this way; whole passes over 24 samples of 400 KB of a tmpfs file 892 and 470 us, 256 of 65 KB of
// an ext4 file through the page cache 9.5 and 8.9 ms).  A file on a memory file system is read by cores even with O_DIRECT.
size_t read_range(const Source &src, std::atomic<bool> &direct_broken, uint8_t *dst, uint64_t lo, size_t len) {
    constexpr size_t kThrough = 64 * 1024;
    struct Free {
        void operator()(uint8_t *p) const { free(p); }
    };
    thread_local std::unique_ptr<uint8_t, Free> through;
    size_t done = 0;
    bool use_direct = src.fd_direct >= 0 && !direct_broken.load(std::memory_order_relaxed);
    while (done < len) {
        const bool copied = !use_direct || src.in_memory;
        if (copied && !through) through.reset(static_cast<uint8_t *>(aligned_alloc(4096, kThrough)));
        const bool past = copied && through;
        const size_t want = past && len - done > kThrough ? kThrough : len - done;
        const ssize_t got = pread(use_direct ? src.fd_direct : src.fd, past ? through.get() : dst + done, want, (off_t)(lo + done));
        if (got < 0) {
            if (errno == EINTR) continue;
            if (use_direct && errno == EINVAL) { // O_DIRECT not supported here after all
                direct_broken.store(true, std::memory_order_relaxed);
                use_direct = false;
                continue;
            }
            break;
        }
        if (got == 0) break; // end of file
        if (past) stream_copy(dst + done, through.get(), (size_t)got);
        done += (size_t)got;
        if (use_direct && (done & 4095)) break; // a short direct read only happens at the end of the file
    }
    _mm_sfence(); // (streaming stores are weakly ordered)
    if (!use_direct && !src.in_memory && done) posix_fadvise(src.fd, (off_t)lo, (off_t)done, POSIX_FADV_DONTNEED);
    return done;
}

int stage_impl(ffcvb_ctx *ctx, int slot, const Source &source, const uint64_t *ptrs,
               const uint64_t *sizes, const uint8_t *modes, const uint16_t *heights,
               const uint16_t *widths, int n, const ffcvb_plan *plan, const int32_t *params) {
    const uint8_t *file_base = source.base;
    const bool from_fd = source.from_fd();
    if (!ctx) return FFCVB_E_ARG;
    if (slot < 0 || slot >= (int)ctx->slots.size() || n <= 0 || (!file_base && source.fd < 0) || !ptrs || !sizes ||
        !modes || !heights || !widths || !params)
        return fail(ctx, FFCVB_E_ARG, "ffcvb_stage_batch: bad argument");
    if (!valid_plan(plan)) return fail(ctx, FFCVB_E_ARG, "ffcvb_stage_batch: invalid plan");
    CU(cudaSetDevice(ctx->device));
    Slot &s = ctx->slots[slot];
    if (s.in_flight) { // normally complete long ago (the caller fences the ring): returns at once
        CU(cudaEventSynchronize(s.ev_copied));
        s.in_flight = false;
    }
    s.staged = false;
    s.plan = *plan;
    s.n = n;
    const int n_params = 4 + 2 * plan->n_ops;
    const auto t0 = std::chrono::steady_clock::now();
    // A source that lives in pinned (page-locked, device-mapped) host memory is not copied by the
    // CPU: the GPU gathers the payloads itself.
    uint64_t src_dev_base = 0;
    if (!from_fd) {
        cudaPointerAttributes attr;
        memset(&attr, 0, sizeof(attr));
        if (cudaPointerGetAttributes(&attr, file_base) == cudaSuccess && attr.type == cudaMemoryTypeHost &&
            attr.devicePointer != nullptr)
            src_dev_base = (uint64_t)(uintptr_t)attr.devicePointer;
        else
            cudaGetLastError(); // pageable memory: not an error
    }
    const bool direct = src_dev_base != 0;
    s.direct = direct;
    {   // a copy of this very slot that was never submitted may still be running
        bool done;
        {
            std::lock_guard<std::mutex> g(ctx->copy_m);
            done = s.copy_done;
        }
        if (!done) ctx->pool->wait(Pool::kAsync);
    }
    std::vector<ImageDesc> &descs = s.descs;
    descs.assign(n, ImageDesc{});
    s.src_ptrs.assign(ptrs, ptrs + n);
    s.headers.resize(n);

    // ---- reading from file descriptors: every sample's bytes get their place in the pinned buffer
    // before anything is parsed (a JPEG header can only be parsed once it has been read), so the
    // parts of the blob whose size depends on the headers (tables, index lists) follow the payloads.
    // With O_DIRECT a sample is read as the 4 KiB file blocks that contain it, into a 4 KiB aligned
    // place: its first byte sits at the same offset inside a block as in the file.
    struct Span {
        uint64_t lo = 0;   // file offset the read starts at
        size_t len = 0;    // bytes to read
        size_t dst = 0;    // offset in the pinned buffer the read goes to
        size_t skip = 0;   // the sample's first byte is dst + skip
        uint64_t want = 0; // bytes of the sample needed from lo + skip on
    };
    std::vector<Span> spans;
    std::vector<uint8_t> short_read;
    const int n_params_early = 4 + 2 * plan->n_ops;
    size_t fd_payload_begin = 0, fd_payload_end = 0;
    if (from_fd) {
        const size_t A = source.fd_direct >= 0 && !ctx->direct_broken.load() ? 4096 : kPayloadAlign;
        size_t off = align_up(sizeof(BatchHeader), 16);
        off = align_up(off + sizeof(ImageDesc) * (size_t)n, 16);
        off = align_up(off + sizeof(int32_t) * (size_t)n * n_params_early, 16);
        off = align_up(off + 2 * sizeof(int32_t) * (size_t)n, 16);
        if (plan->resize) off += sizeof(ResizeItem) * (size_t)n;
        for (const auto &r : s.pending_riders) off = align_up(off, 64) + r.item_bytes * (uint64_t)n;
        fd_payload_begin = off = align_up(off, A);
        spans.resize(n);
        for (int i = 0; i < n; i++) {
            uint64_t start = ptrs[i], want = sizes[i];
            if (modes[i] != FFCVB_MODE_JPG) {
                int r0 = 0, rows = heights[i];
                const int32_t *p = params + (size_t)i * n_params_early;
                if (plan->resize && p[0] >= 0 && p[2] > 0 && p[0] + p[2] <= (int)heights[i] && p[1] >= 0 && p[3] > 0 &&
                    p[1] + p[3] <= (int)widths[i]) {
                    r0 = p[0];
                    rows = p[2];
                }
                const uint64_t pitch = (uint64_t)widths[i] * 3;
                if (sizes[i] < pitch * heights[i]) rows = 0; // short payload: flagged below, nothing read
                start += (uint64_t)r0 * pitch;
                want = (uint64_t)rows * pitch;
            }
            Span &sp = spans[i];
            sp.want = want;
            sp.lo = start / A * A;
            sp.skip = (size_t)(start - sp.lo);
            sp.len = want ? align_up(sp.skip + want, A) : 0;
            sp.dst = off = align_up(off, A);
            off += sp.len;
        }
        fd_payload_end = off;
        // room behind the payloads for what is laid out after the parse: more tables of each kind than the images of
        // a few encoders have (with more of them the buffer grows below)
        size_t tail = 16 * (sizeof(HuffTable) + sizeof(MultTable)) + 4 * (sizeof(int32_t) * (size_t)n + 16) + 256;
        for (int i = 0; i < n; i++) { // and the tables of CTAs: at most those of whole images and of the shortest segments
            tail += sizeof(uint2) * (size_t)quad_tiles_x(widths[i]) * quad_tiles_y(heights[i]);
            tail += sizeof(uint2) * ((size_t)((heights[i] + 15) / 8) * ((widths[i] + 15) / 8) * 3 / kBlockTile + 4);
            tail += sizeof(uint2) * (size_t)(sizes[i] / (64 * kSegSubs / 8) + 2);
            tail += sizeof(uint4) * (size_t)(sizes[i] / (64 * kSegSubs / 8 * kRepairPart) + 3);
        }
        int grc;
        if ((grc = grow_host(ctx, s.host, s.host_cap, fd_payload_end + tail))) return grc;
        short_read.assign(n, 0);
        // Few samples that cores copy are shared out in pieces (that end on pages of the file), or the largest ones would decide.  What a
        // disk sends by itself is not: 24 samples of 400 KB from an ext4 file with O_DIRECT take 4.0 to 4.9 ms in pieces, 3.5 to 4.4
        // whole, one of 1.5 MB 0.78 to 0.95 and 0.68 to 0.86.
        struct Piece {
            int sample;
            size_t from, len;
        };
        std::vector<Piece> pieces;
        const uint64_t step = n < 4 * ctx->pool->size() && (source.in_memory || source.fd_direct < 0) ? 128 * 1024 : ~0ull;
        for (int i = 0; i < n; i++)
            for (size_t from = 0; from < spans[i].len;) {
                const uint64_t room = step - (step == ~0ull ? 0 : (spans[i].lo + from) % step), left = spans[i].len - from;
                pieces.push_back(Piece{i, from, (size_t)(left < room ? left : room)});
                from += pieces.back().len;
            }
        ctx->pool->parallel_for((int)pieces.size(), 1, [&](int k) {
            const Piece &c = pieces[k];
            const Span &sp = spans[c.sample];
            const uint64_t need = sp.skip + sp.want; // of the sample's place
            const size_t got = read_range(source, ctx->direct_broken, s.host + sp.dst + c.from, sp.lo + c.from, c.len);
            if (c.from < need && got < c.len && c.from + got < need) __atomic_store_n(&short_read[c.sample], (uint8_t)1, __ATOMIC_RELAXED);
        });
    }
    auto bytes_of = [&](int i) -> const uint8_t * { return from_fd ? s.host + spans[i].dst + spans[i].skip : file_base + ptrs[i]; };

    // ---- headers: from the cache, or parsed (in parallel when there are many)
    if (ctx->tables.full()) {
        ctx->tables.clear();
        ctx->header_cache.clear();
    }
    s.to_parse.clear();
    for (int i = 0; i < n; i++) {
        if (modes[i] != FFCVB_MODE_JPG) continue;
        const StreamHeader *hit = ctx->cache_headers ? ctx->header_cache.find(ptrs[i]) : nullptr;
        if (hit && hit->size == sizes[i] && !(from_fd && short_read[i]))
            s.headers[i] = *hit;
        else
            s.to_parse.push_back(i);
    }
    if (!s.to_parse.empty()) {
        const int m = (int)s.to_parse.size();
        s.parsed.resize(m);
        s.hashes.resize(m);
        auto parse = [&](int k) {
            const int i = s.to_parse[k];
            JpegHeader &h = s.parsed[k];
            StreamHeader &o = s.headers[i];
            o = StreamHeader{};
            o.size = sizes[i];
            o.status = (int16_t)(from_fd && short_read[i] ? kErrData : parse_jpeg_header(bytes_of(i), (size_t)sizes[i], &h));
            if (o.status != 0) return;
            o.scan_off = (uint32_t)h.scan_off;
            o.scan_len = (uint32_t)h.scan_len;
            o.restart_interval = (uint16_t)h.restart_interval;
            o.width = (uint16_t)h.width;
            o.height = (uint16_t)h.height;
            o.ncomp = (uint8_t)h.ncomp;
            o.hs = (uint8_t)h.hs[0];
            o.vs = (uint8_t)h.vs[0];
            // (bits[17] and vals[256] lie next to each other in RawHuff)
            static_assert(offsetof(RawHuff, vals) == 17, "RawHuff: vals must follow bits");
            for (int c = 0; c < h.ncomp; c++) {
                uint64_t *th = &s.hashes[k][3 * c];
                if (c == 2 && h.td[2] == h.td[1] && h.ta[2] == h.ta[1] && h.tq[2] == h.tq[1]) {
                    memcpy(th, th - 3, 3 * sizeof(uint64_t));
                    continue;
                }
                th[0] = hash_bytes(h.dc[h.td[c]].bits, 17 + 256) & ~1ull; // (the same code as a DC and as an AC table: two tables)
                th[1] = hash_bytes(h.ac[h.ta[c]].bits, 17 + 256) | 1ull;
                th[2] = hash_bytes(h.quant[h.tq[c]], 128);
            }
            o.table_set = ctx->tables.find(h, s.hashes[k].data()); // (here, where the tables are in this thread's cache)
        };
        if (m < 12) // waking the staging threads takes longer
            for (int k = 0; k < m; k++) parse(k);
        else
            ctx->pool->parallel_for(m, 8, parse);
        for (int k = 0; k < m; k++) { // their tables enter the stores, the headers the cache
            const int i = s.to_parse[k];
            if (s.headers[i].status != 0) continue;
            if (s.headers[i].table_set == TableStore::kNone) s.headers[i].table_set = ctx->tables.add(s.parsed[k], s.hashes[k].data());
            if (ctx->cache_headers && ctx->header_cache.size() < (size_t)1 << 23) // ~0.9 GB of host memory at most
                ctx->header_cache.insert(ptrs[i], s.headers[i]);
        }
    }

    // ---- what is needed of every sample
    for (int i = 0; i < n; i++) {
        ImageDesc &d = descs[i];
        d.mode = modes[i];
        d.height = heights[i];
        d.width = widths[i];
        const int32_t *p = params + (size_t)i * n_params;
        const bool box_ok = plan->resize && p[0] >= 0 && p[2] > 0 && p[0] + p[2] <= (int)d.height && p[1] >= 0 && p[3] > 0 &&
                            p[1] + p[3] <= (int)d.width;
        if (modes[i] == FFCVB_MODE_JPG) {
            const StreamHeader &h = s.headers[i];
            d.payload_size = (uint32_t)sizes[i];
            d.host_status = h.status == 0 && (h.width != d.width || h.height != d.height) ? (int16_t)kErrDims : h.status;
            if (d.host_status == 0) {
                d.scan_off = h.scan_off;
                d.scan_len = h.scan_len;
                d.ncomp = h.ncomp;
                d.hs = h.hs;
                d.vs = h.vs;
                d.bpm = (uint8_t)(h.ncomp == 1 ? 1 : h.hs * h.vs + 2);
                d.mcus_x = (uint16_t)((h.width + 8 * h.hs - 1) / (8 * h.hs));
                d.mcus_y = (uint16_t)((h.height + 8 * h.vs - 1) / (8 * h.vs));
                d.restart_interval = h.restart_interval;
                d.mcu_rows = d.mcus_y;
                d.idct_row0 = d.idct_col0 = 0;
                d.idct_col1 = d.mcus_x;
                const bool three = h.ncomp == 3, even = h.hs == 1 && h.vs == 1, quad = h.hs == 2 && h.vs == 2;
                // With a crop box only part of the image is needed.  The colour kernels of 4:2:0
                // and 4:4:4 images convert the box alone and reach at most one chroma sample
                // (two pixels, three with an odd edge) beyond it; other layouts convert the whole image.
                if (box_ok && three && ((quad && (h.width + 1) / 2 >= 3) || even)) {
                    const int mh = 8 * d.vs, mw = 8 * d.hs;
                    const int y0 = p[0] - 3 < 0 ? 0 : p[0] - 3, x0 = p[1] - 3 < 0 ? 0 : p[1] - 3;
                    const int y1 = p[0] + p[2] + 3 > (int)d.height ? (int)d.height : p[0] + p[2] + 3;
                    const int x1 = p[1] + p[3] + 3 > (int)d.width ? (int)d.width : p[1] + p[3] + 3;
                    d.idct_row0 = (uint16_t)(y0 / mh);
                    d.mcu_rows = (uint16_t)((y1 - 1) / mh + 1);
                    d.idct_col0 = (uint16_t)(x0 / mw);
                    d.idct_col1 = (uint16_t)((x1 - 1) / mw + 1);
                }
                d.nblocks = (uint32_t)d.bpm * d.mcus_x * d.mcu_rows;
                // scale of the decode (plan->dct_scale): only layouts whose planes end up at one resolution
                const bool scalable = three && (even || quad);
                int shift = 0;
                if (plan->dct_scale > 0) {
                    shift = plan->dct_scale;
                    if (!scalable) d.host_status = (int16_t)kErrUnsupported;
                } else if (plan->dct_scale < 0 && scalable && box_ok) {
                    while (shift < 3 && (p[2] >> (shift + 1)) >= plan->out_h && (p[3] >> (shift + 1)) >= plan->out_w) shift++;
                }
                d.scale_shift = (uint8_t)shift;
                d.bs_luma = (uint8_t)(8 >> shift);
                d.bs_chroma = (uint8_t)((8 >> shift) * h.hs > 8 ? 8 : (8 >> shift) * h.hs);
            }
            d.dec_height = (uint16_t)((d.height + (1 << d.scale_shift) - 1) >> d.scale_shift);
            d.dec_width = (uint16_t)((d.width + (1 << d.scale_shift) - 1) >> d.scale_shift);
            if (d.bs_luma == 0) d.bs_luma = d.bs_chroma = 8; // rejected stream: fields stay consistent
            if (direct) d.src_addr = src_dev_base + ptrs[i];
        } else {
            d.dec_height = d.height;
            d.dec_width = d.width;
            int r0 = 0, rows = d.height, c0 = 0, cols = d.width;
            if (box_ok) {
                r0 = p[0];
                rows = p[2];
                c0 = p[1];
                cols = p[3];
            }
            const uint64_t need = (uint64_t)d.height * d.width * 3;
            if (sizes[i] < need || (from_fd && short_read[i])) {
                d.host_status = (int16_t)kErrData;
                rows = 0;
            }
            if (from_fd) { // whole rows were read: the crop's columns are picked on the GPU
                c0 = 0;
                cols = d.width;
            }
            d.row0 = (uint16_t)r0;
            d.rows = (uint16_t)rows;
            d.col0 = (uint16_t)c0;
            d.cols = (uint16_t)cols;
            d.raw_pitch = (uint32_t)cols * 3;
            d.payload_size = (uint32_t)((size_t)rows * d.raw_pitch);
            if (direct && rows > 0) d.src_addr = src_dev_base + ptrs[i] + ((uint64_t)r0 * d.width + c0) * 3;
        }
    }

    const auto t1 = std::chrono::steady_clock::now();
    // Split staging: with a pinned source the staging threads (and the copy engine) can carry part
    // of the bytes while the GPU gathers the rest, so that neither path alone has to fill the link.
    // Samples are dealt to the CPU side greedily so that its share of the running byte count holds.
    // Samples that follow one another in the file (a sequential pass) need no gather: the copy engine
    // takes the whole piece, at the link's full rate and beside the kernels.  Worth it as long as little
    // else lies between them.
    s.range_len = 0;
    if (direct) {
        uint64_t lo = ~0ull, hi = 0, sum = 0;
        bool whole = true;
        for (int i = 0; i < n && whole; i++) {
            const ImageDesc &d = descs[i];
            if (d.src_addr == 0 || d.payload_size == 0) continue;
            whole = d.mode == FFCVB_MODE_JPG || d.cols == d.width;
            lo = d.src_addr < lo ? d.src_addr : lo;
            hi = d.src_addr + d.payload_size > hi ? d.src_addr + d.payload_size : hi;
            sum += d.payload_size;
        }
        if (whole && sum > 0 && hi - lo <= sum + sum / 16 + 4096) {
            lo &= ~15ull;
            s.range_src = file_base + (lo - src_dev_base);
            s.range_len = (size_t)(hi - lo);
        }
    }
    if (direct && ctx->adaptive_split && s.range_len == 0) {
        // The slot's previous batch tells how long its two halves took: the staging threads' copy
        // (host clock) and the GPU's gather (events).  While the gather takes most of the time between two
        // batches the link is what they wait for: move the share towards equal times, in small steps
        // because the measurement is several batches old.  Otherwise the threads' help is not needed.
        const auto now = std::chrono::steady_clock::now();
        const double since = ctx->last_staged.time_since_epoch().count()
                                 ? std::chrono::duration<double, std::milli>(now - ctx->last_staged).count() : 0.0;
        ctx->last_staged = now;
        if (since > 0 && since < 100) ctx->batch_interval = ctx->batch_interval > 0 ? 0.75 * ctx->batch_interval + 0.25 * since : since;
        float tg = 0;
        if (s.gather_timed && cudaEventElapsedTime(&tg, s.ev_gather_start, s.ev_gathered) == cudaSuccess) {
            const double tc = s.staged_end > s.hdr.payload_off ? s.stage_ms[2] : 0.0;
            if (tg < 0.7 * ctx->batch_interval && tc < 0.7 * ctx->batch_interval)
                ctx->share = ctx->share < 0.02 ? 0 : 0.8 * ctx->share;
            else if (tg + tc > 0)
                ctx->share += 0.04 * ((double)tg - tc) / ((double)tg + tc);
            if (ctx->share < 0) ctx->share = 0;
            if (ctx->share > kMaxAdaptiveShare) ctx->share = kMaxAdaptiveShare;
        } else {
            cudaGetLastError(); // not run yet, or still running: keep the share
        }
        s.gather_timed = false;
        ctx->cpu_share_permille = (int)(ctx->share * 1000 + 0.5);
    }
    if (direct && ctx->cpu_share_permille > 0 && s.range_len == 0) {
        uint64_t total = 0, cpu = 0;
        for (int i = 0; i < n; i++) {
            total += descs[i].payload_size;
            if (cpu * 1000 < total * (uint64_t)ctx->cpu_share_permille) {
                cpu += descs[i].payload_size;
                descs[i].src_addr = 0;
            }
        }
    }
    // ---- layout of the JPEG samples' work; the batch's own table lists (indices into the store ->
    // indices into the blob), worked out once per table set
    std::vector<uint32_t> huff_src, mult_src;
    struct BatchSet {
        uint32_t set;
        uint8_t tab_id[6], q_tab[kMaxComponents];
    };
    std::vector<BatchSet> batch_sets;
    int last_set = -1;
    std::vector<int32_t> &jpeg_list = s.jpeg_list, &slot_images = s.slot_images, &restart = s.restart;
    std::vector<uint2> &segs = s.seg_list, &blk_tiles = s.blk_tiles, &quad_tiles = s.quad_tiles;
    jpeg_list.clear();
    s.parts.clear();
    s.wholes.clear();
    slot_images.clear();
    s.slot_segs.clear();
    restart.clear();
    segs.clear();
    blk_tiles.clear();
    quad_tiles.clear();
    size_t clean_bytes = 0, plane_bytes = 0, rgb_bytes = 0;
    uint32_t total_blocks = 0;
    EntropyWork &work = s.work;
    work = EntropyWork{};
    work.max_tables = 1;
    work.alike = true;
    int first_jpeg = -1;
    // Subsequence length: by the batch's bits, or, with a decode index, a function of the stream alone
    // (1024 bits), so that the recorded states stay usable whatever batch the sample lands in.
    uint32_t target_bits = 1024, seg_total = 0;
    uint64_t records = 0; // room for them, / 4
    bool few = false; // few enough bits to decode from every slot at once
    uint64_t bits = 0;
    for (int i = 0; i < n; i++)
        if (descs[i].mode == FFCVB_MODE_JPG && descs[i].host_status == 0) bits += (uint64_t)descs[i].scan_len * 8;
    if (!ctx->index_pool.p) {
        target_bits = subseq_target(bits);
        few = bits <= kSlotModeBits && !ctx->tune_subseq_bits;
    }
    if (ctx->tune_subseq_bits) target_bits = (uint32_t)ctx->tune_subseq_bits;
    work.local_repair = !ctx->index_pool.p && local_repair(target_bits, n);
    if (ctx->index_pool.p) {
        for (size_t k = 0; k < ctx->slots.size(); k++) { // whose writers have ended
            if (!ctx->index.unsettled((int)k)) continue;
            if (cudaEventQuery(ctx->slots[k].ev_done) == cudaSuccess)
                ctx->index.ended((int)k);
            else
                cudaGetLastError(); // still running
        }
        ctx->index.staged(slot);
    }
    s.index_life = ctx->index_life;
    int max_w = 0, max_h = 0, n_quad = 0, n_444 = 0, n_other = 0;
    const bool can_fuse = plan->resize && !s.packed;
    ResizeItems items(n, plan->out_h, plan->out_w, plan->out_kind);
    s.items.resize(plan->resize ? n : 0);
    for (int i = 0; i < n; i++) {
        ImageDesc &d = descs[i];
        if (plan->resize) {
            // The resize kernel converts the planes of a 4:2:0 or equal-resolution image itself, into its window
            // of source pixels, if the regime is one that works from a window and enough rows fit.
            int32_t box[4];
            memcpy(box, params + (size_t)i * n_params, sizeof(box));
            if (d.scale_shift) scaled_box(d, box);
            ResizeItems::Fuse fuse = ResizeItems::kPacked;
            if (can_fuse && d.mode == FFCVB_MODE_JPG && d.host_status == 0 && d.ncomp == 3) {
                if (d.scale_shift != 0 || (d.hs == 1 && d.vs == 1))
                    fuse = ResizeItems::kFusePlain;
                else if (d.hs == 2 && d.vs == 2 && (d.width + 1) / 2 >= 3)
                    fuse = ResizeItems::kFuseQuad;
            }
            s.items[i] = items.make(box, d.dec_height, d.dec_width, fuse);
            if (fuse != ResizeItems::kPacked) d.fuse_rows = (uint16_t)s.items[i].window;
        }
        if (d.mode != FFCVB_MODE_JPG) continue;
        jpeg_list.push_back(i);
        if (d.host_status != 0) { // (no kernel touches it: its status word says so)
            d.block_base = total_blocks;
            continue;
        }
        const uint32_t set_id = s.headers[i].table_set;
        const TableSet &ts = ctx->tables.set(set_id);
        if (last_set < 0 || batch_sets[last_set].set != set_id) {
            for (last_set = (int)batch_sets.size() - 1; last_set >= 0 && batch_sets[last_set].set != set_id;) last_set--;
            if (last_set < 0) {
                BatchSet bs{};
                bs.set = set_id;
                for (int k = 0; k < ts.n_tab; k++) {
                    size_t u = 0;
                    while (u < huff_src.size() && huff_src[u] != ts.huff[k]) u++;
                    if (u == huff_src.size()) huff_src.push_back(ts.huff[k]);
                    bs.tab_id[k] = (uint8_t)u;
                }
                for (int c = 0; c < d.ncomp; c++) {
                    size_t u = 0;
                    while (u < mult_src.size() && mult_src[u] != ts.quant[c]) u++;
                    if (u == mult_src.size()) mult_src.push_back(ts.quant[c]);
                    bs.q_tab[c] = (uint8_t)u;
                }
                if (huff_src.size() > 255 || mult_src.size() > 255)
                    return fail(ctx, FFCVB_E_LIMIT, "more than 255 distinct Huffman or quantisation tables in a batch");
                last_set = (int)batch_sets.size();
                batch_sets.push_back(bs);
            }
        }
        d.fast_tables = ts.fast;
        d.n_tab = ts.n_tab;
        d.n_dc_tab = ts.n_dc_tab;
        memcpy(d.tab_id, batch_sets[last_set].tab_id, sizeof(d.tab_id));
        memcpy(d.dc_tab, ts.dc_tab, sizeof(d.dc_tab));
        memcpy(d.ac_tab, ts.ac_tab, sizeof(d.ac_tab));
        memcpy(d.q_tab, batch_sets[last_set].q_tab, sizeof(d.q_tab));
        d.block_base = total_blocks;
        total_blocks += d.nblocks;
        if (2 * d.n_tab - d.n_dc_tab > work.max_tables) work.max_tables = 2 * d.n_tab - d.n_dc_tab;
        if (first_jpeg < 0) first_jpeg = i;
        const ImageDesc &f = descs[first_jpeg];
        work.alike = work.alike && d.bpm == f.bpm && d.hs == f.hs && d.n_tab == f.n_tab && d.n_dc_tab == f.n_dc_tab &&
                memcmp(d.tab_id, f.tab_id, sizeof(d.tab_id)) == 0 && memcmp(d.dc_tab, f.dc_tab, sizeof(d.dc_tab)) == 0 &&
                memcmp(d.ac_tab, f.ac_tab, sizeof(d.ac_tab)) == 0;
        d.clean_off = clean_bytes;
        if (d.restart_interval) { // table of interval starts behind the clean stream
            clean_bytes += align_up((size_t)d.scan_len + 96, 16);
            d.rst_off = clean_bytes;
            const size_t mcus = (size_t)d.mcus_x * d.mcus_y;
            clean_bytes += align_up(4 * ((mcus + d.restart_interval - 1) / d.restart_interval + 2), 16);
            restart.push_back(i);
        } else {
            const bool slots = few && d.bpm > 3; // (a guess among three slots falls in step within 1.4 kbit)
            const ScanLayout l = slots ? layout_scan_slots(d.scan_len) : layout_scan(d.scan_len, target_bits, d.bpm, work.local_repair, ctx->index_pool.p != nullptr);
            d.subseq_bits = l.subseq_bits;
            d.seg_raw = l.seg_raw;
            d.seg_warm = l.seg_warm;
            d.seg_run_up = l.seg_run_up;
            d.seg_stride = l.seg_stride;
            d.seg_count = l.seg_count;
            d.seg_lanes = l.seg_lanes;
            d.seg_first = seg_total;
            seg_total += l.seg_count;
            clean_bytes += (size_t)l.seg_count * l.seg_stride;
            if (slots) {
                d.slots = 1 + (uint32_t)s.slot_segs.size();
                slot_images.push_back(i);
                if ((int)l.seg_count > work.max_slot_segs) work.max_slot_segs = (int)l.seg_count;
            } else {
                const uint32_t parts = repair_parts(l.seg_count, work.local_repair);
                for (uint32_t k = 0; k < parts; k++) s.parts.push_back(repair_part((uint32_t)i, l.seg_count, parts, k));
                if (parts > 1) s.wholes.push_back(make_uint4((uint32_t)i, 0, l.seg_count, 0));
                if (l.subseq_bits > work.max_subseq_bits) work.max_subseq_bits = l.subseq_bits;
                d.rec_room = record_room(l.subseq_bits, d.scan_len, (uint32_t)d.bpm * d.mcus_x * d.mcus_y, bits <= kAllRecordsBits);
                d.rec_first = (uint32_t)records;
                records += (uint64_t)l.seg_count * l.seg_lanes * d.rec_room / 4;
            }
            for (uint32_t k = 0; k < l.seg_count; k++) (slots ? s.slot_segs : segs).push_back(make_uint2((uint32_t)i, k));
            const uint32_t raw = l.seg_stride - 64 - 16; // (at least run-up, own bytes and overlap)
            if (raw > work.max_raw) work.max_raw = raw;
            if (ctx->index_pool.p) {
                const DecodeIndex::Place place = ctx->index.take(ptrs[i], l.seg_count, decode_index_bytes(l.seg_count, l.seg_lanes), slot);
                d.index_off = place.off;
                d.index_use = place.use;
            }
        }
        {
            const uint32_t tiles = block_tiles(d);
            for (uint32_t k = 0; k < tiles; k++) blk_tiles.push_back(make_uint2((uint32_t)i, k));
        }
        for (int c = 0; c < d.ncomp; c++) {
            d.plane_off[c] = plane_bytes;
            const size_t pw = (size_t)d.mcus_x * (c == 0 ? d.hs * d.bs_luma : d.bs_chroma);
            const size_t ph = (size_t)d.mcus_y * (c == 0 ? d.vs * d.bs_luma : d.bs_chroma);
            plane_bytes += align_up(pw * ph, 16);
        }
        d.rgb_off = rgb_bytes;
        d.rgb_pitch = s.packed ? (uint32_t)d.dec_width * 3 : (uint32_t)align_up((size_t)d.dec_width * 3, 16);
        if (d.fuse_rows) continue;
        rgb_bytes += (size_t)d.dec_height * d.rgb_pitch;
        int bw = d.dec_width, bh = d.dec_height;
        {   // extent the colour kernels' grids must cover: the crop box (plus the odd edge of a
            // chroma cell) where the kernel converts only that, else the whole image
            const bool boxed = d.ncomp == 3 && ((d.hs == 2 && d.vs == 2 && (d.width + 1) / 2 >= 3) || (d.hs == 1 && d.vs == 1));
            if (plan->resize && boxed) {
                const int32_t *p = params + (size_t)i * n_params;
                if (p[0] >= 0 && p[2] > 0 && p[0] + p[2] <= (int)d.height && p[1] >= 0 && p[3] > 0 &&
                    p[1] + p[3] <= (int)d.width) {
                    const int sw = (p[3] >> d.scale_shift) + 2, sh = (p[2] >> d.scale_shift) + 2; // the box at the decode's scale
                    bw = sw < bw ? sw : bw;
                    bh = sh < bh ? sh : bh;
                }
            }
            if (bw > max_w) max_w = bw;
            if (bh > max_h) max_h = bh;
        }
        if (d.scale_shift != 0)
            n_444++; // decoded at reduced scale: all planes at one resolution, no upsampling
        else if (d.ncomp == 3 && d.hs == 2 && d.vs == 2 && (d.width + 1) / 2 >= 3) {
            n_quad++;
            // the tiles of 64 x 8 chroma samples (one CTA each) that cover this image's box
            const uint32_t tiles_x = quad_tiles_x(bw), tiles_y = quad_tiles_y(bh);
            for (uint32_t ty = 0; ty < tiles_y; ty++)
                for (uint32_t tx = 0; tx < tiles_x; tx++) quad_tiles.push_back(make_uint2((uint32_t)i, tx | ty << 16));
        } else if (d.ncomp == 3 && d.hs == 1 && d.vs == 1)
            n_444++;
        else
            n_other++;
    }

    BatchHeader &hd = s.hdr;
    memset(&hd, 0, sizeof(hd));
    hd.n = (uint32_t)n;
    hd.n_huff = (uint32_t)huff_src.size();
    hd.n_mult = (uint32_t)mult_src.size();
    hd.n_params = (uint32_t)n_params;
    size_t off = align_up(sizeof(BatchHeader), 16);
    hd.desc_off = off;
    off = align_up(off + sizeof(ImageDesc) * (size_t)n, 16);
    auto place_tables = [&] {
        hd.huff_off = off;
        off = align_up(off + sizeof(HuffTable) * huff_src.size(), 16);
        hd.mult_off = off;
        off = align_up(off + sizeof(MultTable) * mult_src.size(), 16);
    };
    auto place_lists = [&] {
        s.jpeg_list_off = off;
        off = align_up(off + sizeof(int32_t) * jpeg_list.size(), 16);
        s.parts_off = off;
        off = align_up(off + sizeof(uint4) * (s.parts.size() + s.wholes.size()), 16);
        s.slot_images_off = off;
        off = align_up(off + sizeof(int32_t) * slot_images.size(), 16);
        s.restart_off = off;
        off = align_up(off + sizeof(int32_t) * restart.size(), 16);
        s.segs_off = off;
        off = align_up(off + sizeof(uint2) * (segs.size() + s.slot_segs.size()), 16);
        s.block_tiles_off = off;
        off = align_up(off + sizeof(uint2) * blk_tiles.size(), 16);
        s.quad_tiles_off = off;
        off = align_up(off + sizeof(uint2) * quad_tiles.size(), 16);
        s.gather_off = off;
        s.gather_ctas = direct && s.range_len == 0 ? (ctx->gather_ctas < 1 ? kGatherCtas : ctx->gather_ctas) : 0;
        if (s.gather_ctas) off = align_up(off + sizeof(uint2) * (s.gather_ctas + 1), 16);
    };
    if (!from_fd) place_tables();
    hd.params_off = off;
    off = align_up(off + sizeof(int32_t) * (size_t)n * n_params, 16);
    s.status_off = off;
    off = align_up(off + 2 * sizeof(int32_t) * (size_t)n, 16);
    s.items_off = off;
    off += sizeof(ResizeItem) * s.items.size();
    s.riders.swap(s.pending_riders);
    s.pending_riders.clear();
    for (auto &r : s.riders) {
        r.bytes = r.item_bytes * (uint64_t)n;
        if ((!r.inline_bytes.empty() && r.inline_bytes.size() != r.bytes) ||
            (r.inline_bytes.empty() && r.ptrs.size() != (size_t)n)) {
            s.riders.clear();
            return fail(ctx, FFCVB_E_ARG, "ffcvb_stage_batch: a rider was set for a different number of samples");
        }
        r.off = off = align_up(off, 64);
        off += r.bytes;
    }
    off = align_up(off, 16);
    if (from_fd) {
        // the payloads were read into their places before the parse; tables and lists follow them
        if (off > fd_payload_begin) return fail(ctx, FFCVB_E_ARG, "ffcvb_stage_batch: the riders changed while the batch was staged");
        hd.payload_off = fd_payload_begin;
        for (int i = 0; i < n; i++) descs[i].payload_off = spans[i].dst + spans[i].skip;
        off = align_up(fd_payload_end, 16);
        place_tables();
        place_lists();
        s.staged_end = off;
    } else {
        place_lists();
        hd.payload_off = off;
        // payloads the staging threads copy come first: they travel with the head of the blob
        for (int i = 0; i < n; i++) {
            if (descs[i].src_addr != 0) continue;
            descs[i].payload_off = off;
            off = align_up(off + descs[i].payload_size, kPayloadAlign);
        }
        s.staged_end = off;
        if (s.range_len) {
            const uint64_t lo = src_dev_base + (uint64_t)(s.range_src - file_base);
            for (int i = 0; i < n; i++)
                if (descs[i].src_addr != 0) descs[i].payload_off = off + (descs[i].src_addr - lo);
            off = align_up(off + s.range_len, kPayloadAlign);
        }
        for (int i = 0; i < n && s.range_len == 0; i++) {
            ImageDesc &d = descs[i];
            if (d.src_addr == 0) continue;
            // Gathered payloads keep their source alignment mod 16 so that both sides move in whole
            // 16-byte words.  A crop box is fetched row by row: every row gets a 16-byte aligned slot
            // wide enough for the aligned words that contain it, and its pixels start inside the slot
            // at the row's own source alignment (ImageDesc::raw_skew tells the reader).
            const bool rowwise = d.mode == FFCVB_MODE_RAW && d.cols != d.width;
            if (rowwise) {
                d.raw_pitch = (uint32_t)align_up((size_t)d.cols * 3 + 15, 16);
                d.payload_size = (uint32_t)((size_t)d.rows * d.raw_pitch);
                d.raw_skew = 1;
                d.payload_off = off;
            } else {
                d.payload_off = off + (d.src_addr & 15);
            }
            off = align_up(d.payload_off + d.payload_size, kPayloadAlign);
        }
    }
    hd.total_bytes = off;

    int rc;
    // A pinned source needs room for the part that is staged.  That part varies from batch to batch and
    // regrowing page-locked memory stalls the device: room for the most that the split may stage.
    size_t host_need = off;
    if (s.range_len) {
        host_need = s.staged_end;
    } else if (direct) {
        const double most = ctx->adaptive_split ? kMaxAdaptiveShare : ctx->cpu_share_permille / 1000.0;
        host_need = hd.payload_off + (size_t)(most * (double)(off - hd.payload_off));
        if (host_need < s.staged_end) host_need = s.staged_end;
    }
    if (from_fd) // (the payloads lie in the buffer already)
        rc = grow_host_keeping(ctx, s.host, s.host_cap, host_need + 64, fd_payload_end);
    else
        rc = grow_host(ctx, s.host, s.host_cap, host_need + 64);
    if (rc) return rc;
    if ((rc = grow_needed(ctx, s.blob, off + 64))) return rc;
    if ((rc = grow_needed(ctx, s.clean, clean_bytes + 512))) return rc;
    if ((rc = grow_needed(ctx, s.segs, seg_total * kSegScratch + 64))) return rc;
    if (!s.slot_segs.empty() && (rc = grow_needed(ctx, s.slot_tables, s.slot_segs.size() * sizeof(SlotTables)))) return rc;
    if ((rc = grow_needed(ctx, s.index, (size_t)total_blocks * 6 + 64))) return rc;
    if ((rc = grow_needed(ctx, s.planes, plane_bytes + 64))) return rc;
    if ((rc = grow_needed(ctx, s.rgb, rgb_bytes + 64))) return rc;
    s.keep_records = grow_records(ctx, s, (size_t)records * 4 * sizeof(uint16_t)); // (last: the batch can do without)

    memcpy(s.host, &hd, sizeof(hd));
    // (past the caches: the lines were last read by a transfer, and the next one finds them in memory)
    auto place = [&](uint64_t off, const void *src, size_t bytes) { stream_copy(s.host + off, static_cast<const uint8_t *>(src), bytes); };
    place(hd.desc_off, descs.data(), sizeof(ImageDesc) * (size_t)n);
    for (size_t k = 0; k < huff_src.size(); k++)
        memcpy(s.host + hd.huff_off + k * sizeof(HuffTable), &ctx->tables.built(huff_src[k]), sizeof(HuffTable));
    for (size_t k = 0; k < mult_src.size(); k++)
        build_mult_table(ctx->tables.quant(mult_src[k]), reinterpret_cast<MultTable *>(s.host + hd.mult_off) + k);
    place(hd.params_off, params, sizeof(int32_t) * (size_t)n * n_params);
    {
        int32_t *st = reinterpret_cast<int32_t *>(s.host + s.status_off);
        for (int i = 0; i < n; i++) {
            st[i] = descs[i].mode == FFCVB_MODE_JPG ? descs[i].host_status : 0;
            st[n + i] = 0;
        }
    }
    for (int i = 0; i < n; i++) {
        // a sample decoded at reduced scale: its crop box, for the kernels, is the box of the scaled
        // image that covers it
        if (descs[i].scale_shift == 0 || !plan->resize) continue;
        scaled_box(descs[i], reinterpret_cast<int32_t *>(s.host + hd.params_off) + (size_t)i * n_params);
    }
    if (!s.items.empty()) place(s.items_off, s.items.data(), sizeof(ResizeItem) * s.items.size());
    s.bands = items.bands();
    s.plain = items.plain();
    for (const auto &r : s.riders) {
        if (!r.inline_bytes.empty()) {
            memcpy(s.host + r.off, r.inline_bytes.data(), r.bytes);
        } else {
            for (int i = 0; i < n; i++) {
                uint8_t *dst = s.host + r.off + (size_t)i * r.item_bytes;
                if (!from_fd) {
                    memcpy(dst, file_base + r.ptrs[i], r.item_bytes);
                } else { // small items: buffered reads
                    size_t done = 0;
                    while (done < r.item_bytes) {
                        const ssize_t got = pread(source.fd, dst + done, r.item_bytes - done, (off_t)(r.ptrs[i] + done));
                        if (got < 0 && errno == EINTR) continue;
                        if (got <= 0) {
                            memset(dst + done, 0, r.item_bytes - done);
                            break;
                        }
                        done += (size_t)got;
                    }
                }
            }
        }
    }
    if (!jpeg_list.empty()) memcpy(s.host + s.jpeg_list_off, jpeg_list.data(), 4 * jpeg_list.size());
    if (!s.parts.empty()) place(s.parts_off, s.parts.data(), sizeof(uint4) * s.parts.size());
    if (!s.wholes.empty()) memcpy(s.host + s.parts_off + sizeof(uint4) * s.parts.size(), s.wholes.data(), sizeof(uint4) * s.wholes.size());
    if (!slot_images.empty()) memcpy(s.host + s.slot_images_off, slot_images.data(), 4 * slot_images.size());
    if (!restart.empty()) memcpy(s.host + s.restart_off, restart.data(), 4 * restart.size());
    if (!segs.empty()) place(s.segs_off, segs.data(), sizeof(uint2) * segs.size());
    if (!s.slot_segs.empty()) memcpy(s.host + s.segs_off + sizeof(uint2) * segs.size(), s.slot_segs.data(), sizeof(uint2) * s.slot_segs.size());
    if (!blk_tiles.empty()) place(s.block_tiles_off, blk_tiles.data(), sizeof(uint2) * blk_tiles.size());
    if (!quad_tiles.empty()) place(s.quad_tiles_off, quad_tiles.data(), sizeof(uint2) * quad_tiles.size());
    if (s.gather_ctas) gather_ranges(descs.data(), n, s.gather_ctas, reinterpret_cast<uint2 *>(s.host + s.gather_off));
    s.n_quad_tiles = (int)quad_tiles.size();
    s.n_block_tiles = (int)blk_tiles.size();
    work.n_guess = (int)segs.size();
    work.n_slots = (int)s.slot_segs.size();
    work.n_parts = (int)s.parts.size();
    work.n_whole = (int)s.wholes.size();
    work.n_slot_images = (int)slot_images.size();
    work.n_restart = (int)restart.size();
    _mm_sfence();

    const auto t2 = std::chrono::steady_clock::now();
    // ---- parallel: gather the payload bytes into pinned memory
    uint8_t *host = s.host;
    if (!from_fd && s.staged_end > hd.payload_off) {
        Slot *sp = &s; // the job may outlive this call: it only touches slot-owned data and the source
        ctx->pool->wait(Pool::kAsync); // one copy at a time: the batch staged before this one
        int copy_threads = direct ? ctx->split_copy_threads : 0;
        if (ctx->tune_copy_threads) copy_threads = ctx->tune_copy_threads;
        {
            std::lock_guard<std::mutex> g(ctx->copy_m);
            s.copy_done = false;
        }
        // a few large streams are shared out in pieces
        const size_t piece = n < 4 * ctx->pool->size() ? 128 * 1024 : ~(size_t)0;
        sp->copies.clear();
        for (int i = 0; i < n; i++) {
            const ImageDesc &d = descs[i];
            if (d.payload_size == 0 || d.src_addr != 0) continue;
            const bool rows = d.mode == FFCVB_MODE_RAW && d.cols != d.width;
            const size_t step = rows ? d.payload_size : (piece < d.payload_size ? piece : d.payload_size);
            for (size_t from = 0; from < d.payload_size; from += step)
                sp->copies.push_back(Slot::Copy{i, from, d.payload_size - from < step ? d.payload_size - from : step});
        }
        ctx->pool->post(
            Pool::kAsync, (int)sp->copies.size(), 1,
            [sp, host, file_base](int k) {
                const Slot::Copy &c = sp->copies[k];
                const ImageDesc &d = sp->descs[c.sample];
                const uint8_t *src = file_base + sp->src_ptrs[c.sample];
                uint8_t *dst = host + d.payload_off;
                if (d.mode == FFCVB_MODE_RAW && d.cols != d.width) {
                    // only the crop box travels: one run per row.  Plain copies: streaming stores on
                    // ~1 KB rows leave partial write-combining lines and measured almost twice slower
                    const size_t pitch = (size_t)d.width * 3, run = (size_t)d.cols * 3;
                    src += (size_t)d.row0 * pitch + (size_t)d.col0 * 3;
                    for (int r = 0; r < d.rows; r++) memcpy(dst + r * (size_t)d.raw_pitch, src + r * pitch, run);
                } else {
                    if (d.mode == FFCVB_MODE_RAW) src += (size_t)d.row0 * d.width * 3;
                    stream_copy(dst + c.from, src + c.from, c.bytes);
                }
                _mm_sfence(); // streaming stores are weakly ordered: publish them before the copy is reported done
            },
            [ctx, sp, t2] {
                std::lock_guard<std::mutex> g(ctx->copy_m);
                sp->stage_ms[2] = std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t2).count();
                sp->copy_done = true;
                ctx->copy_cv.notify_all();
            },
            copy_threads);
        if (!ctx->async_staging) ctx->pool->wait(Pool::kAsync);
    }
    const auto t3 = std::chrono::steady_clock::now();
    auto ms = [](auto a, auto b) { return std::chrono::duration<double, std::milli>(b - a).count(); };
    s.stage_ms[0] = ms(t0, t1);
    s.stage_ms[1] = ms(t1, t2);
    if (from_fd || s.staged_end <= hd.payload_off) s.stage_ms[2] = 0; // else: written when the copy completes
    s.stage_ms[3] = ms(t0, t3);
    s.n_jpeg = (int)jpeg_list.size();
    s.total_blocks = total_blocks;
    s.max_w = max_w;
    s.max_h = max_h;
    s.n_quad = n_quad;
    s.n_444 = n_444;
    s.n_other = n_other;
    s.clean_bytes = clean_bytes;
    s.plane_bytes = plane_bytes;
    s.rgb_bytes = rgb_bytes;
    s.scan_bytes = s.raw_bytes = s.jpeg_bytes = 0;
    for (int i = 0; i < n; i++) {
        if (descs[i].mode == FFCVB_MODE_JPG) {
            s.jpeg_bytes += descs[i].payload_size;
            if (descs[i].host_status == 0) s.scan_bytes += descs[i].scan_len;
        } else {
            s.raw_bytes += descs[i].payload_size;
        }
    }
    s.staged = true;
    return FFCVB_OK;
}

} // namespace

extern "C" {

int ffcvb_stage_batch(ffcvb_ctx *ctx, int slot, const uint8_t *file_base, const uint64_t *ptrs,
                      const uint64_t *sizes, const uint8_t *modes, const uint16_t *heights,
                      const uint16_t *widths, int n, const ffcvb_plan *plan, const int32_t *params) {
    if (ctx && !file_base) return fail(ctx, FFCVB_E_ARG, "ffcvb_stage_batch: bad argument");
    Source src;
    src.base = file_base;
    return stage_impl(ctx, slot, src, ptrs, sizes, modes, heights, widths, n, plan, params);
}

int ffcvb_stage_batch_fd(ffcvb_ctx *ctx, int slot, int fd, int fd_direct, const uint64_t *ptrs,
                         const uint64_t *sizes, const uint8_t *modes, const uint16_t *heights,
                         const uint16_t *widths, int n, const ffcvb_plan *plan, const int32_t *params) {
    if (ctx && fd < 0) return fail(ctx, FFCVB_E_ARG, "ffcvb_stage_batch_fd: bad file descriptor");
    Source src;
    src.fd = fd;
    src.fd_direct = fd_direct;
    struct statfs fs; // (TMPFS_MAGIC, RAMFS_MAGIC, HUGETLBFS_MAGIC)
    src.in_memory = fstatfs(fd, &fs) == 0 && ((uint64_t)fs.f_type == 0x01021994u || (uint64_t)fs.f_type == 0x858458f6u || (uint64_t)fs.f_type == 0x958458f6u);
    return stage_impl(ctx, slot, src, ptrs, sizes, modes, heights, widths, n, plan, params);
}

// Stream callback: holds the stream until the staging threads have finished the slot's payload
// copy, so that a batch can be queued while its bytes are still being staged.  Makes no CUDA call.
// The wait is bounded; running out of time is recorded and reported by the next call.
static void CUDART_CB wait_for_copy(void *arg) {
    WaitArg *w = static_cast<WaitArg *>(arg);
    ffcvb_ctx *c = w->ctx;
    std::unique_lock<std::mutex> g(c->copy_m);
    if (!c->copy_cv.wait_for(g, std::chrono::seconds(120), [&] { return c->slots[w->slot].copy_done; }))
        c->copy_timeout.store(true);
}

static int hold_for_copy(ffcvb_ctx *ctx, Slot &s, cudaStream_t st) {
    bool done;
    {
        std::lock_guard<std::mutex> g(ctx->copy_m);
        done = s.copy_done;
    }
    if (!done) CU(cudaLaunchHostFunc(st, wait_for_copy, &ctx->wait_args[&s - ctx->slots.data()]));
    return FFCVB_OK;
}

// An error, once, when a gather of an earlier batch has given up since the last call.
static int report_gather(ffcvb_ctx *ctx) {
    volatile int32_t *failed = ctx->gather_failed;
    if (!failed || !*failed) return FFCVB_OK;
    *failed = 0;
    return fail(ctx, FFCVB_E_CUDA, "the payloads of an earlier batch did not arrive in time: ffcvb_batch_status flags its samples");
}

// Where a single-image decode leaves its pixels (instead of the slot's scratch, and with no resize
// behind it) and its status word: device or page-locked host memory.
struct Single {
    uint8_t *rgb;
    int32_t *status;
    bool whole_rows; // see launch_color
};

// `outputs_free`: an event the work that writes to the caller's buffers (out_dev, the riders'
// destinations) has to wait for; all before it only touches memory of the slot.
static int run_batch(ffcvb_ctx *ctx, Slot &s, cudaStream_t st, void *out_dev, bool copy, const Single *single = nullptr,
                     cudaEvent_t outputs_free = nullptr) {
    if (ctx->copy_timeout.load())
        return fail(ctx, FFCVB_E_CUDA, "a payload copy did not finish within its time limit: the batch that waited for it is invalid");
    int hrc;
    if (single && ctx->gather_failed)
        *ctx->gather_failed = 0; // (its call has returned the image's status)
    else if ((hrc = report_gather(ctx)))
        return hrc;
    const int slot = (int)(&s - ctx->slots.data());
    const bool indexed = ctx->index_pool.p && s.index_life == ctx->index_life;
    const BatchHeader &hd = s.hdr;
    uint8_t *blob = (uint8_t *)s.blob.p;
    const bool prof = ctx->profile;
    s.timed = false;
    if (prof) {
        for (auto &e : s.ev)
            if (!e) CU(cudaEventCreate(&e));
        CU(cudaEventRecord(s.ev[0], st));
    }
    if (!s.ev_copied) {
        CU(cudaEventCreateWithFlags(&s.ev_copied, cudaEventDisableTiming));
        CU(cudaEventCreateWithFlags(&s.ev_done, cudaEventDisableTiming));
    }
    if (s.last_stream != st && s.last_stream != nullptr) CU(cudaStreamWaitEvent(st, s.ev_done, 0)); // (the slot changed streams)
    s.last_stream = st;
    if (copy && !s.direct) {
        if ((hrc = hold_for_copy(ctx, s, st))) return hrc;
        CU(cudaMemcpyAsync(blob, s.host, hd.total_bytes, cudaMemcpyHostToDevice, st));
    } else if (copy) {
        if (!ctx->copy_stream) {
            CU(cudaHostAlloc((void **)&ctx->gather_failed, 64, cudaHostAllocDefault));
            *ctx->gather_failed = 0;
            int lo = 0, hi = 0;
            CU(cudaDeviceGetStreamPriorityRange(&lo, &hi));
            CU(cudaStreamCreateWithPriority(&ctx->copy_stream, cudaStreamNonBlocking, hi));
        }
        if (!s.ev_begin) {
            CU(cudaEventCreateWithFlags(&s.ev_begin, cudaEventDisableTiming));
            CU(cudaEventCreate(&s.ev_gather_start));
            CU(cudaEventCreate(&s.ev_gathered));
        }
        CU(cudaEventRecord(s.ev_begin, st)); // the slot's previous batch
        CU(cudaStreamWaitEvent(ctx->copy_stream, s.ev_begin, 0));
        CU(cudaMemcpyAsync(blob, s.host, hd.payload_off, cudaMemcpyHostToDevice, ctx->copy_stream));
        s.gather_timed = s.range_len == 0;
        if (s.gather_timed) {
            CU(cudaEventRecord(s.ev_gather_start, ctx->copy_stream));
            launch_gather_payloads(reinterpret_cast<ImageDesc *>(blob + hd.desc_off), reinterpret_cast<const uint2 *>(blob + s.gather_off), s.gather_ctas, blob,
                                   reinterpret_cast<int32_t *>(blob + s.status_off), ctx->gather_limit_ns, ctx->gather_failed, ctx->copy_stream);
        } else {
            CU(cudaMemcpyAsync(blob + hd.payload_off, s.range_src, s.range_len, cudaMemcpyHostToDevice, ctx->copy_stream));
        }
        CU(cudaEventRecord(s.ev_gathered, ctx->copy_stream));
        if (s.range_len == 0 && s.staged_end > hd.payload_off) { // the CPU-staged share rides the copy engine meanwhile
            if ((hrc = hold_for_copy(ctx, s, st))) return hrc;
            CU(cudaMemcpyAsync(blob + hd.payload_off, s.host + hd.payload_off, s.staged_end - hd.payload_off,
                               cudaMemcpyHostToDevice, st));
        }
        CU(cudaStreamWaitEvent(st, s.ev_gathered, 0));
    }
    if (copy) {
        CU(cudaEventRecord(s.ev_copied, st));
        s.in_flight = true;
        if (indexed) ctx->index.submitted(slot);
    }
    if (prof) CU(cudaEventRecord(s.ev[1], st));
    const ImageDesc *descs = reinterpret_cast<const ImageDesc *>(blob + hd.desc_off);
    const HuffTable *huff = reinterpret_cast<const HuffTable *>(blob + hd.huff_off);
    const MultTable *mult = reinterpret_cast<const MultTable *>(blob + hd.mult_off);
    const int32_t *params = reinterpret_cast<const int32_t *>(blob + hd.params_off);
    int32_t *status = single ? single->status : reinterpret_cast<int32_t *>(blob + s.status_off);
    uint8_t *rgb = single ? single->rgb : (uint8_t *)s.rgb.p;
    bool early = false;
    if (s.n_jpeg > 0) {
        const int32_t *jl = reinterpret_cast<const int32_t *>(blob + s.jpeg_list_off);
        EntropyScratch scratch{};
        scratch.clean = (uint8_t *)s.clean.p;
        EntropyWork work = s.work;
        work.segs = reinterpret_cast<const uint2 *>(blob + s.segs_off);
        work.parts = reinterpret_cast<const uint4 *>(blob + s.parts_off);
        work.slot_images = reinterpret_cast<const int32_t *>(blob + s.slot_images_off);
        work.restart = reinterpret_cast<const int32_t *>(blob + s.restart_off);
        const size_t n_segs = (size_t)work.n_guess + work.n_slots;
        scratch.seg_dc = (int32_t *)s.segs.p;
        scratch.sub_info = (uint32_t *)(scratch.seg_dc + 4 * n_segs);
        scratch.sub_exit = (uint16_t *)(scratch.sub_info + kSegSubs * n_segs);
        scratch.meta = (SegMeta *)(scratch.sub_exit + kSegSubs * n_segs); // (everything before it is a multiple of 16 bytes)
        scratch.slots = (SlotTables *)s.slot_tables.p;
        scratch.records = s.keep_records ? (uint16_t *)s.records.p : nullptr;
        scratch.done = (uint32_t *)(blob + s.status_off) + s.n;
        scratch.pos = (uint32_t *)s.index.p;
        scratch.dc = (int16_t *)(scratch.pos + s.total_blocks);
        early = work.early() && !prof;
        launch_entropy_decode(descs, work, blob, huff, scratch, status, indexed ? (uint8_t *)ctx->index_pool.p : nullptr,
                              (unsigned long long *)ctx->index_stats.p, st);
        if (prof) CU(cudaEventRecord(s.ev[2], st));
        launch_blocks(descs, reinterpret_cast<const uint2 *>(blob + s.block_tiles_off), s.n_block_tiles, huff, mult, scratch,
                      (uint8_t *)s.planes.p, early, st);
        if (prof) CU(cudaEventRecord(s.ev[3], st));
        launch_color(descs, jl, s.n_jpeg, s.n_quad, s.n_444, s.n_other, s.max_w, s.max_h,
                     reinterpret_cast<const uint2 *>(blob + s.quad_tiles_off), s.n_quad_tiles, (const uint8_t *)s.planes.p,
                     rgb, s.plan.resize ? params : nullptr, (int)hd.n_params, single && single->whole_rows, early, st);
        if (prof) CU(cudaEventRecord(s.ev[4], st));
    } else if (prof) {
        for (int k = 2; k <= 4; k++) CU(cudaEventRecord(s.ev[k], st));
    }
    if (outputs_free) CU(cudaStreamWaitEvent(st, outputs_free, 0));
    if (!single) {
        static_assert(FFCVB_MAX_RIDERS <= sizeof(SmallCopies::src) / sizeof(uint8_t *), "a batch's riders fit one launch");
        SmallCopies small{};
        const Slot::Rider *large[FFCVB_MAX_RIDERS];
        int n_large = 0;
        uint64_t words = 0;
        for (const auto &r : s.riders) {
            if (!copy) break;
            const uint64_t mine = small_copy_words(r.bytes, blob + r.off, r.dst_dev);
            if (words + mine > kSmallCopyWords) {
                large[n_large++] = &r;
                continue;
            }
            words += mine;
            small.src[small.n] = blob + r.off;
            small.bytes[small.n] = r.bytes;
            small.dst[small.n++] = (uint8_t *)r.dst_dev;
        }
        ResizeSource src{};
        src.descs = descs;
        src.blob = blob;
        src.rgb = rgb;
        src.planes = (const uint8_t *)s.planes.p;
        launch_resize_augment(src, s.n, params, (int)hd.n_params, reinterpret_cast<const ResizeItem *>(blob + s.items_off), make_oplist(s.plan), s.plan.resize,
                              s.plan.out_h, s.plan.out_w, s.plan.out_kind, s.bands, s.plain, s.plan.lut_dev, out_dev, status, small,
                              early && !outputs_free, st);
        for (int k = 0; k < n_large; k++) // (behind the kernel, which may have been launched early)
            CU(cudaMemcpyAsync(large[k]->dst_dev, blob + large[k]->off, large[k]->bytes, cudaMemcpyDeviceToDevice, st));
    }
    CU(cudaGetLastError());
    if (prof) {
        CU(cudaEventRecord(s.ev[5], st));
        s.timed = true;
    }
    CU(cudaEventRecord(s.ev_done, st));
    if (indexed) ctx->index.marked(slot);
    return FFCVB_OK;
}

int ffcvb_set_batch_riders(ffcvb_ctx *ctx, int slot, const ffcvb_rider *riders, int n_riders, int n) {
    if (!ctx) return FFCVB_E_ARG;
    if (slot < 0 || slot >= (int)ctx->slots.size() || n_riders < 0 || n_riders > FFCVB_MAX_RIDERS || n <= 0 ||
        (n_riders > 0 && !riders))
        return fail(ctx, FFCVB_E_ARG, "ffcvb_set_batch_riders: bad argument");
    Slot &s = ctx->slots[slot];
    s.pending_riders.clear();
    for (int k = 0; k < n_riders; k++) {
        const ffcvb_rider &in = riders[k];
        if (!in.dst_dev || in.item_bytes == 0 || in.item_bytes > (1u << 24) || (!in.host == !in.ptrs)) {
            s.pending_riders.clear();
            return fail(ctx, FFCVB_E_ARG, "ffcvb_set_batch_riders: rider %d needs a destination, an item size and "
                                          "exactly one of host / ptrs", k);
        }
        Slot::Rider r;
        r.item_bytes = in.item_bytes;
        r.dst_dev = in.dst_dev;
        if (in.host) {
            const uint8_t *b = static_cast<const uint8_t *>(in.host);
            r.inline_bytes.assign(b, b + (size_t)n * in.item_bytes);
        } else {
            r.ptrs.assign(in.ptrs, in.ptrs + n);
        }
        s.pending_riders.push_back(std::move(r));
    }
    return FFCVB_OK;
}

int ffcvb_set_header_cache(ffcvb_ctx *ctx, int enabled) {
    if (!ctx) return FFCVB_E_ARG;
    ctx->pool->wait_all();
    ctx->cache_headers = enabled != 0;
    ctx->header_cache.clear();
    return FFCVB_OK;
}

int ffcvb_set_decode_index(ffcvb_ctx *ctx, uint64_t bytes) {
    if (!ctx) return FFCVB_E_ARG;
    ctx->pool->wait_all();
    CU(cudaSetDevice(ctx->device));
    CU(cudaDeviceSynchronize());
    if (ctx->index_pool.p) {
        CU(cudaFree(ctx->index_pool.p));
        ctx->index_pool = DevBuf{};
    }
    ctx->index.reset(0, (int)ctx->slots.size());
    ctx->index_life++;
    if (bytes == 0) return FFCVB_OK;
    bytes = align_up((size_t)bytes, 1 << 20);
    CU(cudaMalloc(&ctx->index_pool.p, (size_t)bytes));
    ctx->index_pool.cap = (size_t)bytes;
    ctx->index.reset((size_t)bytes, (int)ctx->slots.size());
    CU(cudaMemset(ctx->index_pool.p, 0, (size_t)bytes)); // no entry is valid yet
    if (!ctx->index_stats.p) {
        CU(cudaMalloc(&ctx->index_stats.p, 64));
        ctx->index_stats.cap = 64;
    }
    CU(cudaMemset(ctx->index_stats.p, 0, 64));
    return FFCVB_OK;
}

int ffcvb_decode_index_stats(ffcvb_ctx *ctx, uint64_t *out) {
    if (!ctx || !out) return FFCVB_E_ARG;
    out[0] = out[1] = 0;
    out[2] = ctx->index.entries();
    out[3] = ctx->index.used();
    if (!ctx->index_stats.p) return FFCVB_OK;
    CU(cudaSetDevice(ctx->device));
    CU(cudaMemcpy(out, ctx->index_stats.p, 16, cudaMemcpyDeviceToHost));
    return FFCVB_OK;
}

int ffcvb_set_async_staging(ffcvb_ctx *ctx, int enabled) {
    if (!ctx) return FFCVB_E_ARG;
    ctx->pool->wait_all();
    ctx->async_staging = enabled != 0;
    return FFCVB_OK;
}

int ffcvb_set_staging_split(ffcvb_ctx *ctx, int cpu_share_permille) {
    if (!ctx) return FFCVB_E_ARG;
    if (cpu_share_permille < -1 || cpu_share_permille > 1000)
        return fail(ctx, FFCVB_E_ARG, "ffcvb_set_staging_split: share must be 0..1000, or -1");
    ctx->adaptive_split = cpu_share_permille < 0;
    ctx->share = ctx->adaptive_split ? 0.3 : cpu_share_permille / 1000.0;
    ctx->cpu_share_permille = (int)(ctx->share * 1000 + 0.5);
    return FFCVB_OK;
}

int ffcvb_staging_split(const ffcvb_ctx *ctx) { return ctx ? ctx->cpu_share_permille : -1; }

int ffcvb_set_profiling(ffcvb_ctx *ctx, int enabled) {
    if (!ctx) return FFCVB_E_ARG;
    ctx->profile = enabled != 0;
    return FFCVB_OK;
}

int ffcvb_batch_times(ffcvb_ctx *ctx, int slot, float *ms) {
    if (!ctx) return FFCVB_E_ARG;
    if (slot < 0 || slot >= (int)ctx->slots.size() || !ms)
        return fail(ctx, FFCVB_E_ARG, "ffcvb_batch_times: bad argument");
    Slot &s = ctx->slots[slot];
    if (!s.timed) return fail(ctx, FFCVB_E_ARG, "ffcvb_batch_times: slot %d was not run with profiling on", slot);
    CU(cudaSetDevice(ctx->device));
    CU(cudaEventSynchronize(s.ev[5]));
    for (int k = 0; k < 5; k++) CU(cudaEventElapsedTime(&ms[k], s.ev[k], s.ev[k + 1]));
    return FFCVB_OK;
}

int ffcvb_submit_batch(ffcvb_ctx *ctx, int slot, void *stream, void *out_dev) {
    return ffcvb_submit_batch_after(ctx, slot, stream, out_dev, nullptr);
}

int ffcvb_submit_batch_after(ffcvb_ctx *ctx, int slot, void *stream, void *out_dev, void *outputs_free) {
    if (!ctx) return FFCVB_E_ARG;
    if (slot < 0 || slot >= (int)ctx->slots.size() || !out_dev)
        return fail(ctx, FFCVB_E_ARG, "ffcvb_submit_batch: bad argument");
    Slot &s = ctx->slots[slot];
    if (!s.staged) return fail(ctx, FFCVB_E_ARG, "ffcvb_submit_batch: slot %d has no staged batch", slot);
    CU(cudaSetDevice(ctx->device));
    return run_batch(ctx, s, (cudaStream_t)stream, out_dev, true, nullptr, (cudaEvent_t)outputs_free);
}

/* Re-runs the kernels of a batch whose bytes a previous ffcvb_submit_batch already put in HBM
 * (no host->device copy).  For measuring the device-resident rate. */
int ffcvb_rerun_batch(ffcvb_ctx *ctx, int slot, void *stream, void *out_dev) {
    if (!ctx) return FFCVB_E_ARG;
    if (slot < 0 || slot >= (int)ctx->slots.size() || !out_dev)
        return fail(ctx, FFCVB_E_ARG, "ffcvb_rerun_batch: bad argument");
    Slot &s = ctx->slots[slot];
    if (!s.staged) return fail(ctx, FFCVB_E_ARG, "ffcvb_rerun_batch: slot %d has no staged batch", slot);
    CU(cudaSetDevice(ctx->device));
    return run_batch(ctx, s, (cudaStream_t)stream, out_dev, false);
}

int64_t ffcvb_staged_bytes(const ffcvb_ctx *ctx, int slot) {
    if (!ctx || slot < 0 || slot >= (int)ctx->slots.size() || !ctx->slots[slot].staged) return -1;
    return (int64_t)ctx->slots[slot].hdr.total_bytes;
}

int ffcvb_stage_times(const ffcvb_ctx *ctx, int slot, double *ms) {
    // (no `staged` check: the figures of the slot's last completed staging stay readable while
    // another thread stages the slot again)
    if (!ctx || !ms || slot < 0 || slot >= (int)ctx->slots.size()) return FFCVB_E_ARG;
    for (int k = 0; k < 4; k++) ms[k] = ctx->slots[slot].stage_ms[k];
    return FFCVB_OK;
}

int ffcvb_gather_time(ffcvb_ctx *ctx, int slot, float *ms) {
    if (!ctx) return FFCVB_E_ARG;
    if (!ms || slot < 0 || slot >= (int)ctx->slots.size()) return fail(ctx, FFCVB_E_ARG, "ffcvb_gather_time: bad argument");
    Slot &s = ctx->slots[slot];
    *ms = -1.0f;
    if (!s.gather_timed) return FFCVB_OK; // this slot's last batch was not gathered by the GPU
    CU(cudaSetDevice(ctx->device));
    // (a loader's worker may submit the slot's next batch between the wait and the reading: wait for that one then)
    cudaError_t e = cudaErrorNotReady;
    for (int k = 0; k < 100 && e == cudaErrorNotReady; k++) {
        CU(cudaEventSynchronize(s.ev_gathered));
        e = cudaEventElapsedTime(ms, s.ev_gather_start, s.ev_gathered);
    }
    if (e == cudaErrorNotReady) cudaGetLastError();
    CU(e);
    return FFCVB_OK;
}

int ffcvb_batch_info(const ffcvb_ctx *ctx, int slot, int64_t *info) {
    if (!ctx || !info || slot < 0 || slot >= (int)ctx->slots.size() || !ctx->slots[slot].staged) return FFCVB_E_ARG;
    const Slot &s = ctx->slots[slot];
    info[0] = s.n;
    info[1] = s.n_jpeg;
    info[2] = s.total_blocks;
    info[3] = (int64_t)s.scan_bytes;
    info[4] = (int64_t)s.plane_bytes;
    info[5] = (int64_t)s.rgb_bytes;
    info[6] = (int64_t)s.raw_bytes;
    info[7] = (int64_t)s.jpeg_bytes;
    return FFCVB_OK;
}

int ffcvb_batch_launches(const ffcvb_ctx *ctx, int slot) {
    if (!ctx || slot < 0 || slot >= (int)ctx->slots.size() || !ctx->slots[slot].staged) return -1;
    const Slot &s = ctx->slots[slot];
    int k = 1 + (s.direct && s.range_len == 0 ? 1 : 0); // fused resize/augment/normalise (+ payload gather)
    k += (s.n_quad > 0) + (s.n_444 > 0) + (s.n_other > 0) + (s.n_block_tiles > 0) + 2 * (s.work.n_guess > 0) + (s.work.n_whole > 0) +
         2 * (s.work.n_slots > 0) + (s.work.n_guess > 0) + (s.work.n_slots > 0) + (s.work.n_restart > 0);
    return k;
}

int ffcvb_check(ffcvb_ctx *ctx) { return ctx ? report_gather(ctx) : FFCVB_E_ARG; }

int ffcvb_batch_status(ffcvb_ctx *ctx, int slot, void *stream, int32_t *status, int n) {
    if (!ctx) return FFCVB_E_ARG;
    if (slot < 0 || slot >= (int)ctx->slots.size() || !status || n < 0)
        return fail(ctx, FFCVB_E_ARG, "ffcvb_batch_status: bad argument");
    Slot &s = ctx->slots[slot];
    if (!s.staged || n > s.n) return fail(ctx, FFCVB_E_ARG, "ffcvb_batch_status: nothing staged");
    CU(cudaSetDevice(ctx->device));
    CU(cudaMemcpyAsync(status, (const uint8_t *)s.blob.p + s.status_off, sizeof(int32_t) * (size_t)n, cudaMemcpyDeviceToHost,
                       (cudaStream_t)stream));
    CU(cudaStreamSynchronize((cudaStream_t)stream));
    int bad = 0;
    for (int i = 0; i < n; i++) {
        if (status[i] != 0) {
            status[i] = FFCVB_E_DECODE;
            bad++;
        }
    }
    return bad;
}

} // extern "C"

// Small per-call parameter arrays travel through a ring of sixteen pinned/device buffer pairs: copies
// the `bytes` that `fill` writes to the next pair's device side on `st`.  The caller holds aux_m and records
// a->ev on `st` once its kernels are queued.
template <class Fill>
static int stage_aux(ffcvb_ctx *ctx, cudaStream_t st, size_t bytes, Fill &&fill, AuxBuf **out) {
    AuxBuf &a = ctx->aux[ctx->aux_next];
    ctx->aux_next = (ctx->aux_next + 1) % 16;
    if (!a.ev) CU(cudaEventCreateWithFlags(&a.ev, cudaEventDisableTiming));
    if (a.used) CU(cudaEventSynchronize(a.ev));
    int rc;
    if ((rc = grow_dev(ctx, a.dev, bytes))) return rc;
    if ((rc = grow_host(ctx, a.host, a.host_cap, bytes))) return rc;
    fill(a.host);
    CU(cudaMemcpyAsync(a.dev.p, a.host, bytes, cudaMemcpyHostToDevice, st));
    *out = &a;
    return FFCVB_OK;
}

extern "C" {

int ffcvb_transform_device(ffcvb_ctx *ctx, void *stream, const uint8_t *src_dev, int n, int h, int w,
                           const ffcvb_plan *plan, const int32_t *params, void *out_dev) {
    if (!ctx) return FFCVB_E_ARG;
    if (!src_dev || n <= 0 || h <= 0 || w <= 0 || !params || !out_dev || !valid_plan(plan))
        return fail(ctx, FFCVB_E_ARG, "ffcvb_transform_device: bad argument");
    CU(cudaSetDevice(ctx->device));
    cudaStream_t st = (cudaStream_t)stream;
    const int n_params = 4 + 2 * plan->n_ops;
    const size_t items_off = plan->resize ? sizeof(ResizeItem) * (size_t)n : 0, bytes = items_off + sizeof(int32_t) * (size_t)n * n_params; // (the items lie first)
    ResizeItems items(n, plan->out_h, plan->out_w, plan->out_kind);
    std::lock_guard<std::mutex> guard(ctx->aux_m);
    AuxBuf *ap;
    int rc;
    if ((rc = stage_aux(ctx, st, bytes, [&](uint8_t *host) {
             for (int i = 0; i < n && plan->resize; i++)
                 reinterpret_cast<ResizeItem *>(host)[i] = items.make(params + (size_t)i * n_params, h, w, ResizeItems::kPacked);
             memcpy(host + items_off, params, bytes - items_off);
         }, &ap)))
        return rc;
    AuxBuf &a = *ap;
    ResizeSource src{};
    src.uniform = src_dev;
    src.uniform_h = h;
    src.uniform_w = w;
    launch_resize_augment(src, n, (const int32_t *)((const uint8_t *)a.dev.p + items_off), n_params, (const ResizeItem *)a.dev.p, make_oplist(*plan), plan->resize,
                          plan->out_h, plan->out_w, plan->out_kind, items.bands(), items.plain(), plan->lut_dev, out_dev, nullptr, SmallCopies{}, false, st);
    CU(cudaGetLastError());
    CU(cudaEventRecord(a.ev, st));
    a.used = true;
    return FFCVB_OK;
}

// `values` per image; pixels unless it is no multiple of three (mixup alone)
static int pixel_chain(ffcvb_ctx *ctx, void *stream, const uint8_t *src_dev, int n, int64_t values, int n_ops, const int32_t *kinds,
                       const uint8_t *apply, const double *ratio, const double *lam, int out_size, const void *lut_dev, void *dst_dev) {
    const int64_t pixels = values / 3;
    const bool bytes_only = values % 3 != 0 && n_ops == 0 && lam && out_size == 1;
    if (!src_dev || !dst_dev || n <= 0 || values <= 0 || (values % 3 != 0 && !bytes_only) || pixels > (int64_t)1 << 30 || n_ops < 0 || n_ops > kMaxChainOps ||
        (n_ops > 0 && (!kinds || !apply || !ratio)) || (out_size != 1 && out_size != 2 && out_size != 4) || (out_size != 1 && !lut_dev) ||
        (lam && src_dev == dst_dev) || (out_size != 1 && src_dev == dst_dev))
        return fail(ctx, FFCVB_E_ARG, "ffcvb_pixel_chain: bad argument");
    PixelChain chain{};
    chain.n = n;
    chain.n_ops = n_ops;
    bool contrast = false;
    for (int k = 0; k < n_ops; k++) {
        if (kinds[k] < FFCVB_JITTER_BRIGHTNESS || kinds[k] > FFCVB_JITTER_SATURATION)
            return fail(ctx, FFCVB_E_ARG, "ffcvb_pixel_chain: unknown operation %d", kinds[k]);
        chain.kind[k] = kinds[k];
        contrast = contrast || kinds[k] == FFCVB_JITTER_CONTRAST;
    }
    for (int i = 0; lam && i < n; i++)
        if (!(lam[i] >= 0.0 && lam[i] <= 1.0)) return fail(ctx, FFCVB_E_ARG, "ffcvb_pixel_chain: lam[%d] outside [0, 1]", i);
    CU(cudaSetDevice(ctx->device));
    cudaStream_t st = (cudaStream_t)stream;
    // [ratio: doubles][lam: doubles][grey sums: zeroes, if there is a contrast][apply: bytes].  (A copy of up to one
    // kilobyte arrives 4 us sooner than a larger one.)
    const size_t entries = (size_t)n_ops * n, lam_off = sizeof(double) * entries, sums_off = lam_off + (lam ? sizeof(double) * (size_t)n : 0);
    const size_t sums = contrast ? sizeof(unsigned long long) * entries : 0, apply_off = sums_off + sums, bytes = apply_off + entries;
    uint8_t *dev = nullptr;
    std::lock_guard<std::mutex> guard(ctx->aux_m);
    AuxBuf *a = nullptr;
    if (bytes > 0) {
        int rc;
        if ((rc = stage_aux(ctx, st, bytes, [&](uint8_t *host) {
                 if (entries) memcpy(host, ratio, sizeof(double) * entries);
                 if (lam) memcpy(host + lam_off, lam, sizeof(double) * (size_t)n);
                 memset(host + sums_off, 0, sums);
                 if (entries) memcpy(host + apply_off, apply, entries);
             }, &a)))
            return rc;
        dev = (uint8_t *)a->dev.p;
        chain.ratio = (const double *)dev;
        chain.lam = lam ? (const double *)(dev + lam_off) : nullptr;
        chain.grey_sum = (unsigned long long *)(dev + sums_off);
        chain.apply = dev + apply_off;
    }
    if (bytes_only)
        launch_mixup_bytes(src_dev, (uint8_t *)dst_dev, (long long)values, chain, st);
    else
        launch_pixel_chain(src_dev, dst_dev, (int)pixels, chain, out_size, lut_dev, st);
    CU(cudaGetLastError());
    if (a) {
        CU(cudaEventRecord(a->ev, st));
        a->used = true;
    }
    return FFCVB_OK;
}

int ffcvb_pixel_chain(ffcvb_ctx *ctx, void *stream, const uint8_t *src_dev, int n, int64_t pixels, int n_ops, const int32_t *kinds,
                      const uint8_t *apply, const double *ratio, const double *lam, int out_size, const void *lut_dev, void *dst_dev) {
    if (!ctx) return FFCVB_E_ARG;
    return pixel_chain(ctx, stream, src_dev, n, 3 * pixels, n_ops, kinds, apply, ratio, lam, out_size, lut_dev, dst_dev);
}

int ffcvb_onehot_mix(ffcvb_ctx *ctx, void *stream, int n, int classes, const int32_t *label, const float *lam, float *dst_dev) {
    if (!ctx) return FFCVB_E_ARG;
    if (n <= 0 || classes <= 0 || !label || !lam || !dst_dev) return fail(ctx, FFCVB_E_ARG, "ffcvb_onehot_mix: bad argument");
    for (int i = 0; i < n; i++)
        if (label[i] < 0 || label[i] >= classes) return fail(ctx, FFCVB_E_ARG, "ffcvb_onehot_mix: label[%d] = %d with %d classes", i, label[i], classes);
    CU(cudaSetDevice(ctx->device));
    cudaStream_t st = (cudaStream_t)stream;
    std::lock_guard<std::mutex> guard(ctx->aux_m);
    AuxBuf *a;
    int rc;
    if ((rc = stage_aux(ctx, st, 8 * (size_t)n, [&](uint8_t *host) {
             memcpy(host, label, 4 * (size_t)n);
             memcpy(host + 4 * (size_t)n, lam, 4 * (size_t)n);
         }, &a)))
        return rc;
    launch_onehot_mix(dst_dev, n, classes, (const int32_t *)a->dev.p, (const float *)a->dev.p + n, st);
    CU(cudaGetLastError());
    CU(cudaEventRecord(a->ev, st));
    a->used = true;
    return FFCVB_OK;
}

int ffcvb_color_jitter(ffcvb_ctx *ctx, void *stream, uint8_t *images_dev, int n, int h, int w, int kind,
                       const uint8_t *apply, const double *ratio) {
    if (!ctx) return FFCVB_E_ARG;
    if (!images_dev || n <= 0 || h <= 0 || w <= 0 || kind < 0 || kind > 2 || !apply || !ratio ||
        (int64_t)h * w > (int64_t)1 << 30)
        return fail(ctx, FFCVB_E_ARG, "ffcvb_color_jitter: bad argument");
    const int32_t kinds[1] = {kind};
    return ffcvb_pixel_chain(ctx, stream, images_dev, n, (int64_t)h * w, 1, kinds, apply, ratio, nullptr, 1, nullptr, images_dev);
}

int ffcvb_mixup(ffcvb_ctx *ctx, void *stream, const uint8_t *src_dev, uint8_t *dst_dev, int n, int64_t count,
                const double *lam) {
    if (!ctx) return FFCVB_E_ARG;
    if (!src_dev || !dst_dev || src_dev == dst_dev || n <= 0 || count <= 0 || !lam)
        return fail(ctx, FFCVB_E_ARG, "ffcvb_mixup: bad argument");
    return pixel_chain(ctx, stream, src_dev, n, count, 0, nullptr, nullptr, nullptr, lam, 1, nullptr, dst_dev);
}

int ffcvb_poison(ffcvb_ctx *ctx, void *stream, uint8_t *images_dev, int n, int64_t count, const uint8_t *apply,
                 const double *one_minus_alpha_dev, const double *mask_dev, double clamp_lo, double clamp_hi) {
    if (!ctx) return FFCVB_E_ARG;
    if (!images_dev || n <= 0 || count <= 0 || !apply || !one_minus_alpha_dev || !mask_dev || !(clamp_lo <= clamp_hi))
        return fail(ctx, FFCVB_E_ARG, "ffcvb_poison: bad argument");
    CU(cudaSetDevice(ctx->device));
    cudaStream_t st = (cudaStream_t)stream;
    std::lock_guard<std::mutex> guard(ctx->aux_m);
    AuxBuf *a;
    int rc;
    if ((rc = stage_aux(ctx, st, (size_t)n, [&](uint8_t *host) { memcpy(host, apply, (size_t)n); }, &a))) return rc;
    launch_poison(images_dev, n, (long long)count, (const uint8_t *)a->dev.p, one_minus_alpha_dev, mask_dev,
                  (float)clamp_lo, (float)clamp_hi, st);
    CU(cudaGetLastError());
    CU(cudaEventRecord(a->ev, st));
    a->used = true;
    return FFCVB_OK;
}

int ffcvb_host_register(void *ptr, uint64_t bytes) {
    if (!ptr || bytes == 0) return FFCVB_E_ARG;
    if (cudaHostRegister(ptr, (size_t)bytes, cudaHostRegisterDefault) != cudaSuccess) {
        cudaGetLastError(); // refused (a read-only mapping, a file on disk): not an error of the process
        return FFCVB_E_CUDA;
    }
    return FFCVB_OK;
}

int ffcvb_host_unregister(void *ptr) {
    if (!ptr) return FFCVB_E_ARG;
    // gather kernels and copies that still read the range must be through before it is released
    cudaDeviceSynchronize();
    if (cudaHostUnregister(ptr) != cudaSuccess) {
        cudaGetLastError();
        return FFCVB_E_CUDA;
    }
    return FFCVB_OK;
}

// ------------------------------------------------------------ reference-signature entry points

static ffcvb_ctx *g_ctx = nullptr;
static std::mutex g_mutex;

static ffcvb_ctx *global_ctx() {
    if (!g_ctx) {
        int dev = 0;
        if (cudaGetDevice(&dev) != cudaSuccess) return nullptr;
        const long cores = sysconf(_SC_NPROCESSORS_ONLN);
        if (ffcvb_create(dev, 1, cores >= 16 ? 8 : (cores >= 4 ? (int)cores / 2 : 1), &g_ctx) != FFCVB_OK) return nullptr;
        if (cudaStreamCreateWithFlags(&g_ctx->one_stream, cudaStreamNonBlocking) != cudaSuccess) {
            ffcvb_destroy(g_ctx);
            g_ctx = nullptr;
        }
    }
    return g_ctx;
}

// Results of up to kZeroCopyBytes are written by the kernels straight into page-locked memory, which
// saves a copy's launch and latency; larger ones go through device memory, from where the copy engine
// fetches them piece by piece while the staging threads move the pieces that have landed on to the
// caller's pageable buffer (one thread alone moves about 10 GB/s, the link 55).
static constexpr size_t kZeroCopyBytes = 512 * 1024, kResultHead = 64; // (the head holds the status word)
static constexpr size_t kInputHead = 128;                              // parameters and ResizeItem of a resize call

// Queues the pieces of `bytes` from dev to the pinned result buffer, and copies them on into `out` when
// `ok` says so (asked when the first piece has landed).  Returns false on a CUDA error.
static bool fetch_result(ffcvb_ctx *ctx, const uint8_t *dev, uint8_t *out, size_t bytes, const std::function<bool()> &ok) {
    cudaStream_t st = ctx->one_stream;
    uint8_t *host = ctx->one_host + kResultHead;
    constexpr size_t kUnit = 128 * 1024;
    size_t piece = align_up((bytes + 15) / 16, kUnit);
    if (piece < 4 * kUnit) piece = 4 * kUnit;
    const int pieces = (int)((bytes + piece - 1) / piece);
    for (int k = 0; k < pieces; k++) {
        const size_t from = k * piece, len = bytes - from < piece ? bytes - from : piece;
        if (!ctx->one_ev[k] && cudaEventCreateWithFlags(&ctx->one_ev[k], cudaEventDisableTiming) != cudaSuccess) return false;
        if (cudaMemcpyAsync(host + from, dev + from, len, cudaMemcpyDeviceToHost, st) != cudaSuccess) return false;
        if (cudaEventRecord(ctx->one_ev[k], st) != cudaSuccess) return false;
    }
    std::atomic<bool> good{true};
    ctx->pool->parallel_for((int)((bytes + kUnit - 1) / kUnit), 1, [&](int i) {
        const size_t from = i * kUnit, len = bytes - from < kUnit ? bytes - from : kUnit;
        if (cudaEventSynchronize(ctx->one_ev[from / piece]) != cudaSuccess)
            good.store(false);
        else if (ok())
            memcpy(out + from, host + from, len);
    });
    return good.load() && cudaStreamSynchronize(st) == cudaSuccess;
}

int imdecode(unsigned char *input_buffer, uint64_t input_size, uint32_t source_height,
             uint32_t source_width, unsigned char *output_buffer, uint32_t crop_height,
             uint32_t crop_width, uint32_t offset_x, uint32_t offset_y, uint32_t scale_num,
             uint32_t scale_denom, bool enable_crop, bool hflip) {
    (void)source_height;
    (void)source_width;
    (void)offset_x;
    (void)offset_y;
    // Every call the reference makes passes the identity transform and scale 1/1
    // (rgb_image.py:131-132,196-197).  Scales 1/2, 1/4 and 1/8 are decoded too: as in the reference's
    // call, the output then has TJSCALED(crop, scale) = ceil(crop * num / denom) pixels a side.
    if (enable_crop || hflip || !input_buffer || !output_buffer || scale_num == 0 || scale_denom % scale_num != 0) return -1;
    const uint32_t denom = scale_denom / scale_num;
    if (denom != 1 && denom != 2 && denom != 4 && denom != 8) return -1;
    const int shift = denom == 1 ? 0 : (denom == 2 ? 1 : (denom == 4 ? 2 : 3));
    std::lock_guard<std::mutex> g(g_mutex);
    ffcvb_ctx *ctx = global_ctx();
    if (!ctx) return -1;
    if (crop_height == 0 || crop_width == 0 || crop_height > 65535 || crop_width > 65535) return -1;
    ffcvb_plan plan{};
    plan.out_h = (int32_t)((crop_height + denom - 1) / denom);
    plan.out_w = (int32_t)((crop_width + denom - 1) / denom);
    plan.resize = 0;
    plan.dct_scale = shift;
    plan.out_kind = FFCVB_OUT_U8_NHWC;
    const uint64_t ptr = 0, size = input_size;
    const uint8_t mode = FFCVB_MODE_JPG;
    const uint16_t hh = (uint16_t)crop_height, ww = (uint16_t)crop_width;
    const int32_t params[4] = {0, 0, (int32_t)crop_height, (int32_t)crop_width};
    Slot &s = ctx->slots[0];
    s.packed = true;
    if (ffcvb_stage_batch(ctx, 0, input_buffer, &ptr, &size, &mode, &hh, &ww, 1, &plan, params)) return -1;
    if (s.descs[0].host_status != 0) return -1;
    const size_t out_bytes = (size_t)plan.out_h * plan.out_w * 3;
    const bool zero_copy = out_bytes <= kZeroCopyBytes;
    if (grow_host(ctx, ctx->one_host, ctx->one_host_cap, kResultHead + out_bytes)) return -1;
    if (!zero_copy && grow_dev(ctx, ctx->one_dst, out_bytes)) return -1;
    volatile int32_t *status = (volatile int32_t *)ctx->one_host;
    *status = 0;
    const Single single{zero_copy ? ctx->one_host + kResultHead : (uint8_t *)ctx->one_dst.p, (int32_t *)ctx->one_host,
                        zero_copy || plan.out_w % 4 != 0};
    if (run_batch(ctx, s, ctx->one_stream, nullptr, true, &single)) return -1;
    if (zero_copy) {
        if (cudaStreamSynchronize(ctx->one_stream) != cudaSuccess || *status != 0) return -1;
        memcpy(output_buffer, ctx->one_host + kResultHead, out_bytes);
        return 0;
    }
    return fetch_result(ctx, (const uint8_t *)ctx->one_dst.p, output_buffer, out_bytes, [&] { return *status == 0; }) && *status == 0 ? 0 : -1;
}

void resize(int64_t cresizer, int64_t source_p, int64_t sx, int64_t sy, int64_t start_row,
            int64_t end_row, int64_t start_col, int64_t end_col, int64_t dest_p, int64_t tx, int64_t ty) {
    (void)cresizer;
    std::lock_guard<std::mutex> g(g_mutex);
    ffcvb_ctx *ctx = global_ctx();
    if (!ctx || !source_p || !dest_p || sx <= 0 || sy <= 0 || tx <= 0 || ty <= 0) return;
    if (start_row < 0 || start_col < 0 || end_row > sx || end_col > sy || end_row <= start_row ||
        end_col <= start_col)
        return;
    // Only the region travels to the GPU, behind its parameters.
    const int rows = (int)(end_row - start_row), cols = (int)(end_col - start_col);
    const size_t pitch = (size_t)cols * 3, src_bytes = kInputHead + (size_t)rows * pitch, dst_bytes = (size_t)tx * ty * 3;
    const bool zero_copy = dst_bytes <= kZeroCopyBytes;
    if (cudaSetDevice(ctx->device) != cudaSuccess) return;
    if (grow_dev(ctx, ctx->one_src, src_bytes + 64) || grow_host(ctx, ctx->one_in, ctx->one_in_cap, src_bytes) ||
        grow_host(ctx, ctx->one_host, ctx->one_host_cap, kResultHead + dst_bytes) || (!zero_copy && grow_dev(ctx, ctx->one_dst, dst_bytes)))
        return;
    const int32_t params[4] = {0, 0, rows, cols};
    ResizeItems items(1, (int)tx, (int)ty, FFCVB_OUT_U8_NHWC);
    const ResizeItem item = items.make(params, rows, cols, ResizeItems::kPacked);
    memcpy(ctx->one_in, params, sizeof(params));
    memcpy(ctx->one_in + 64, &item, sizeof(item));
    const uint8_t *src = (const uint8_t *)(intptr_t)source_p + ((size_t)start_row * sy + start_col) * 3;
    uint8_t *in = ctx->one_in + kInputHead;
    auto copy_rows = [&](int lo, int hi, auto copy) {
        if (cols == sy)
            copy(in + lo * pitch, src + lo * pitch, (hi - lo) * pitch);
        else
            for (int r = lo; r < hi; r++) copy(in + r * pitch, src + (size_t)r * sy * 3, pitch);
    };
    cudaStream_t st = ctx->one_stream;
    // Up to two parts of about 256 KB: each under way while the next one is copied.  More: copied by all threads, then
    // one transfer (1.2 MB: 139 -> 98 us; 2 MB: 197 -> 113; 4.3 MB: 355 -> 180).
    const int part = (int)(256 * 1024 / pitch) + 1, parts = (rows + part - 1) / part;
    const bool together = parts > 2;
    if (together)
        ctx->pool->parallel_for(parts, 1, [&](int k) {
            copy_rows(k * part, (k + 1) * part < rows ? (k + 1) * part : rows, stream_copy_lines);
            _mm_sfence();
        });
    for (int k = 0; k < (together ? 1 : parts); k++) {
        const int lo = k * part, hi = together || lo + part > rows ? rows : lo + part;
        if (!together) copy_rows(lo, hi, memcpy);
        const size_t from = k == 0 ? 0 : kInputHead + lo * pitch, to = kInputHead + hi * pitch;
        if (cudaMemcpyAsync((uint8_t *)ctx->one_src.p + from, ctx->one_in + from, to - from, cudaMemcpyHostToDevice, st) != cudaSuccess) return;
    }
    ResizeSource rs{};
    rs.uniform = (const uint8_t *)ctx->one_src.p + kInputHead;
    rs.uniform_h = rows;
    rs.uniform_w = cols;
    uint8_t *out = zero_copy ? ctx->one_host + kResultHead : (uint8_t *)ctx->one_dst.p;
    launch_resize_augment(rs, 1, (const int32_t *)ctx->one_src.p, 4, (const ResizeItem *)((const uint8_t *)ctx->one_src.p + 64), OpList{}, 1, (int)tx, (int)ty,
                          FFCVB_OUT_U8_NHWC, items.bands(), items.plain(), nullptr, out, nullptr, SmallCopies{}, false, st);
    if (cudaGetLastError() != cudaSuccess) return;
    if (zero_copy) {
        if (cudaStreamSynchronize(st) == cudaSuccess) memcpy((void *)(intptr_t)dest_p, out, dst_bytes);
    } else {
        fetch_result(ctx, out, (uint8_t *)(intptr_t)dest_p, dst_bytes, [] { return true; });
    }
}

void my_memcpy(void *source, void *dst, uint64_t size) { memcpy(dst, source, size); }

void my_fread(int64_t fp, int64_t offset, void *destination, int64_t size) {
    FILE *f = reinterpret_cast<FILE *>(static_cast<intptr_t>(fp));
    if (!f || !destination || size <= 0 || offset < 0) return;
    if (fseek(f, (long)offset, SEEK_SET) != 0) return;
    size_t got = fread(destination, 1, (size_t)size, f);
    (void)got;
}

} // extern "C"
