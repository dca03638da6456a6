// Payload gather from pinned host memory over PCIe (sm_100a): the GPU reads the sample bytes of a
// batch straight out of the page-locked dataset file, so no host core touches them.
#include "kernels.h"

namespace ffcvb {

namespace {

// The bytes go through shared memory as bulk copies (host -> shared, shared -> device) that one thread
// per CTA issues: a ring of kStages pieces per CTA, half of them on their way in while the others leave.
// What bounds it is the link, and there the number of read requests: about 400 million a second, one for every
// line of 128 bytes that a piece touches.  Pieces therefore end at multiples of kLine of the source, so that no
// line is asked for twice: alone, one CTA per SM with 8 KB moves 49.5 / 50.3 / 50.9 GB/s of JPEG streams of 16 KB,
// 60 KB and 1.7 MB (46.7 / 47.3 / 48.0 with pieces cut from the stream's first word on) and 44.7 GB/s of 0.7 KB crop
// rows (44.1); pieces of 512 bytes and of 2 KB: the same.  A plain DMA copy: 54.5; 64 CTAs: 33 GB/s of rows; two per SM:
// 3 % more rows, but the decode kernels beside it slow down by as much.  As important is what it leaves to the decode
// kernels: no issue slots, and 8 KB of shared memory per SM, which two CTAs of the entropy decoder do not need.
constexpr int kStages = 8, kPiece = 1024, kAhead = 5; // kAhead: pieces on their way in
constexpr uint32_t kLine = 128;

__device__ __forceinline__ uint32_t shared_address(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

struct Ring {
    uint64_t dst[kStages];
    uint32_t len[kStages];
    uint32_t issued, stored;
    uint64_t limit; // of a wait, in nanoseconds
    bool failed;
};

// Waits for the piece in stage `st`, `limit` nanoseconds at most (0: looks once); false: it did not arrive.
__device__ __forceinline__ bool arrived(uint64_t *bars, uint32_t st, uint32_t parity, uint64_t limit) {
    uint64_t begin = 0;
    for (;;) {
        uint32_t ok;
        if (limit == 0) {
            asm volatile("{\n\t.reg .pred p;\n\tmbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                         : "=r"(ok)
                         : "r"(shared_address(&bars[st])), "r"(parity)
                         : "memory");
            return ok != 0;
        }
        asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                     : "=r"(ok)
                     : "r"(shared_address(&bars[st])), "r"(parity)
                     : "memory");
        if (ok) return true;
        uint64_t now;
        asm volatile("mov.u64 %0, %globaltimer;" : "=l"(now));
        if (begin == 0) begin = now;
        if (now - begin > limit) return false;
    }
}

// Sends the oldest piece on its way in out again.
__device__ __forceinline__ void store_oldest(Ring &r, uint8_t *buf, uint64_t *bars, uint8_t *blob) {
    const uint32_t st = r.stored % kStages;
    if (!arrived(bars, st, (r.stored / kStages) & 1, r.limit)) {
        r.failed = true;
        return;
    }
    asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(blob + r.dst[st]), "r"(shared_address(buf + st * kPiece)),
                 "r"(r.len[st])
                 : "memory");
    asm volatile("cp.async.bulk.commit_group;" ::: "memory");
    r.stored++;
}

// Sends `len` bytes (a multiple of 16, as both addresses) through the ring.
__device__ __forceinline__ void send(Ring &r, uint8_t *buf, uint64_t *bars, uint8_t *blob, uint64_t src, uint64_t dst, uint32_t len) {
    uint32_t take;
    for (uint32_t off = 0; off < len && !r.failed; off += take) {
        if (r.issued - r.stored >= kAhead) store_oldest(r, buf, bars, blob);
        if (r.failed) return;
        const uint32_t st = r.issued % kStages;
        take = min(len - off, (uint32_t)kPiece - ((uint32_t)(src + off) & (kLine - 1)));
        // the piece that used this stage last has been read out: at most kStages - kAhead stores are younger
        if (r.issued >= kStages) asm volatile("cp.async.bulk.wait_group.read %0;" ::"n"(kStages - kAhead) : "memory");
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(shared_address(&bars[st])), "r"(take) : "memory");
        asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(shared_address(buf + st * kPiece)),
                     "l"(src + off), "r"(take), "r"(shared_address(&bars[st]))
                     : "memory");
        r.dst[st] = dst + off;
        r.len[st] = take;
        r.issued++;
    }
}

// CTA k fetches what lies between ranges[k] and ranges[k + 1] (see gather_ranges).  One that gives up marks all of its
// samples as failed, for the kernels that follow and in `status`.
__global__ void __launch_bounds__(32)
gather_payloads_kernel(ImageDesc *descs, const uint2 *__restrict__ ranges, uint8_t *__restrict__ blob, int32_t *status, uint64_t limit,
                       int32_t *failed) {
    __shared__ __align__(128) uint8_t s_buf[kStages * kPiece];
    __shared__ __align__(8) uint64_t s_bars[kStages];
    const int lane = threadIdx.x;
    if (lane < kStages) asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(shared_address(&s_bars[lane])) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncwarp();
    const uint2 from = ranges[blockIdx.x], to = ranges[blockIdx.x + 1];
    const uint32_t behind = to.x + (to.y != 0 ? 1 : 0); // samples [from.x, behind) have bytes for this CTA
    Ring ring{};
    ring.limit = limit;
    for (uint32_t first = from.x; first < behind; first += 32) {
        // the descriptors of this CTA's next 32 samples, one per lane: rows, or one run
        const uint32_t item = first + lane;
        uint64_t src = 0, dst = 0;
        uint32_t run = 0, rows = 0, src_pitch = 0, dst_pitch = 0;
        if (item < behind) {
            const ImageDesc &d = descs[item];
            const uint32_t begin = item == from.x ? from.y : 0, end = item == to.x ? to.y : 0xFFFFFFFFu;
            if (d.src_addr != 0 && d.payload_size != 0) {
                if (d.mode == 1 && d.raw_skew) { // a crop box: rows, each as the aligned 16-byte words that hold it
                    const uint32_t last = min((uint32_t)d.rows, end);
                    src_pitch = (uint32_t)d.width * 3;
                    dst_pitch = d.raw_pitch;
                    run = (uint32_t)d.cols * 3;
                    rows = last > begin ? last - begin : 0;
                    src = d.src_addr + (uint64_t)begin * src_pitch;
                    dst = d.payload_off + (uint64_t)begin * dst_pitch;
                } else { // source and destination have the same alignment
                    const uint32_t lead = (uint32_t)(d.src_addr & 15), last = min(lead + d.payload_size, end);
                    rows = last > begin ? 1 : 0;
                    run = last - begin;
                    src = d.src_addr - lead + begin;
                    dst = d.payload_off - lead + begin;
                }
            }
        }
        for (uint32_t k = 0; k < 32 && first + k < behind; k++) {
            const uint64_t s = __shfl_sync(0xffffffffu, src, k), t = __shfl_sync(0xffffffffu, dst, k);
            const uint32_t len = __shfl_sync(0xffffffffu, run, k), m = __shfl_sync(0xffffffffu, rows, k);
            const uint32_t sp = __shfl_sync(0xffffffffu, src_pitch, k), dp = __shfl_sync(0xffffffffu, dst_pitch, k);
            if (lane == 0)
                for (uint32_t r = 0; r < m && !ring.failed; r++) {
                    // (a word that holds one byte of the run lies in the same page as that byte: the reads stay
                    // inside the pinned allocation)
                    const uint64_t at = s + (uint64_t)r * sp;
                    const uint32_t lead = (uint32_t)(at & 15);
                    send(ring, s_buf, s_bars, blob, at - lead, t + (uint64_t)r * dp, (lead + len + 15) & ~15u);
                }
            __syncwarp();
        }
    }
    if (lane == 0) {
        while (ring.stored != ring.issued && !ring.failed) store_oldest(ring, s_buf, s_bars, blob);
        asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
        if (ring.failed) {
            for (uint32_t item = from.x; item < behind; item++) {
                ImageDesc &d = descs[item];
                if (d.src_addr == 0 || d.payload_size == 0) continue;
                d.host_status = (int16_t)kErrData;
                status[item] = kErrData;
            }
            *failed = 1;
            const uint64_t drain = max(limit, (uint64_t)2000000000ull); // (shared memory must outlive the copies into it)
            for (; ring.stored != ring.issued; ring.stored++) arrived(s_bars, ring.stored % kStages, (ring.stored / kStages) & 1, drain);
        }
    }
}

} // namespace

void gather_ranges(const ImageDesc *descs, int n, int ctas, uint2 *ranges) {
    auto rowwise = [](const ImageDesc &d) { return d.mode == 1 && d.raw_skew != 0; };
    // of a row; and of a run, without the lines that its ends share with nothing
    auto row_lines = [](const ImageDesc &d) { return ((uint64_t)d.cols * 3 + kLine - 1) / kLine + 1; };
    auto run_lines = [](const ImageDesc &d) { return ((d.src_addr & (kLine - 1)) + d.payload_size + kLine - 1) / kLine; };
    auto lines = [&](const ImageDesc &d) -> uint64_t {
        if (d.src_addr == 0 || d.payload_size == 0) return 0;
        return rowwise(d) ? d.rows * row_lines(d) : run_lines(d);
    };
    std::vector<uint32_t> of(n);
    uint64_t total = 0, before = 0; // before sample i
    for (int i = 0; i < n; i++) total += of[i] = (uint32_t)lines(descs[i]);
    int i = 0;
    for (int k = 0; k <= ctas; k++) {
        const uint64_t want = total * (uint64_t)k / (uint64_t)ctas;
        while (i < n && before + of[i] <= want) before += of[i++];
        if (k == 0 || k == ctas || i == n) {
            ranges[k] = make_uint2((uint32_t)(k == 0 ? 0 : n), 0);
            continue;
        }
        const ImageDesc &d = descs[i];
        const uint64_t inside = want - before; // lines of it that come before (fewer than it has)
        const uint64_t lead = d.src_addr & (kLine - 1), words = d.src_addr & 15; // a run begins with the word of its first byte
        const uint64_t at = rowwise(d) ? inside / row_lines(d) : (inside == 0 ? 0 : inside * kLine - lead + words);
        ranges[k] = make_uint2((uint32_t)i, (uint32_t)at);
    }
}

void launch_gather_payloads(ImageDesc *descs, const uint2 *ranges, int ctas, uint8_t *blob, int32_t *status, uint64_t limit_ns, int32_t *failed,
                            cudaStream_t stream) {
    gather_payloads_kernel<<<ctas, 32, 0, stream>>>(descs, ranges, blob, status, limit_ns, failed);
}

} // namespace ffcvb
