// Which batches may write and which may read the entries of the decode index (host only; what an entry
// holds: DecodeIndexHeader).  An entry is written by one batch and only read afterwards.  A batch on another
// stream may read it once the writing batch has ended on the device, one in the writer's own slot, whose
// batches run in order, as soon as that is queued.
#pragma once
#include <stddef.h>
#include <stdint.h>

#include <unordered_map>
#include <vector>

namespace ffcvb {

class DecodeIndex {
  public:
    enum Use : uint32_t { kNone = 0, kRead = 1, kWrite = 3 };
    struct Place {
        uint64_t off = 0;
        Use use = kNone;
    };
    // `bytes` of the pool, for batches in n_slots slots.
    void reset(size_t bytes, int n_slots) {
        room_ = bytes;
        used_ = 0;
        entries_.clear();
        slots_.assign(n_slots, Batches{});
    }
    size_t entries() const { return entries_.size(); }
    size_t used() const { return used_; }

    // A batch is being staged in the slot, in place of the one before: what that one was to write is free again
    // unless it was submitted.
    void staged(int slot) {
        Batches &b = slots_[slot];
        if (b.submitted != b.staged)
            for (uint64_t key : b.writes) entries_[key].slot = kUnclaimed;
        b.writes.clear();
        b.staged++;
    }
    // Its kernels are about to be queued; `marked`: an event behind them has been recorded.
    void submitted(int slot) { slots_[slot].submitted = slots_[slot].staged; }
    void marked(int slot) { slots_[slot].marked = slots_[slot].submitted; }
    // That event has not been seen to complete yet / has completed.
    bool unsettled(int slot) const { return slots_[slot].ended < slots_[slot].marked; }
    void ended(int slot) { slots_[slot].ended = slots_[slot].marked; }

    // What the batch being staged in `slot` does with the entry of stream `key`, of `bytes` bytes for a scan of
    // `segments`.
    Place take(uint64_t key, uint32_t segments, size_t bytes, int slot) {
        Batches &b = slots_[slot];
        auto it = entries_.find(key);
        if (it == entries_.end()) {
            if (used_ + bytes > room_) return Place{}; // this stream stays without
            it = entries_.emplace(key, Entry{used_, segments, kUnclaimed, 0}).first;
            used_ += bytes;
        }
        Entry &e = it->second;
        if (e.segments != segments) return Place{};
        if (e.slot == kUnclaimed) {
            e.slot = slot;
            e.batch = b.staged;
            b.writes.push_back(key);
            return Place{e.off, kWrite};
        }
        if (e.slot == kWritten) return Place{e.off, kRead};
        const Batches &w = slots_[e.slot];
        if (e.batch <= w.ended) {
            e.slot = kWritten;
            return Place{e.off, kRead};
        }
        return e.slot == slot && e.batch < b.staged ? Place{e.off, kRead} : Place{};
    }

  private:
    static constexpr int kUnclaimed = -1, kWritten = -2;
    struct Entry {
        uint64_t off = 0;
        uint32_t segments = 0;
        int slot = kUnclaimed; // of the batch that writes it
        uint64_t batch = 0;    // ... counted by the slot's staging calls
    };
    struct Batches { // of a slot: the last one staged, submitted, marked by an event, seen to have ended
        uint64_t staged = 0, submitted = 0, marked = 0, ended = 0;
        std::vector<uint64_t> writes; // keys that the staged one was given to write
    };
    std::unordered_map<uint64_t, Entry> entries_;
    std::vector<Batches> slots_;
    size_t room_ = 0, used_ = 0;
};

} // namespace ffcvb
