// The distinct Huffman and quantisation tables of the JPEG streams a context has seen (host only).  An index
// names a table until clear(); a store that is full() is cleared by its owner, with all that holds indices, before
// it takes more: streams whose encoder optimises its tables bring new ones with every image.
#pragma once
#include <stdint.h>
#include <string.h>

#include <array>
#include <memory>
#include <unordered_map>
#include <vector>

#include "jpeg_header.h"
#include "types.h"

namespace ffcvb {

// The distinct tables of a JPEG stream: what all images of one encoder share.
struct TableSet {
    uint8_t ncomp, n_tab, n_dc_tab, fast, dc_tab[kMaxComponents], ac_tab[kMaxComponents]; // as in ImageDesc
    uint32_t huff[6];                                                              // of the n_tab tables
    uint32_t quant[kMaxComponents];
};

class TableStore {
  public:
    static constexpr size_t kMost = 60000; // tables or sets kept, and those of the batch that brings more: some 25 MB
    bool full() const { return huff_.size() >= kMost || quant_.size() >= kMost || sets_.size() >= kMost; }
    void clear() {
        huff_.clear();
        quant_.clear();
        sets_.clear();
        huff_by_hash_.clear();
        quant_by_hash_.clear();
        set_by_hash_.clear();
        for (Built &b : built_) b.index = kNone;
    }

    static constexpr uint32_t kNone = 0xFFFFFFFFu;
    // Index of the table set of a parsed header, kNone if it is not there; `hash`: of its tables, three per component
    // (DC, AC, quantisation).  Several threads may look at once.
    uint32_t find(const JpegHeader &h, const uint64_t *hash) const {
        const auto range = set_by_hash_.equal_range(key_of(h, hash));
        for (auto it = range.first; it != range.second; ++it)
            if (is(sets_[it->second], h)) return it->second;
        return kNone;
    }
    // The same, put there if it is not.
    uint32_t add(const JpegHeader &h, const uint64_t *hash) {
        const uint32_t known = find(h, hash);
        if (known != kNone) return known;
        TableSet ts;
        memset(&ts, 0, sizeof(ts));
        ts.ncomp = (uint8_t)h.ncomp;
        ts.fast = 1;
        for (int k = 0; k < 2; k++) { // DC tables first
            for (int c = 0; c < h.ncomp; c++) {
                const uint32_t t = add_huff(k == 0 ? h.dc[h.td[c]] : h.ac[h.ta[c]], k == 0, hash[3 * c + k]);
                int u = k == 0 ? 0 : ts.n_dc_tab;
                while (u < ts.n_tab && ts.huff[u] != t) u++;
                if (u == ts.n_tab) ts.huff[ts.n_tab++] = t;
                (k == 0 ? ts.dc_tab : ts.ac_tab)[c] = (uint8_t)u;
                if (!huff_[t].fast) ts.fast = 0;
            }
            if (k == 0) ts.n_dc_tab = ts.n_tab;
        }
        for (int c = 0; c < h.ncomp; c++) ts.quant[c] = add_quant(h.quant[h.tq[c]], hash[3 * c + 2]);
        set_by_hash_.emplace(key_of(h, hash), (uint32_t)sets_.size());
        sets_.push_back(ts);
        return (uint32_t)sets_.size() - 1;
    }
    uint32_t add_huff(const RawHuff &raw, bool dc, uint64_t hash) {
        const auto range = huff_by_hash_.equal_range(hash);
        for (auto it = range.first; it != range.second; ++it) {
            const Huff &t = huff_[it->second];
            if (t.dc == dc && same(t.raw, raw)) return it->second;
        }
        const uint32_t index = (uint32_t)huff_.size();
        huff_by_hash_.emplace(hash, index);
        huff_.push_back(Huff{raw, dc, false});
        huff_.back().fast = built(index).fast_ok != 0;
        return index;
    }
    uint32_t add_quant(const uint16_t *quant, uint64_t hash) {
        const auto range = quant_by_hash_.equal_range(hash);
        for (auto it = range.first; it != range.second; ++it)
            if (memcmp(quant_[it->second].data(), quant, 128) == 0) return it->second;
        quant_by_hash_.emplace(hash, (uint32_t)quant_.size());
        quant_.emplace_back();
        memcpy(quant_.back().data(), quant, 128);
        return (uint32_t)quant_.size() - 1;
    }

    const TableSet &set(uint32_t index) const { return sets_[index]; }
    const uint16_t *quant(uint32_t index) const { return quant_[index].data(); }
    // The table in the form the kernels use, valid until the next call.  The last few stay built: a table is ten
    // kilobytes then, 35 times its description.
    const HuffTable &built(uint32_t index) {
        Built &b = built_[index % kBuilt];
        if (b.index != index) {
            if (!b.table) b.table.reset(new HuffTable());
            build_huff_table(huff_[index].raw, huff_[index].dc, b.table.get());
            b.index = index;
        }
        return *b.table;
    }

  private:
    static constexpr uint32_t kBuilt = 256; // (a batch has at most 255)
    struct Huff {
        RawHuff raw;
        bool dc, fast;
    };
    struct Built {
        uint32_t index = kNone;
        std::unique_ptr<HuffTable> table;
    };
    static bool same(const RawHuff &a, const RawHuff &b) { return memcmp(a.bits, b.bits, 17) == 0 && memcmp(a.vals, b.vals, 256) == 0; }
    static uint64_t key_of(const JpegHeader &h, const uint64_t *hash) {
        uint64_t key = (uint64_t)h.ncomp;
        for (int c = 0; c < 3 * h.ncomp; c++) {
            key = (key ^ hash[c]) * 0xFF51AFD7ED558CCDull;
            key ^= key >> 29;
        }
        return key;
    }
    // Whether `ts` holds the tables of this header, each where its components look for it.
    bool is(const TableSet &ts, const JpegHeader &h) const {
        if (ts.ncomp != h.ncomp) return false;
        for (int c = 0; c < h.ncomp; c++) {
            if (c == 2 && h.td[2] == h.td[1] && h.ta[2] == h.ta[1] && h.tq[2] == h.tq[1])
                return ts.dc_tab[2] == ts.dc_tab[1] && ts.ac_tab[2] == ts.ac_tab[1] && ts.quant[2] == ts.quant[1];
            if (!same(huff_[ts.huff[ts.dc_tab[c]]].raw, h.dc[h.td[c]]) || !same(huff_[ts.huff[ts.ac_tab[c]]].raw, h.ac[h.ta[c]]) ||
                memcmp(quant_[ts.quant[c]].data(), h.quant[h.tq[c]], 128) != 0)
                return false;
        }
        return true;
    }
    std::vector<Huff> huff_;
    std::vector<std::array<uint16_t, 64>> quant_;
    std::vector<TableSet> sets_;
    std::unordered_multimap<uint64_t, uint32_t> huff_by_hash_, quant_by_hash_, set_by_hash_;
    std::array<Built, kBuilt> built_;
};

} // namespace ffcvb
