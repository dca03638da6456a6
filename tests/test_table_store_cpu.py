"""The store of Huffman and quantisation tables (csrc/table_store.h), compiled on its own: tables whose hashes
collide, more tables than stay built, as many as it keeps, and the memory they take."""
import os
import subprocess

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), 'ffcv_b200', 'csrc')
PROGRAM = r'''
#include <malloc.h>
#include <stdio.h>
#include <stdlib.h>
#include "table_store.h"
using namespace ffcvb;
#define CHECK(x) do { if (!(x)) { printf("line %d: %s\n", __LINE__, #x); return 1; } } while (0)

// 16 codes of 6 bits and `n` of 8, symbols told apart by `seed`
static RawHuff table(int n, unsigned seed) {
    RawHuff t{};
    t.bits[6] = 16;
    t.bits[8] = (uint8_t)n;
    for (int k = 0; k < 16 + n; k++) t.vals[k] = (uint8_t)(seed >> (8 * (k % 4)));
    t.present = true;
    return t;
}
static JpegHeader header(unsigned seed) {
    static JpegHeader h;
    memset(&h, 0, sizeof(h));
    h.ncomp = 3;
    h.tq[1] = h.tq[2] = h.td[1] = h.td[2] = h.ta[1] = h.ta[2] = 1;
    for (int k = 0; k < 2; k++) {
        h.dc[k] = table(8 + k, seed);
        h.ac[k] = table(8 + k, seed);
        for (int z = 0; z < 64; z++) h.quant[k][z] = (uint16_t)(1 + seed % 250 + k);
    }
    return h;
}
static bool same_table(const HuffTable &a, const RawHuff &raw, bool dc) {
    static HuffTable want;
    build_huff_table(raw, dc, &want);
    return memcmp(&a, &want, sizeof(want)) == 0;
}

int main() {
    static TableStore store;
    // the same hash: values, code lengths or use differ
    RawHuff a = table(5, 1), b = table(5, 2), c = a;
    c.bits[8] = 4, c.bits[9] = 1; // as many codes, the same values
    const uint32_t ia = store.add_huff(a, false, 7), ib = store.add_huff(b, false, 7), ic = store.add_huff(c, false, 7), id = store.add_huff(a, true, 7);
    CHECK(ia != ib && ia != ic && ib != ic && id != ia && id != ib && id != ic);
    CHECK(store.add_huff(a, false, 7) == ia && store.add_huff(b, false, 7) == ib && store.add_huff(c, false, 7) == ic && store.add_huff(a, true, 7) == id);
    CHECK(same_table(store.built(ic), c, false) && same_table(store.built(id), a, true));
    uint16_t q[64] = {}, r[64] = {};
    r[63] = 1;
    const uint32_t iq = store.add_quant(q, 9), ir = store.add_quant(r, 9);
    CHECK(iq != ir && store.add_quant(q, 9) == iq && store.quant(ir)[63] == 1);
    store.clear();

    // headers whose hashes are all alike, in more or fewer components
    uint64_t none[9] = {};
    JpegHeader heads[5] = {header(1), header(2), header(1), header(1), header(1)};
    heads[2].ta[2] = 0;
    heads[3].tq[1] = 0;
    heads[4].ncomp = 1;
    for (int k = 0; k < 5; k++) CHECK(store.find(heads[k], none) == TableStore::kNone && store.add(heads[k], none) == (uint32_t)k);
    for (int k = 0; k < 5; k++) CHECK(store.find(heads[k], none) == (uint32_t)k);
    CHECK(store.set(2).ac_tab[2] == store.set(2).ac_tab[0] && store.set(3).quant[1] == store.set(3).quant[0]);
    store.clear();

    // as many distinct tables as are kept, four a header
    const size_t before = mallinfo2().uordblks + mallinfo2().hblkhd;
    unsigned n = 0;
    uint64_t hash[9] = {};
    for (; !store.full(); n++) {
        const JpegHeader h = header(n);
        for (int k = 0; k < 9; k++) hash[k] = (uint64_t)n * 16 + (k < 3 ? k : 3 + k % 3);
        CHECK(n % 1000 != 0 || store.find(h, hash) == TableStore::kNone);
        const uint32_t set = store.add(h, hash);
        CHECK(set == n && store.add(h, hash) == set && store.find(h, hash) == set);
        const TableSet &ts = store.set(set);
        CHECK(ts.n_tab == 4 && ts.n_dc_tab == 2 && ts.dc_tab[0] == 0 && ts.dc_tab[1] == 1 && ts.dc_tab[2] == 1 && ts.ac_tab[0] == 2 && ts.ac_tab[2] == 3);
    }
    const double mb = (mallinfo2().uordblks + mallinfo2().hblkhd - before) / 1e6;
    CHECK(n == TableStore::kMost / 4);
    for (unsigned k : {0u, 1u, 255u, 256u, n / 2, n - 1}) { // the oldest ones and those built last
        const JpegHeader h = header(k);
        const TableSet &ts = store.set(k);
        CHECK(same_table(store.built(ts.huff[0]), h.dc[0], true) && same_table(store.built(ts.huff[1]), h.dc[1], true));
        CHECK(same_table(store.built(ts.huff[2]), h.ac[0], false) && same_table(store.built(ts.huff[3]), h.ac[1], false));
        CHECK(memcmp(store.quant(ts.quant[1]), h.quant[1], 128) == 0);
    }
    store.clear();
    CHECK(!store.full());
    const JpegHeader h = header(5);
    CHECK(store.add(h, hash) == 0 && same_table(store.built(store.set(0).huff[0]), h.dc[0], true));
    printf("%.1f\n", mb);
    return 0;
}
'''


def test_table_store(tmp_path):
    (tmp_path / 'main.cpp').write_text(PROGRAM)
    subprocess.run(['g++', '-std=c++17', '-O1', '-I', CSRC, '-o', str(tmp_path / 'main'), str(tmp_path / 'main.cpp'),
                    os.path.join(CSRC, 'jpeg_header.cpp')], check=True)
    res = subprocess.run([str(tmp_path / 'main')], capture_output=True, text=True)
    assert res.returncode == 0, res.stdout
    assert float(res.stdout) < 40  # MB; built, the 60 000 tables would take 580
