"""Who writes and who reads the entries of the decode index, over random orders of staging, submitting and
ending batches: the host's bookkeeping (csrc/decode_index.h), compiled on its own."""
import os
import random
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), 'ffcv_b200', 'csrc')
PROGRAM = r'''
#include <stdio.h>
#include "decode_index.h"
int main() {
    ffcvb::DecodeIndex index;
    char op;
    unsigned long long a, b, c;
    while (scanf(" %c %llu %llu %llu", &op, &a, &b, &c) == 4) {
        if (op == 'r') index.reset(a, (int)b);
        if (op == 's') index.staged((int)a);
        if (op == 'q') { index.submitted((int)a); index.marked((int)a); }
        if (op == 'f') index.submitted((int)a);
        if (op == 'e' && index.unsettled((int)a)) index.ended((int)a);
        if (op == 't') {
            const auto p = index.take(a, (unsigned)b, 100, (int)c);
            printf("%d %llu\n", (int)p.use, (unsigned long long)p.off);
        }
    }
}
'''


@pytest.fixture(scope='module')
def program(tmp_path_factory):
    d = tmp_path_factory.mktemp('index')
    (d / 'main.cpp').write_text(PROGRAM)
    subprocess.run(['g++', '-std=c++17', '-I', CSRC, '-o', str(d / 'main'), str(d / 'main.cpp')], check=True)

    def run(ops):
        text = '\n'.join('%s %d %d %d' % (tuple(op) + (0,) * (4 - len(op))) for op in ops) + '\n'
        out = subprocess.run([str(d / 'main')], input=text, capture_output=True, text=True, check=True).stdout.split()
        return list(zip(map(int, out[::2]), map(int, out[1::2])))
    return run


NONE, READ, WRITE = 0, 1, 3


def test_an_entry_is_not_read_while_another_slot_writes_it(program):
    # two slots; the writer, in slot 0, is queued and still runs while slot 1 takes batch after batch
    ops = [('r', 1000, 2), ('s', 0), ('t', 7, 1, 0), ('q', 0)]
    for _ in range(4):
        ops += [('s', 1), ('t', 7, 1, 1), ('q', 1)]
    ops += [('s', 0), ('t', 7, 1, 0), ('q', 0), ('e', 0), ('s', 1), ('t', 7, 1, 1)]
    assert [use for use, _ in program(ops)] == [WRITE, NONE, NONE, NONE, NONE, READ, READ]


def test_limits(program):
    # the same stream twice in a batch; no room; another way of cutting it; a batch that is never submitted
    ops = [('r', 250, 2), ('s', 0), ('t', 1, 1, 0), ('t', 1, 1, 0), ('t', 2, 1, 0), ('t', 3, 1, 0), ('t', 1, 2, 0),
           ('s', 0), ('t', 1, 1, 0), ('q', 0), ('s', 1), ('t', 2, 1, 1), ('s', 0), ('t', 1, 1, 0)]
    assert program(ops) == [(WRITE, 0), (NONE, 0), (WRITE, 100), (NONE, 0), (NONE, 0), (WRITE, 0), (WRITE, 100), (READ, 0)]


@pytest.mark.parametrize('seed', range(20))
def test_random_orders(program, seed):
    rng = random.Random(seed)
    slots, keys = rng.randint(1, 5), rng.randint(1, 6)
    ops, events = [('r', 10 ** 6, slots)], []
    for _ in range(3000):
        w, kind = rng.randrange(slots), rng.choice('stttqqe')
        if kind == 't':
            k = rng.randrange(keys)
            ops.append(('t', k, 1, w))
            events.append(('t', w, k))
        elif kind == 'q' and rng.random() < 0.05:
            ops.append(('f', w))  # submitted, failed before its event was recorded
            events.append(('f', w))
        else:
            ops.append((kind, w))
            events.append((kind, w))
    answers = iter(program(ops))
    staged, submitted, marked, ended = ([0] * slots for _ in range(4))
    writer = {}  # key -> (slot, batch)
    reads = 0
    for ev in events:
        w = ev[1]
        if ev[0] == 's':
            if submitted[w] != staged[w]:
                writer = {k: v for k, v in writer.items() if v != (w, staged[w])}
            staged[w] += 1
        elif ev[0] in 'qf':
            submitted[w] = staged[w]
            if ev[0] == 'q':
                marked[w] = staged[w]
        elif ev[0] == 'e':
            ended[w] = max(ended[w], marked[w])
        else:
            use, off = next(answers)
            known = writer.get(ev[2])
            if known is None:
                assert use == WRITE
                writer[ev[2]] = (w, staged[w])
            else:
                slot, batch = known
                safe = batch <= ended[slot] or (slot == w and batch <= submitted[w] and batch < staged[w])
                assert use == (READ if safe else NONE), (ev, known)
                reads += use == READ
    assert reads > 0
