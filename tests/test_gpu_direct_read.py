"""Reads of few samples are shared out in pieces of 128 KB, except those with O_DIRECT from a disk: samples on both sides of that size, anywhere in the file, on a
memory file system and on a disk's, with and without O_DIRECT, and a file that ends too early."""
import os

import numpy as np
import pytest
import torch as ch

from ffcv_b200 import libffcv as L

pytestmark = pytest.mark.gpu
H = 8


def _open(kind, tmp_path, data):
    if kind == 'memory':
        fd = os.memfd_create('samples')
        path = '/proc/self/fd/%d' % fd
    else:
        path = str(tmp_path / 'samples')
        fd = os.open(path, os.O_RDWR | os.O_CREAT)
    view = memoryview(data.tobytes())
    while view:
        view = view[os.write(fd, view):]
    os.fsync(fd)
    try:
        direct = os.open(path, os.O_RDONLY | os.O_DIRECT)
    except OSError:
        direct = -1
    return fd, direct


@pytest.mark.parametrize('kind', ['memory', 'disk'])
@pytest.mark.parametrize('use_direct', [False, True], ids=['buffered', 'o_direct'])
@pytest.mark.parametrize('n', [1, 5, 130])
@pytest.mark.parametrize('cut', [0, 1, 140000])
def test_pieces_of_samples(kind, use_direct, n, cut, tmp_path):
    rng = np.random.default_rng(n + cut)
    piece = 128 * 1024
    widths = [max(1, (size + int(rng.integers(-40, 41))) // (3 * H)) for size in rng.choice([200, 4096, piece // 2, piece, 2 * piece, 3 * piece + 5000], n)]
    widths[-1] = 12000  # 288000 bytes, the last ones of the file
    samples = [rng.integers(0, 256, (H, w, 3), np.uint8) for w in widths]
    gaps = rng.integers(0, 3000, n)
    offsets = np.cumsum(np.concatenate([[0], [s.size for s in samples][:-1]]) + gaps).astype(np.uint64)
    data = np.zeros(int(offsets[-1]) + samples[-1].size, np.uint8)
    for s, at in zip(samples, offsets):
        data[int(at):int(at) + s.size] = s.reshape(-1)
    fd, direct = _open(kind, tmp_path, data[:data.size - cut])
    order = rng.permutation(n)
    params = np.zeros((n, 4), np.int32)
    for k in range(n):  # (a crop of whole rows' height: 8 columns out of each)
        params[k] = 0, int(rng.integers(0, max(widths[k] - 8, 0) + 1)), H, min(8, widths[k])
    params[-1] = 0, widths[-1] - 8, H, 8
    ctx = L.Context(0, 1, 4)
    out = ch.zeros((n, H, 8, 3), dtype=ch.uint8, device='cuda')
    stream = ch.cuda.current_stream().cuda_stream
    for _ in range(2):
        ctx.stage(0, (fd, direct if use_direct else -1), offsets[order], np.array([s.size for s in samples], np.uint64)[order], np.ones(n, np.uint8),
                  np.full(n, H, np.uint16), np.array(widths, np.uint16)[order], L.make_plan(H, 8, 1, L.OUT_U8_NHWC), np.ascontiguousarray(params[order]))
        ctx.submit(0, stream, out.data_ptr())
        status = ctx.status(0, stream, n)
    got = out.cpu().numpy()
    for row, k in enumerate(order):
        if k == n - 1 and cut:
            assert not got[row].any()  # (a raw sample that is not whole stays blank)
            continue
        assert status[row] == 0
        if widths[k] >= 8:
            r0, c0 = params[k, 0], params[k, 1]
            assert np.array_equal(got[row], samples[k][:, c0:c0 + 8]), k
    ctx.close()
    os.close(fd)
    if direct >= 0:
        os.close(direct)
