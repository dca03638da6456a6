"""The payload gather cuts what it fetches at multiples of 128 bytes of the source: crop rows that begin at every
place inside such a line, of lengths on both sides of one piece and of two, and streams likewise."""
import cv2
import numpy as np
import pytest
import torch as ch

from ffcv_b200 import libffcv as L
from ffcv_b200.synthetic import synth_content
from parity import O

pytestmark = pytest.mark.gpu


def gathered(payloads, modes, hs, ws, params, out_h, out_w):
    """The batch from page-locked memory, the payload of sample k at k mod 128, samples out of order."""
    n = len(payloads)
    sizes = np.array([p.size for p in payloads], np.uint64)
    room = int(sizes.max()) + 256 & ~127
    ptrs = (np.arange(n) * room + np.arange(n) % 128).astype(np.uint64)
    pinned = ch.zeros(n * room, dtype=ch.uint8).pin_memory()
    for p, at in zip(payloads, ptrs):
        pinned[int(at):int(at) + p.size] = ch.from_numpy(p)
    order = np.random.default_rng(n).permutation(n)
    ctx = L.Context(0, 1, 2)
    out = ch.zeros((n, out_h, out_w, 3), dtype=ch.uint8, device='cuda')
    stream = ch.cuda.current_stream().cuda_stream
    ctx.stage(0, pinned.data_ptr(), ptrs[order], sizes[order], modes[order], hs[order], ws[order], L.make_plan(out_h, out_w, 1, L.OUT_U8_NHWC),
              np.ascontiguousarray(params[order]))
    ctx.submit(0, stream, out.data_ptr())
    assert (ctx.status(0, stream, n) == 0).all() and ctx.gather_time(0) is not None
    ctx.close()
    got = np.empty((n, out_h, out_w, 3), np.uint8)
    got[order] = out.cpu().numpy()
    return got


@pytest.mark.parametrize('cols', [1, 5, 42, 43, 300, 341, 342, 384, 683, 725])
def test_rows_of_every_alignment(cols):
    n, rows = 128, 3
    rng = np.random.default_rng(cols)
    images = rng.integers(0, 256, (n, rows + 2, cols + 7, 3), dtype=np.uint8)
    at = rng.integers(0, (3, 8), (n, 2))
    params = np.concatenate([at, np.tile([rows, cols], (n, 1))], 1).astype(np.int32)
    got = gathered([im.reshape(-1) for im in images], np.ones(n, np.uint8), np.full(n, rows + 2, np.uint16), np.full(n, cols + 7, np.uint16), params,
                   rows, cols)
    for k in range(n):
        assert np.array_equal(got[k], images[k, at[k, 0]:at[k, 0] + rows, at[k, 1]:at[k, 1] + cols]), k


def test_streams_of_every_alignment():
    n, out_size = 128, 24
    rng = np.random.default_rng(0)
    hs, ws = rng.integers(16, 90, n).astype(np.uint16), rng.integers(16, 90, n).astype(np.uint16)
    payloads = [cv2.imencode('.jpg', synth_content(rng, int(h), int(w)), [cv2.IMWRITE_JPEG_QUALITY, 90])[1].reshape(-1) for h, w in zip(hs, ws)]
    params = np.stack([0 * hs, 0 * ws, hs, ws], 1).astype(np.int32)
    modes = np.zeros(n, np.uint8)
    want, _ = O.run_batch(payloads, modes, hs, ws, params, True, out_size, out_size, [[] for _ in range(n)], None, L.OUT_U8_NHWC, 2)
    assert np.array_equal(gathered(payloads, modes, hs, ws, params, out_size, out_size), want)


@pytest.mark.parametrize('ctas', [1, 7, 148, 1024])
@pytest.mark.parametrize('n', [1, 3, 40])
def test_samples_shared_out_to_any_number_of_ctas(ctas, n, monkeypatch):
    """More CTAs than lines, one CTA for all, shares that begin and end inside rows' and streams' samples, samples of
    less than a line among large ones."""
    monkeypatch.setenv('FFCV_B200_GATHER_CTAS', str(ctas))
    rng = np.random.default_rng(100 * ctas + n)
    payloads, modes, hs, ws, params, wants = [], [], [], [], [], []
    for k in range(n):
        h, w = (2, 3) if k % 4 == 0 and n > 1 else (int(v) for v in rng.integers(20, 260, 2))
        img = synth_content(rng, h, w)
        raw = k % 3 != 1
        payloads.append(img.reshape(-1) if raw else cv2.imencode('.jpg', img[..., ::-1], [cv2.IMWRITE_JPEG_QUALITY, 95])[1].reshape(-1).copy())
        ch_, cw_ = int(rng.integers(1, h + 1)), int(rng.integers(1, w + 1))
        r0, c0 = int(rng.integers(0, h - ch_ + 1)), int(rng.integers(0, w - cw_ + 1))
        modes.append(int(raw))
        hs.append(h)
        ws.append(w)
        params.append((r0, c0, ch_, cw_))
        pixels = img if raw else O.jpeg_decode(payloads[-1])
        wants.append(O.resize_area(pixels, r0, r0 + ch_, c0, c0 + cw_, 24, 24))
    got = gathered(payloads, np.array(modes, np.uint8), np.array(hs, np.uint16), np.array(ws, np.uint16), np.array(params, np.int32), 24, 24)
    assert np.array_equal(got, np.stack(wants))
