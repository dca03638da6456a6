"""Riders on both sides of the size up to which they travel inside the resize kernel."""
import numpy as np
import pytest
import torch as ch

from ffcv_b200 import libffcv as L

pytestmark = pytest.mark.gpu
WORDS = 2048  # a batch's riders that the kernel copies itself, in words of 16, 4 or 1 bytes


def _batch(ctx, n, riders, out):
    rng = np.random.default_rng(n)
    pixels = rng.integers(0, 256, n * 16, np.uint8)
    pixels = np.concatenate([pixels] * 3)  # n images of 4x4
    ctx.set_riders(0, riders, n)
    ctx.stage(0, pixels, np.arange(n, dtype=np.uint64) * 48, np.full(n, 48, np.uint64), np.ones(n, np.uint8), np.full(n, 4, np.uint16),
              np.full(n, 4, np.uint16), L.make_plan(4, 4, 0, L.OUT_U8_NHWC), np.tile(np.array([0, 0, 4, 4], np.int32), (n, 1)))
    ctx.submit(0, ch.cuda.current_stream().cuda_stream, out.data_ptr())
    assert np.array_equal(out.cpu().numpy().reshape(-1), pixels)


@pytest.mark.parametrize('align', [16, 4, 1])
@pytest.mark.parametrize('beyond', [-WORDS + 1, -1, 0, 1, 3 * WORDS])
def test_riders_arrive_whole(align, beyond):
    """One rider of about the most that travels in the kernel, for destinations of every alignment, beside a small
    one before it and behind it; nothing around the destinations changes."""
    n = 3
    item = max(1, ((WORDS + beyond) * align + n - 1) // n - (1 if align > 1 else 0))  # (no multiple of a word)
    rng = np.random.default_rng(align * 10000 + beyond)
    values = [rng.integers(0, 256, (n, k), np.uint8) for k in (8, item, 5)]
    ctx = L.Context(0, 1, 2)
    out = ch.empty((n, 4, 4, 3), dtype=ch.uint8, device='cuda')
    buffers = [ch.full((v.size + 128,), 77, dtype=ch.uint8, device='cuda') for v in values]
    starts = [b.data_ptr() + 32 + (0 if align == 16 else align) for b in buffers]
    _batch(ctx, n, [(v, None, v.shape[1], p) for v, p in zip(values, starts)], out)
    for v, b, p in zip(values, buffers, starts):
        got, lead = b.cpu().numpy(), p - b.data_ptr()
        assert np.array_equal(got[lead:lead + v.size], v.reshape(-1))
        assert (got[:lead] == 77).all() and (got[lead + v.size:] == 77).all()
    ctx.close()


def test_large_riders_do_not_hold_the_batch_up():
    """16 MB of array values: microseconds of copying, not the milliseconds that one CTA takes."""
    n, item = 1024, 16000
    values = np.random.default_rng(1).integers(0, 256, (n, item), np.uint8)
    dst = ch.zeros((n, item), dtype=ch.uint8, device='cuda')
    out = ch.empty((n, 4, 4, 3), dtype=ch.uint8, device='cuda')
    ctx = L.Context(0, 1, 2)
    ctx.set_profiling(True)
    times = []
    for _ in range(5):
        _batch(ctx, n, [(values, None, item, dst.data_ptr())], out)
        times.append(ctx.batch_times(0)[4])
    assert np.array_equal(dst.cpu().numpy(), values)
    assert min(times) < 2.0, times  # ms; one CTA's bytewise copy took 20, the copy engine about 0.02
    ctx.close()
