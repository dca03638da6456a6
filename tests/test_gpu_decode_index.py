"""The decode index with batches of several slots under way at once."""
import cv2
import numpy as np
import pytest
import torch as ch

from ffcv_b200 import libffcv as L
from ffcv_b200.synthetic import synth_content
from parity import O

pytestmark = pytest.mark.gpu


class _Job:
    def __init__(self, n, h, w, bufs=None):
        rng = np.random.default_rng(n)
        bufs = bufs or [cv2.imencode('.jpg', synth_content(rng, h, w), [cv2.IMWRITE_JPEG_QUALITY, 90])[1].reshape(-1) for _ in range(n)]
        self.want = np.stack([O.jpeg_decode(b) for b in bufs])
        sizes = np.array([b.size for b in bufs], np.uint64)
        self.args = (np.concatenate(bufs), np.concatenate([[0], np.cumsum(sizes)[:-1]]).astype(np.uint64), sizes, np.zeros(n, np.uint8),
                     np.full(n, h, np.uint16), np.full(n, w, np.uint16), L.make_plan(h, w, 0, L.OUT_U8_NHWC),
                     np.tile(np.array([0, 0, h, w], np.int32), (n, 1)))

    def queue(self, ctx, slot, stream):
        out = ch.zeros(self.want.shape, dtype=ch.uint8, device='cuda')
        ch.cuda.current_stream().synchronize()
        ctx.stage(slot, *self.args)
        ctx.submit(slot, stream.cuda_stream, out.data_ptr())
        return out


def test_entries_are_handed_out_when_their_writer_has_ended():
    """Slot 0's batch, which writes the entries, waits behind other work of its stream; the batches that slot 1
    decodes meanwhile neither read nor write them."""
    job, n = _Job(6, 120, 144), 6
    ctx = L.Context(0, 2, 2)
    ctx.set_decode_index(1 << 20)
    held, free = ch.cuda.Stream(), ch.cuda.Stream()
    job.queue(ctx, 1, free)  # scratch of both slots is there: nothing below allocates and waits for the device
    job.queue(ctx, 0, free)
    ch.cuda.synchronize()
    ctx.set_decode_index(1 << 20)  # empty again
    with ch.cuda.stream(held):
        ch.cuda._sleep(1 << 30)  # about half a second
    first = job.queue(ctx, 0, held)
    for _ in range(4):
        out = job.queue(ctx, 1, free)
        free.synchronize()
        assert np.array_equal(out.cpu().numpy(), job.want)
        stats = ctx.decode_index_stats()
        assert not held.query(), 'the held batch ran too early for this test'
        assert (stats['used'], stats['recorded'], stats['entries']) == (0, 0, n)
    held.synchronize()
    assert np.array_equal(first.cpu().numpy(), job.want)
    assert ctx.decode_index_stats()['recorded'] == n
    out = job.queue(ctx, 1, free)
    free.synchronize()
    assert np.array_equal(out.cpu().numpy(), job.want)
    assert ctx.decode_index_stats()['used'] == n
    ctx.close()


def test_a_batch_staged_before_the_index_was_set_up_again_leaves_it_alone():
    job, n = _Job(3, 64, 80), 3
    ctx = L.Context(0, 1, 2)
    ctx.set_decode_index(1 << 20)
    stream = ch.cuda.Stream()
    for again in (1 << 20, 0):
        out = ch.zeros(job.want.shape, dtype=ch.uint8, device='cuda')
        ch.cuda.synchronize()
        ctx.stage(0, *job.args)
        ctx.set_decode_index(again)
        ctx.submit(0, stream.cuda_stream, out.data_ptr())
        ch.cuda.synchronize()
        assert np.array_equal(out.cpu().numpy(), job.want)
        assert ctx.decode_index_stats()['recorded'] == 0
    ctx.set_decode_index(1 << 20)
    for use in (0, n):
        out = job.queue(ctx, 0, stream)
        ch.cuda.synchronize()
        assert np.array_equal(out.cpu().numpy(), job.want)
        assert ctx.decode_index_stats()['used'] == use
    ctx.close()


@pytest.mark.parametrize('subseq_bits', ['', '128', '2560'])
def test_an_entry_takes_four_bytes_per_subsequence(subseq_bits, monkeypatch):
    """Large streams, whose segments are full but for the last one: a word per subsequence of 1024 bits (or of as many
    as are asked for), a header of 16 bytes and, at most, a segment of 128 words that is nearly empty."""
    monkeypatch.setenv('FFCV_B200_SUBSEQ_BITS', subseq_bits)
    rng = np.random.default_rng(0)
    bufs = [cv2.imencode('.jpg', synth_content(rng, 700, 900), [cv2.IMWRITE_JPEG_QUALITY, q])[1].reshape(-1) for q in (60, 85, 97)]
    bits, n = sum(8 * b.size for b in bufs), len(bufs)
    job = _Job(n, 700, 900, bufs)
    ctx, stream = L.Context(0, 1, 2), ch.cuda.Stream()
    ctx.set_decode_index(1 << 24)
    for _ in range(3):
        out = job.queue(ctx, 0, stream)
        stream.synchronize()
        assert np.array_equal(out.cpu().numpy(), job.want)
    stats = ctx.decode_index_stats()
    assert (stats['used'], stats['recorded'], stats['entries']) == (2 * n, n, n)
    assert stats['bytes'] <= 4 * bits / int(subseq_bits or 1024) * 33 / 32 + n * (16 + 4 * 128)  # (lengths are multiples of 32 bits)
    ctx.close()
