"""Colour jitter, mixup and normalisation as one chain against the oracle's single steps."""
import numpy as np
import pytest
import torch as ch

from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('shape', [(1, 1, 1), (3, 5, 7), (5, 16, 20), (4, 61, 64), (2, 192, 192)], ids=str)
@pytest.mark.parametrize('kinds', [(), (1,), (0, 1, 2), (2, 1, 0, 1)], ids=str)
@pytest.mark.parametrize('out_size,mix', [(1, False), (1, True), (2, True), (4, False), (4, True)])
def test_pixel_chain(shape, kinds, out_size, mix):
    from ffcv_b200 import libffcv as L
    n, h, w = shape
    rng = np.random.default_rng(n * 1000 + h + len(kinds))
    imgs = rng.integers(0, 256, (n, h, w, 3), dtype=np.uint8)
    apply = (rng.random((len(kinds), n)) < 0.7).astype(np.uint8)
    ratio = rng.uniform(0.0, 2.5, (len(kinds), n))
    if len(kinds):
        ratio[0, 0] = 3e7  # far outside what a byte can hold
    lam = rng.beta(0.5, 0.5, n) if mix else None
    table = O.normalize_table(np.array([123.7, 116.3, 103.5]), np.array([58.4, 57.1, 57.4]), {1: np.float16, 2: np.float16, 4: np.float32}[out_size])
    want = imgs
    for k, kind in enumerate(kinds):
        want = O.color_jitter(want, kind, apply[k].astype(bool), ratio[k])
    if mix:
        want = O.mixup(want, lam)
    if out_size > 1:
        want = table[want, np.arange(3)]
    ctx = L.Context(0, 1, 1)
    src = ch.from_numpy(imgs).cuda()
    lut = ch.from_numpy(table.view(np.int16 if out_size < 4 else np.int32)).cuda()
    dst = ch.zeros((n, h, w, 3), dtype={1: ch.uint8, 2: ch.float16, 4: ch.float32}[out_size], device='cuda')
    ctx.pixel_chain(ch.cuda.current_stream().cuda_stream, src.data_ptr(), n, h * w, np.array(kinds, np.int32), apply, ratio, lam,
                    out_size, lut.data_ptr(), dst.data_ptr())
    got = dst.cpu().numpy()
    assert got.tobytes() == np.ascontiguousarray(want).tobytes()
    ctx.close()


@pytest.mark.parametrize('n,count', [(1, 1), (3, 7), (2, 1000)])
def test_mixup_of_values_that_are_no_pixels(n, count):
    from ffcv_b200 import libffcv as L
    rng = np.random.default_rng(count)
    imgs = rng.integers(0, 256, (n, count), dtype=np.uint8)
    lam = rng.random(n)
    src, dst = ch.from_numpy(imgs).cuda(), ch.zeros((n, count), dtype=ch.uint8, device='cuda')
    ctx = L.Context(0, 1, 1)
    ctx.mixup(ch.cuda.current_stream().cuda_stream, src.data_ptr(), dst.data_ptr(), n, count, lam)
    assert np.array_equal(dst.cpu().numpy(), O.mixup(imgs.reshape(n, 1, count, 1), lam).reshape(n, count))
    ctx.close()


def test_threads_share_a_context():
    """Two loaders' threads call the process-wide context at once, each on a stream of its own."""
    import threading
    from ffcv_b200 import libffcv as L
    ctx = L.Context(0, 1, 1)
    wrong = []

    def work(seed):
        rng = np.random.default_rng(seed)
        stream = ch.cuda.Stream()
        for round_ in range(60):
            n, h, w = int(rng.integers(1, 200)), 4, 5
            imgs = rng.integers(0, 256, (n, h, w, 3), dtype=np.uint8)
            lam, apply, ratio = rng.random(n), (rng.random((1, n)) < 0.5).astype(np.uint8), rng.uniform(0.5, 1.5, (1, n))
            with ch.cuda.stream(stream):
                src = ch.from_numpy(imgs).cuda()
                outs = [ch.empty_like(src) for _ in range(20)]
                for out in outs:
                    ctx.pixel_chain(stream.cuda_stream, src.data_ptr(), n, h * w, np.zeros(1, np.int32), apply, ratio, lam, 1, 0, out.data_ptr())
                stream.synchronize()
            want = O.mixup(O.color_jitter(imgs, 0, apply[0].astype(bool), ratio[0]), lam)
            if not all(np.array_equal(out.cpu().numpy(), want) for out in outs):
                wrong.append((seed, round_))
    threads = [threading.Thread(target=work, args=(seed,)) for seed in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong
    ctx.close()


@pytest.mark.parametrize('kind', [0, 1, 2])
@pytest.mark.parametrize('shape', [(1, 1, 1), (5, 3, 7), (3, 16, 20), (130, 8, 8)], ids=str)
def test_one_operation_in_place(shape, kind):
    """A jitter alone has a kernel of its own: words and single pixels, factors far outside a byte's range, images that
    are left alone."""
    from ffcv_b200 import libffcv as L
    n, h, w = shape
    rng = np.random.default_rng(n + kind)
    imgs = rng.integers(0, 256, (n, h, w, 3), dtype=np.uint8)
    apply, ratio = (rng.random(n) < 0.6).astype(np.uint8), rng.uniform(0.0, 2.5, n)
    apply[0], ratio[0] = 1, 3e7
    if n > 1:
        apply[1], ratio[1] = 1, -4.0
    ctx = L.Context(0, 1, 1)
    dev = ch.from_numpy(imgs).cuda()
    ctx.color_jitter(ch.cuda.current_stream().cuda_stream, dev.data_ptr(), n, h, w, kind, apply, ratio)
    assert np.array_equal(dev.cpu().numpy(), O.color_jitter(imgs, kind, apply.astype(bool), ratio))
    ctx.close()
