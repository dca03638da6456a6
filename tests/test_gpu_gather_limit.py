"""A payload gather whose wait for the link runs out: the batch is flagged, blank and reported, and the context
goes on.  (A limit of 0: no piece has arrived when it is first looked for.)"""
import cv2
import numpy as np
import pytest
import torch as ch

from ffcv_b200 import libffcv as L
from ffcv_b200.synthetic import synth_content
from parity import IMAGENET_MEAN, IMAGENET_STD, O, image_executor

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('restart', [0, 4], ids=['segments', 'restart_markers'])
def test_a_gather_that_gives_up_is_reported(monkeypatch, restart):
    rng = np.random.default_rng(restart)
    h, w, out_size = 72, 88, 40
    payloads, modes = [], []
    for k in range(8):
        img = synth_content(rng, h, w)
        modes.append(k % 2)
        flags = [cv2.IMWRITE_JPEG_QUALITY, 90, cv2.IMWRITE_JPEG_RST_INTERVAL, restart]
        payloads.append(img.reshape(-1) if k % 2 else cv2.imencode('.jpg', img, flags)[1].reshape(-1))
    n = len(payloads)
    sizes = np.array([p.size for p in payloads], np.uint64)
    ptrs = np.concatenate([[0], np.cumsum(sizes)[:-1]]).astype(np.uint64)
    order = np.array([0, 5, 2, 7, 4, 1, 6, 3])  # (neighbours would be one copy, no gather)
    pageable = np.concatenate(payloads)
    pinned = ch.from_numpy(pageable).pin_memory()
    params = np.tile(np.array([3, 5, 60, 70], np.int32), (n, 1))
    plan = L.make_plan(out_size, out_size, 1, L.OUT_U8_NHWC)
    args = (ptrs[order], sizes[order], np.array(modes, np.uint8)[order], np.full(n, h, np.uint16), np.full(n, w, np.uint16), plan, params)
    want, _ = O.run_batch([payloads[k] for k in order], args[2], args[3], args[4], params, True, out_size, out_size, [[] for _ in range(n)],
                          None, L.OUT_U8_NHWC, 2)
    stream = ch.cuda.current_stream().cuda_stream

    def run(ctx, base):
        out = ch.full((n, out_size, out_size, 3), 9, dtype=ch.uint8, device='cuda')
        ctx.stage(0, base, *args)
        ctx.submit(0, stream, out.data_ptr())
        return ctx.status(0, stream, n), out.cpu().numpy()

    good = L.Context(0, 1, 2)
    status, got = run(good, pinned.data_ptr())
    assert (status == 0).all() and np.array_equal(got, want)
    assert good.gather_time(0) is not None
    good.check()
    good.close()

    monkeypatch.setenv('FFCV_B200_GATHER_LIMIT_MS', '0')
    ctx = L.Context(0, 1, 2)
    status, got = run(ctx, pageable)  # no gather
    assert (status == 0).all() and np.array_equal(got, want)
    status, got = run(ctx, pinned.data_ptr())
    assert (status != 0).all() and (got == 0).all()
    with pytest.raises(L.FFCVBError, match='did not arrive in time'):
        ctx.check()
    ctx.check()
    status, got = run(ctx, pinned.data_ptr())
    assert (status != 0).all()
    ctx.stage(0, pageable, *args)
    with pytest.raises(L.FFCVBError, match='did not arrive in time'):
        ctx.submit(0, stream, ch.empty(want.shape, dtype=ch.uint8, device='cuda').data_ptr())
    status, got = run(ctx, pageable)
    assert (status == 0).all() and np.array_equal(got, want)
    ctx.close()


def test_the_loader_reports_it(monkeypatch, tmp_path):
    """By the next batch, or, for the last ones of an epoch, when the epoch ends or the next one begins."""
    from ffcv_b200 import Loader, OrderOption
    from ffcv_b200.fields.decoders import RandomResizedCropRGBImageDecoder
    from ffcv_b200.synthetic import write_dataset_isolated
    from ffcv_b200.transforms import NormalizeImage, ToTorchImage
    path = write_dataset_isolated(1, str(tmp_path / 'c1.beton'), 96, num_workers=2)
    pipes = {'image': [RandomResizedCropRGBImageDecoder((64, 64)), ToTorchImage(), NormalizeImage(IMAGENET_MEAN, IMAGENET_STD, np.float16)],
             'label': None}
    monkeypatch.setenv('FFCV_B200_GATHER_LIMIT_MS', '0')
    loader = Loader(path, batch_size=32, order=OrderOption.RANDOM, seed=0, num_workers=2, pin_file=True, cpu_stage_share=0.0,
                    indices=np.arange(0, 96, 3), pipelines=pipes)  # one batch, of samples that are no neighbours
    assert loader.memory_manager.pinned
    it = iter(loader)
    next(it)
    ch.cuda.synchronize()
    assert (image_executor(loader).ctx.status(0, ch.cuda.current_stream().cuda_stream, 32) != 0).all()
    with pytest.raises(L.FFCVBError, match='did not arrive in time'):
        next(it)
    it = iter(loader)  # the failure has been told: the epoch begins
    next(it)
    ch.cuda.synchronize()
    with pytest.raises(L.FFCVBError, match='did not arrive in time'):
        for _ in loader:
            pass
