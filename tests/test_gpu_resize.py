"""The resize kernel's ways to its source pixels at the sizes where they change: windows filled from 4:2:0
and equal-resolution planes or from packed pixels, crops that begin and end anywhere in a unit of eight or
four pixels, at the image's edges, windows too small for a band, and bands that a translation moves."""
import cv2
import numpy as np
import pytest
import torch as ch

from ffcv_b200 import libffcv as L
from ffcv_b200.synthetic import synth_content
from parity import O

pytestmark = pytest.mark.gpu
FILL = (11, 22, 33)
OPS = {'plain': (), 'flip': ((L.OP_FLIP, 0, (0, 0, 0)),),
       'flip_translate_cutout': ((L.OP_FLIP, 0, (0, 0, 0)), (L.OP_TRANSLATE, 3, FILL), (L.OP_CUTOUT, 5, FILL))}


def _run(rng, images, crops, out_h, out_w, ops, kind):
    """images: (mode, height, width, payload).  Both results, as arrays of the output's bytes."""
    n = len(images)
    payloads = [p for _, _, _, p in images]
    modes = np.array([m for m, _, _, _ in images], np.uint8)
    heights, widths = (np.array([im[k] for im in images], np.uint16) for k in (1, 2))
    sizes = np.array([p.size for p in payloads], np.uint64)
    params = np.zeros((n, 4 + 2 * len(ops)), np.int32)
    params[:, :4] = crops
    records = []
    for i in range(n):
        rec = []
        for k, (typ, arg, fill) in enumerate(ops):
            a, b = (int(rng.integers(0, 2)), 0) if typ == L.OP_FLIP else \
                (rng.integers(0, 2 * arg + 1, 2) if typ == L.OP_TRANSLATE else (rng.integers(0, max(1, out_h - arg)), rng.integers(0, max(1, out_w - arg))))
            params[i, 4 + 2 * k:6 + 2 * k] = int(a), int(b)
            rec.append((typ, int(a), 0, 0, fill) if typ == L.OP_FLIP else (typ, arg, int(a), int(b), fill))
        records.append(rec)
    table = None if kind == L.OUT_U8_NHWC else O.normalize_table(np.array([100., 110, 120]), np.array([50., 60, 70]),
                                                                 np.float16 if kind in (L.OUT_F16_NHWC, L.OUT_F16_NCHW) else np.float32)
    want, status = O.run_batch(payloads, modes, heights, widths, params[:, :4], True, out_h, out_w, records, table, kind, 4)
    assert (status == 0).all()
    dtype = {L.OUT_U8_NHWC: ch.uint8, L.OUT_F16_NHWC: ch.int16, L.OUT_F16_NCHW: ch.int16}.get(kind, ch.int32)
    table_dev = ch.from_numpy(table.view(np.int16 if table.dtype == np.float16 else np.int32).copy()).cuda() if table is not None else None
    out = ch.zeros(want.size, dtype=dtype, device='cuda')
    ctx = L.Context(0, 1, 2)
    stream = ch.cuda.current_stream().cuda_stream
    ctx.stage(0, np.concatenate(payloads), np.concatenate([[0], np.cumsum(sizes)[:-1]]).astype(np.uint64), sizes, modes, heights, widths,
              L.make_plan(out_h, out_w, True, kind, ops, table_dev.data_ptr() if table is not None else 0), params)
    ctx.submit(0, stream, out.data_ptr())
    assert (ctx.status(0, stream, n) == 0).all()
    got = out.cpu().numpy()
    ctx.close()
    return got, np.ascontiguousarray(want).reshape(-1).view(got.dtype)


def _image(rng, h, w, form):
    pixels = synth_content(rng, h, w)
    if form == 'raw':
        return (1, h, w, np.ascontiguousarray(pixels).reshape(-1))
    flags = [cv2.IMWRITE_JPEG_QUALITY, 90, cv2.IMWRITE_JPEG_SAMPLING_FACTOR,
             {'420': cv2.IMWRITE_JPEG_SAMPLING_FACTOR_420, '444': cv2.IMWRITE_JPEG_SAMPLING_FACTOR_444, '422': cv2.IMWRITE_JPEG_SAMPLING_FACTOR_422}[form]]
    return (0, h, w, cv2.imencode('.jpg', np.ascontiguousarray(pixels[..., ::-1]), flags)[1].reshape(-1).copy())


@pytest.mark.parametrize('ops', list(OPS))
@pytest.mark.parametrize('kind', [L.OUT_U8_NHWC, L.OUT_F16_NCHW, L.OUT_F32_NHWC])
@pytest.mark.parametrize('out', [(23, 31), (64, 7), (40, 96)], ids=lambda o: f'{o[0]}x{o[1]}')
def test_crops_of_every_alignment(out, kind, ops):
    rng = np.random.default_rng(out[1] + kind)
    images, crops = [], []
    for form in ('420', '444', '422', 'raw'):
        for k in range(12):
            h, w = int(rng.integers(40, 90)), int(rng.integers(40, 90))
            ci, cj = int(rng.integers(0, 12)), k
            ch_, cw = (h - ci, w - cj) if k % 3 == 0 else (int(rng.integers(9, h - ci)), int(rng.integers(9, w - cj)))
            images.append(_image(rng, h, w, form))
            crops.append((ci, cj, ch_, cw))
    got, want = _run(rng, images, crops, *out, OPS[ops], kind)
    assert np.array_equal(got, want)


@pytest.mark.parametrize('form', ['420', '444', 'raw'])
@pytest.mark.parametrize('size', [(700, 900), (60, 2500), (2500, 60), (1, 700), (4, 5)], ids=lambda s: f'{s[0]}x{s[1]}')
def test_windows_of_every_size(size, form):
    """From a few rows of the whole image to more columns than a window takes."""
    rng = np.random.default_rng(size[0])
    h, w = size
    images = [_image(rng, h, w, form) for _ in range(3)]
    crops = [(0, 0, h, w), (h // 3, w // 3, h - h // 3, w - w // 3), (0, 0, max(1, h // 2), max(1, w // 2))]
    for out in ((224, 224), (17, 300), (300, 17), (5, 1100), (9, 1)):
        got, want = _run(rng, images, crops, *out, OPS['flip'], L.OUT_F16_NHWC)
        assert np.array_equal(got, want), out


@pytest.mark.parametrize('ops', ['flip', 'flip_translate_cutout'])
@pytest.mark.parametrize('kind', [L.OUT_U8_NHWC, L.OUT_F16_NCHW, L.OUT_F32_NHWC])
def test_crops_too_wide_for_a_window(kind, ops):
    """A column per thread: both ways to interpolate, odd and even outputs of one to very many columns, beside crops with
    a window."""
    rng = np.random.default_rng(kind)
    images = [_image(rng, h, w, form) for form in ('420', '444', '422', 'raw') for h, w in ((90, 2600), (41, 3001), (70, 80))]
    crops = [(k % 3, k, h - k % 3, w - k - 1) for k, (_, h, w, _) in enumerate(images)]
    for out in ((23, 31), (20, 224), (131, 150), (12, 513), (16, 10)):
        got, want = _run(rng, images, crops, *out, OPS[ops], kind)
        assert np.array_equal(got, want), out


@pytest.mark.parametrize('shape', [(340, 500), (341, 500), (400, 601), (511, 701), (1200, 1200)], ids=lambda s: f'{s[0]}x{s[1]}')
def test_regions_copied_by_all_threads(shape):
    """The reference's resize call with regions around and above the size from which all staging threads copy: whole
    images and regions whose rows begin and end anywhere."""
    h, w = shape
    img = np.random.default_rng(h).integers(0, 256, (h, w, 3), np.uint8)
    for r0, r1, c0, c1 in ((0, h, 0, w), (1, h, 3, w), (0, h - 2, 0, w - 1), (5, h - 3, 7, w - 6)):
        for out_h, out_w in ((100, 101), (r1 - r0, c1 - c0) if h < 512 else (411, 413)):
            got = np.zeros((out_h, out_w, 3), np.uint8)
            L.resize_crop(img, r0, r1, c0, c1, got)
            assert np.array_equal(got, O.resize_area(img, r0, r1, c0, c1, out_h, out_w))


def test_a_large_region_takes_no_longer_than_its_transfer():
    """2.7 MB against 0.3 MB, both down to 300x300: twice as long.  What the staging threads leave dirty in
    their caches made it eight times."""
    import time
    times = []
    for h, w in ((320, 300), (900, 1000)):
        img, out = np.random.default_rng(h).integers(0, 256, (h, w, 3), np.uint8), np.zeros((300, 300, 3), np.uint8)
        laps = []
        for _ in range(80):
            t = time.perf_counter()
            L.resize_crop(img, 0, h, 0, w, out)
            laps.append(time.perf_counter() - t)
        times.append(np.median(laps))
    assert times[1] < 5 * times[0], times
