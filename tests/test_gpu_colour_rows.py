"""Single images of every chroma layout at widths around a warp's row and at every alignment of their rows, in
host memory and behind the device copy: the colour kernels' ways to store a row."""
import cv2
import numpy as np
import pytest
import torch as ch

from ffcv_b200 import libffcv as L
from ffcv_b200.synthetic import synth_content
from parity import O

pytestmark = pytest.mark.gpu
SAMPLING = {'420': cv2.IMWRITE_JPEG_SAMPLING_FACTOR_420, '444': cv2.IMWRITE_JPEG_SAMPLING_FACTOR_444,
            '422': cv2.IMWRITE_JPEG_SAMPLING_FACTOR_422}


def _jpeg(h, w, form):
    img = synth_content(np.random.default_rng(h * 1000 + w), h, w)
    flags = [cv2.IMWRITE_JPEG_QUALITY, 85]
    if form == 'grey':
        return cv2.imencode('.jpg', img[..., 0], flags)[1].reshape(-1).copy()
    return cv2.imencode('.jpg', img, flags + [cv2.IMWRITE_JPEG_SAMPLING_FACTOR, SAMPLING[form]])[1].reshape(-1).copy()


@pytest.mark.parametrize('form', ['420', '444', '422', 'grey'])
@pytest.mark.parametrize('h,w', [(1, 1), (2, 3), (9, 4), (5, 31), (8, 32), (17, 33), (7, 127), (3, 128), (11, 129), (65, 254), (33, 257),
                                 (520, 383), (613, 700), (611, 701)], ids=str)
def test_rows_of_single_images(h, w, form):
    buf = _jpeg(h, w, form)
    out = np.full(h * w * 3 + 64, 7, np.uint8)  # nothing behind the image changes
    assert L.imdecode(buf, out, h, w) == 0
    want = O.jpeg_decode(buf)
    assert np.array_equal(out[:h * w * 3].reshape(h, w, 3), want) and (out[h * w * 3:] == 7).all()
    for shift in (1, 2, 3):  # scaled decodes go through the kernel of 4:4:4
        if form in ('420', '444') and h > 8:
            sh, sw = -(-h >> shift), -(-w >> shift)
            got = np.zeros((sh, sw, 3), np.uint8)
            assert L.imdecode(buf, got, h, w, scale_factor_num=1, scale_factor_denom=1 << shift) == 0
            assert np.array_equal(got, O.jpeg_decode_scaled(buf, 1 << shift))


@pytest.mark.parametrize('form', ['444', '422', 'grey'])
@pytest.mark.parametrize('offset', [0, 1, 2, 3])
def test_rows_that_begin_anywhere_on_the_gpu(form, offset):
    for h, w in ((19, 130), (8, 67), (40, 64)):
        buf = _jpeg(h, w, form)
        dev = ch.from_numpy(buf).cuda()
        out = ch.full((h * w * 3 + 64,), 7, dtype=ch.uint8, device='cuda')
        assert L.imdecode_static(buf, dev.data_ptr(), h, w, out.data_ptr() + 16 + offset) == 0
        ch.cuda.synchronize()
        got = out.cpu().numpy()
        assert np.array_equal(got[16 + offset:16 + offset + h * w * 3].reshape(h, w, 3), O.jpeg_decode(buf))
        assert (got[:16 + offset] == 7).all() and (got[16 + offset + h * w * 3:] == 7).all()


def test_odd_widths_cost_no_more_than_even_ones():
    """A call with a 4:4:4 image whose rows begin on no words, beside one whose rows do: single bytes
    stored into host memory made it 2.7 (224 columns) to 4 times as long."""
    import time
    times = []
    for w in (256, 253):
        buf, out = _jpeg(224, w, '444'), np.zeros((224, w, 3), np.uint8)
        laps = []
        for _ in range(60):
            t = time.perf_counter()
            assert L.imdecode(buf, out, 224, w) == 0
            laps.append(time.perf_counter() - t)
        times.append(min(laps))
    assert times[1] < 1.7 * times[0], times
