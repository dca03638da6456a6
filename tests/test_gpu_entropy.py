"""The entropy decoder's branches at the sizes where they change: one or several segments per scan,
one or four teams per CTA, the last CTA incomplete, Huffman tables its inner loop cannot use."""
import cv2
import numpy as np
import pytest
import torch as ch

from parity import O

pytestmark = pytest.mark.gpu


def _jpeg(rng, h, w, quality=90, sampling=420):
    from ffcv_b200.synthetic import synth_content
    flags = [cv2.IMWRITE_JPEG_QUALITY, quality]
    if sampling == 444:
        flags += [cv2.IMWRITE_JPEG_SAMPLING_FACTOR, cv2.IMWRITE_JPEG_SAMPLING_FACTOR_444]
    return cv2.imencode('.jpg', synth_content(rng, h, w)[..., ::-1], flags)[1].reshape(-1).copy()


def _decode(buf, h, w):
    from ffcv_b200.libffcv import imdecode
    out = np.zeros((h, w, 3), np.uint8)
    assert imdecode(buf, out, h, w) == 0
    return out


@pytest.mark.parametrize('sampling', [420, 444])
def test_scans_around_the_segment_length(sampling):
    # 128 subsequences of 256 bits are 4 KiB: scans of about one, two and three segments
    rng = np.random.default_rng(sampling)
    for h in range(60, 240, 9):
        w = h + int(rng.integers(0, 20))
        buf = _jpeg(rng, h, w, 90, sampling)
        assert np.array_equal(_decode(buf, h, w), O.jpeg_decode(buf)), (h, w, buf.size)


@pytest.mark.parametrize('n,mixed', [(739, False), (743, False), (743, True)], ids=['one_team', 'four_teams', 'tables_differ'])
@pytest.mark.parametrize('subseq_bits', ['', '512', '1280', '2560'], ids=['from_every_slot', 'repaired_on_the_spot', 'repaired_behind', 'longest'])
def test_batches_around_the_team_limit(n, mixed, subseq_bits, monkeypatch):
    """740 segments are where four teams start to share a CTA, when all scans use the same tables and, as these small
    batches only do when asked to, leave the repairs to the kernel behind.  Images with flat parts among them, whose
    subsequences have more blocks than is written down."""
    from ffcv_b200 import libffcv as L
    monkeypatch.setenv('FFCV_B200_SUBSEQ_BITS', subseq_bits)
    rng = np.random.default_rng(n + mixed)
    h, w = 40, 56
    bufs = [_jpeg(rng, h, w, int(rng.integers(60, 98)), 444 if mixed and k % 3 == 0 else 420) for k in range(n)]
    for k in range(7, n, 29):
        img = rng.integers(0, 256, (h, w, 3), np.uint8)
        img[16:] = 99
        bufs[k] = cv2.imencode('.jpg', img, [cv2.IMWRITE_JPEG_QUALITY, 95])[1].reshape(-1).copy()
    sizes = np.array([b.size for b in bufs], np.uint64)
    params = np.tile(np.array([0, 0, h, w], np.int32), (n, 1))
    ctx = L.Context(0, 1, 4)
    out = ch.zeros((n, h, w, 3), dtype=ch.uint8, device='cuda')
    stream = ch.cuda.current_stream().cuda_stream
    ctx.stage(0, np.concatenate(bufs), np.concatenate([[0], np.cumsum(sizes)[:-1]]).astype(np.uint64), sizes, np.zeros(n, np.uint8),
              np.full(n, h, np.uint16), np.full(n, w, np.uint16), L.make_plan(h, w, 0, L.OUT_U8_NHWC), params)
    ctx.submit(0, stream, out.data_ptr())
    assert (ctx.status(0, stream, n) == 0).all()
    got = out.cpu().numpy()
    for k, b in enumerate(bufs):
        assert np.array_equal(got[k], O.jpeg_decode(b)), k
    ctx.close()


def _grey_jpeg(rng, blocks_y, blocks_x, ac_lengths):
    """A greyscale baseline stream of random sparse blocks with the AC code lengths given as {symbol: length}."""
    def codes(lengths):
        order = sorted(lengths, key=lambda s: (lengths[s], s))
        out, code, prev = {}, 0, 0
        for s in order:
            code <<= lengths[s] - prev
            prev = lengths[s]
            out[s] = (code, prev)
            code += 1
        counts = [sum(1 for s in order if lengths[s] == n) for n in range(1, 17)]
        return out, bytes(counts) + bytes(order)
    dc, dc_seg = codes({s: 4 for s in range(12)})
    ac, ac_seg = codes(ac_lengths)
    bits = []

    def put(value, n):
        bits.extend((value >> k) & 1 for k in reversed(range(n)))

    def put_value(v):
        size = int(abs(v)).bit_length()
        put(v if v > 0 else v + (1 << size) - 1, size)
    dc_value = 0
    for _ in range(blocks_y * blocks_x):
        diff = int(rng.integers(-40, 41)) - dc_value
        dc_value += diff
        put(*dc[abs(diff).bit_length()])
        put_value(diff)
        z = 1
        while z < 64 and rng.random() < 0.9:
            run = int(rng.choice([0, 0, 0, 1, 2, 5, 20]))
            v = int(rng.choice([-1, 1])) * int(rng.integers(1, 1 << int(rng.integers(1, 8))))
            if z + run > 63:
                break
            while run > 15:
                put(*ac[0xF0])
                run -= 16
                z += 16
            put(*ac[run << 4 | abs(v).bit_length()])
            put_value(v)
            z += run + 1
        if z < 64:
            put(*ac[0])
    bits += [1] * (-len(bits) % 8)
    scan = np.packbits(np.array(bits, np.uint8)).tobytes().replace(b'\xff', b'\xff\x00')

    def segment(marker, body):
        return bytes([0xFF, marker]) + (len(body) + 2).to_bytes(2, 'big') + body
    h, w = 8 * blocks_y, 8 * blocks_x
    data = (b'\xff\xd8' + segment(0xDB, bytes([0]) + bytes(rng.integers(1, 20, 64).tolist())) +
            segment(0xC0, bytes([8]) + h.to_bytes(2, 'big') + w.to_bytes(2, 'big') + bytes([1, 1, 0x11, 0])) +
            segment(0xC4, bytes([0x00]) + dc_seg) + segment(0xC4, bytes([0x10]) + ac_seg) +
            segment(0xDA, bytes([1, 1, 0x00, 0, 63, 0])) + scan + b'\xff\xd9')
    return np.frombuffer(data, np.uint8).copy(), h, w


@pytest.mark.parametrize('long_length', [12, 16], ids=['codes_of_12_bits', 'codes_of_16_bits'])
@pytest.mark.parametrize('blocks', [(1, 1), (9, 7), (40, 33)])
def test_tables_whose_long_codes_come_early(blocks, long_length):
    """Three codes of 3 bits and all others of 12 or 16: long codes far from the end of the code space, more
    of them than there are second-level tables for."""
    lengths = {s: long_length for s in [0xF0] + [r << 4 | k for r in range(16) for k in range(1, 9)]}
    lengths.update({0x00: 3, 0x01: 3, 0x02: 3})
    buf, h, w = _grey_jpeg(np.random.default_rng(blocks[0] * 100 + long_length), *blocks, lengths)
    want = O.jpeg_decode(buf)
    assert np.abs(want.astype(int) - cv2.imdecode(buf, cv2.IMREAD_COLOR)).mean() < 6  # (cv2's accurate inverse transform)
    assert np.array_equal(_decode(buf, h, w), want)


@pytest.mark.parametrize('quality', [75, 98])
@pytest.mark.parametrize('h,w', [(33, 47), (256, 250), (531, 707), (1300, 1100)], ids=lambda v: str(v))
@pytest.mark.parametrize('subseq_bits', ['', '512'], ids=['from_every_slot', 'from_one_guess'])
def test_few_large_scans(h, w, quality, subseq_bits, monkeypatch):
    """Batches of few scans: one, several and (for the run that follows the real state) very many segments,
    photographs and pure noise, whose blocks are longer than a subsequence."""
    from ffcv_b200 import libffcv as L
    monkeypatch.setenv('FFCV_B200_SUBSEQ_BITS', subseq_bits)
    rng = np.random.default_rng(h + quality)
    bufs = [_jpeg(rng, h, w, quality), cv2.imencode('.jpg', rng.integers(0, 256, (h, w, 3), np.uint8), [cv2.IMWRITE_JPEG_QUALITY, quality])[1].reshape(-1)]
    n = len(bufs)
    sizes = np.array([b.size for b in bufs], np.uint64)
    ctx = L.Context(0, 1, 2)
    out = ch.zeros((n, h, w, 3), dtype=ch.uint8, device='cuda')
    stream = ch.cuda.current_stream().cuda_stream
    ctx.stage(0, np.concatenate(bufs), np.concatenate([[0], np.cumsum(sizes)[:-1]]).astype(np.uint64), sizes, np.zeros(n, np.uint8),
              np.full(n, h, np.uint16), np.full(n, w, np.uint16), L.make_plan(h, w, 0, L.OUT_U8_NHWC),
              np.tile(np.array([0, 0, h, w], np.int32), (n, 1)))
    ctx.submit(0, stream, out.data_ptr())
    assert (ctx.status(0, stream, n) == 0).all()
    got = out.cpu().numpy()
    for k, b in enumerate(bufs):
        assert np.array_equal(got[k], O.jpeg_decode(b)), k
    ctx.close()


@pytest.mark.parametrize('n', [1, 2, 296, 297])
def test_batches_whose_kernels_begin_early(n):
    """Up to 296 segments every kernel is launched while the one before runs.  Both ways of decoding in a batch,
    and batches behind one another in the same slot and buffers."""
    from ffcv_b200 import libffcv as L
    rng = np.random.default_rng(n)
    h, w = 40, 56
    ctx = L.Context(0, 1, 2)
    stream = ch.cuda.current_stream().cuda_stream
    outs, wants = [], []
    for b in range(4):
        bufs = [_jpeg(rng, h, w, int(rng.integers(60, 98)), 444 if k % 3 == 1 else 420) for k in range(n)]
        sizes = np.array([b.size for b in bufs], np.uint64)
        outs.append(ch.zeros((n, h, w, 3), dtype=ch.uint8, device='cuda'))
        ctx.stage(0, np.concatenate(bufs), np.concatenate([[0], np.cumsum(sizes)[:-1]]).astype(np.uint64), sizes, np.zeros(n, np.uint8),
                  np.full(n, h, np.uint16), np.full(n, w, np.uint16), L.make_plan(h, w, 0, L.OUT_U8_NHWC),
                  np.tile(np.array([0, 0, h, w], np.int32), (n, 1)))
        ctx.submit(0, stream, outs[-1].data_ptr())
        wants.append(np.stack([O.jpeg_decode(b) for b in bufs]))
    assert (ctx.status(0, stream, n) == 0).all()
    for got, want in zip(outs, wants):
        assert np.array_equal(got.cpu().numpy(), want)
    ctx.close()


def _grey_noise(rng, h, w, quality=90):
    """A scan that decoders fall in step with slowly: of its subsequences of 600 to 2000 bits some 85 in a hundred are decoded
    wrongly after the run-up, up to 30 in a row."""
    img = np.repeat(rng.integers(0, 256, (h, w, 1), np.uint8), 3, 2)
    return cv2.imencode('.jpg', img, [cv2.IMWRITE_JPEG_QUALITY, quality])[1].reshape(-1).copy()


def _stage_and_check(bufs, h, w):
    """One batch of JPEG streams of one shape, decoded whole."""
    from ffcv_b200 import libffcv as L
    n = len(bufs)
    want = {id(b): O.jpeg_decode(b) for b in {id(b): b for b in bufs}.values()}
    sizes = np.array([b.size for b in bufs], np.uint64)
    ctx = L.Context(0, 1, 4)
    out = ch.zeros((n, h, w, 3), dtype=ch.uint8, device='cuda')
    stream = ch.cuda.current_stream().cuda_stream
    ctx.stage(0, np.concatenate(bufs), np.concatenate([[0], np.cumsum(sizes)[:-1]]).astype(np.uint64), sizes, np.zeros(n, np.uint8),
              np.full(n, h, np.uint16), np.full(n, w, np.uint16), L.make_plan(h, w, 0, L.OUT_U8_NHWC),
              np.tile(np.array([0, 0, h, w], np.int32), (n, 1)))
    ctx.submit(0, stream, out.data_ptr())
    assert (ctx.status(0, stream, n) == 0).all()
    got = out.cpu().numpy()
    for k, b in enumerate(bufs):
        assert np.array_equal(got[k], want[id(b)]), k
    ctx.close()


@pytest.mark.parametrize('records', ['', '0'], ids=['written_down', 'nothing_written_down'])
@pytest.mark.parametrize('subseq_bits', [128, 512, 2560])
@pytest.mark.parametrize('sampling', [420, 444])
def test_subsequences_of_very_many_blocks(subseq_bits, sampling, records, monkeypatch):
    """Flat images: a subsequence holds up to 500 blocks; flat and busy parts in one scan, whose flat subsequences have
    more blocks than there is room to write down, beside others in one warp."""
    monkeypatch.setenv('FFCV_B200_SUBSEQ_BITS', str(subseq_bits))
    monkeypatch.setenv('FFCV_B200_RECORDS_MB', records)
    rng = np.random.default_rng(subseq_bits + sampling)
    h, w = 640, 560
    flat = np.full((h, w, 3), 117, np.uint8)
    half = flat.copy()
    half[200:330] = rng.integers(0, 256, (130, w, 3))
    ramp = np.clip(np.arange(w)[None, :, None] // 9 + np.zeros((h, 1, 3)) + rng.integers(0, 2, (h, w, 3)), 0, 255).astype(np.uint8)
    flags = [cv2.IMWRITE_JPEG_QUALITY, 85]
    if sampling == 444:
        flags += [cv2.IMWRITE_JPEG_SAMPLING_FACTOR, cv2.IMWRITE_JPEG_SAMPLING_FACTOR_444]
    bufs = [cv2.imencode('.jpg', im, flags)[1].reshape(-1).copy() for im in (flat, half, ramp)]
    _stage_and_check(bufs, h, w)


@pytest.mark.parametrize('records', ['', '0'], ids=['written_down', 'nothing_written_down'])
@pytest.mark.parametrize('n', [255, 256, 517, 1030])
def test_images_that_share_a_repair(n, records, monkeypatch):
    """From 256, 512 and 1024 images of the same tables on, two, four and eight of them are repaired by one CTA, here in
    some 30 rounds; the lists of eight (160 subsequences in doubt each, in three segments) are longer than there is room for."""
    monkeypatch.setenv('FFCV_B200_SUBSEQ_BITS', '1280')
    monkeypatch.setenv('FFCV_B200_RECORDS_MB', records)
    rng = np.random.default_rng(n)
    h, w = 192, 192
    few = [_grey_noise(rng, h, w, int(rng.integers(84, 94))) for _ in range(24)]
    few += [cv2.imencode('.jpg', rng.integers(0, 256, (h, w, 3), np.uint8))[1].reshape(-1).copy(), _jpeg(rng, h, w), _jpeg(rng, h, w, 20)]
    _stage_and_check([few[int(rng.integers(0, len(few)))] for _ in range(n)], h, w)


@pytest.mark.parametrize('subseq_bits', ['1280', '2560'])
def test_long_scans_repaired_in_parts(subseq_bits, monkeypatch):
    """Scans of more than 64 segments: parts of 32 of them side by side, each with some 1700 subsequences in doubt at
    once, then their seams."""
    monkeypatch.setenv('FFCV_B200_SUBSEQ_BITS', subseq_bits)
    rng = np.random.default_rng(int(subseq_bits))
    h, w = 1480, 1320
    text = np.full((h, w, 3), 245, np.uint8)
    for y in range(10, h - 12, 16):
        text[y:y + 9, 12:900] = np.where(rng.random((9, 888, 1)) < 0.3, 30, 245)
    _stage_and_check([_grey_noise(rng, h, w), cv2.imencode('.jpg', text, [cv2.IMWRITE_JPEG_QUALITY, 90])[1].reshape(-1).copy()], h, w)
