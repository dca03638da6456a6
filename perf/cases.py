"""The work this framework is used for, as measurable cases.

A case is one of four uses of the public interface:

* ``loader``    one epoch of a few batches through ``Loader`` over a ``.beton`` in memory, which is
                what a training or validation script does: bytes of the stored samples go to the GPU,
                are decoded, cropped, resized, augmented and normalised there;
* ``serve``     one batch of JPEG requests in host memory through ``Context.stage`` / ``submit`` (what
                a server built on the C ABI does), result on the GPU;
* ``imdecode``  one JPEG, host buffer to host buffer, with the reference's single-image call;
* ``resize``    one INTER_AREA crop-and-resize, host buffer to host buffer, likewise.

Everything a case computes is integer arithmetic, or fp32 / fp64 arithmetic whose rounding is fixed
by the format it reproduces, so the outputs are compared bit for bit.

Images are seeded smooth fields (eight sinusoids per channel) with Gaussian noise of sigma 8, the
content of the benchmark's datasets: JPEG files of it have photographic sizes.
"""
import gc
import math
import os
from concurrent.futures import ThreadPoolExecutor

import numpy as np
import torch

from ffcv_b200 import Loader, OrderOption
from ffcv_b200 import libffcv as L
from ffcv_b200.fields import IntField, RGBImageField
from ffcv_b200.fields.decoders import (CenterCropRGBImageDecoder, IntDecoder, RandomResizedCropRGBImageDecoder,
                                       SimpleRGBImageDecoder)
from ffcv_b200.synthetic import make_field
from ffcv_b200.transforms import (Cutout, ImageMixup, LabelMixup, MixupToOneHot, NormalizeImage, RandomBrightness,
                                  RandomContrast, RandomHorizontalFlip, RandomSaturation, RandomTranslate, Squeeze,
                                  ToDevice, ToTensor, ToTorchImage)
from ffcv_b200.writer import DatasetWriter

MEAN = np.array([0.485, 0.456, 0.406]) * 255
STD = np.array([0.229, 0.224, 0.225]) * 255
FILL = (125, 123, 114)
CLASSES = 1000
DTYPES = {'f16': np.float16, 'f32': np.float32}

# JPEG bytes per pixel of the images made here, by (chroma sampling, quality).
JPEG_DENSITY = {(420, 80): 0.16, (420, 85): 0.21, (420, 90): 0.29, (420, 95): 0.48,
                (444, 80): 0.23, (444, 85): 0.32, (444, 90): 0.55, (444, 95): 0.95}


def _loader_case(name=None, **kw):
    case = dict(kind='loader', batch=256, batches=4, batches_ahead=3, mode='jpg', quality=90, sampling=420,
                short_lo=300, short_hi=500, max_side=0, decoder='rrc', scale_lo=0.08, out_h=224, out_w=224,
                ops='flip', colour=False, dtype='f16', channels_last=True, order='random', os_cache=True)
    case.update(kw)
    if name is not None:
        case['name'] = name
    return case


def listed():
    return [
        # one small photo through the reference's decode call: latency and launches
        dict(name='imdecode_224x256', kind='imdecode', height=224, width=256, quality=90, sampling=420),
        # one camera-sized 4:2:0 photo, sides that are no multiples of an MCU
        dict(name='imdecode_1213x1617', kind='imdecode', height=1213, width=1617, quality=90, sampling=420),
        # one large archival image: 4:4:4, quality 95
        dict(name='imdecode_1536x2048_444', kind='imdecode', height=1536, width=2048, quality=95, sampling=444),
        # one crop of a decoded image resized by the reference's resize call
        dict(name='resize_320x300_to_224', kind='resize', height=400, width=500, crop_h=320, crop_w=300, out_h=224,
             out_w=224),
        # an inference server's batch of uploads, planar fp16 for the model
        dict(name='serve_16', kind='serve', batch=16, short_lo=300, short_hi=500, quality=90, sampling=420,
             out_h=224, out_w=224, dtype='f16', channels_last=False),
        # CIFAR training: raw 32 x 32, three augmentations; the host's work per batch is what counts
        _loader_case('cifar_train', batch=512, batches=8, batches_ahead=6, mode='raw', short_lo=32, short_hi=32,
                     decoder='simple', out_h=32, out_w=32, ops='flip,translate,cutout'),
        # low-resolution ImageNet training at progressive-resizing sizes
        _loader_case('lowres_train_160', batch=1024, short_lo=200, short_hi=256, max_side=256, out_h=160, out_w=160),
        # ImageNet training from the half raw, half JPEG file
        _loader_case('mix_train_224', batch=512, mode='proportion', max_side=500, order='quasi_random'),
        # validation pass: centre crop, nothing random
        _loader_case('val_256', batch=1024, short_lo=200, short_hi=256, max_side=256, decoder='center', out_h=256,
                     out_w=256, ops='', order='sequential'),
        # high-resolution 4:4:4 training images, large-area downscale
        _loader_case('hires_train_384', batch=64, batches=2, quality=95, sampling=444, short_lo=1024, short_hi=1536,
                     scale_lo=0.25, out_h=384, out_w=384, ops='flip,cutout'),
        # fine-tuning with colour jitter and mixup on the uint8 batch, fp32 result
        _loader_case('colour_mixup_192', batch=256, short_lo=250, short_hi=400, out_h=192, out_w=192, colour=True,
                     dtype='f32'),
        # a small-batch job on a file larger than RAM (read, not mapped), odd output size, planar fp32
        _loader_case('direct_read_small', batch=48, mode='proportion', max_side=500, out_h=187, out_w=187, dtype='f32',
                     channels_last=False, os_cache=False),
    ]


# The largest listed loader cases: bounds of a drawn one.
MAX_SOURCE_PIXELS = 200_000_000
MAX_OUTPUT_PIXELS = 110_000_000


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(['imdecode', 'imdecode', 'resize', 'serve', 'loader', 'loader', 'loader', 'loader', 'loader'])
    if kind == 'imdecode':
        h = _log_int(rng, 64, 1536)
        w = min(2048, max(48, int(h * math.exp(rng.uniform(math.log(3 / 4), math.log(16 / 9))))))
        return dict(kind=kind, height=h, width=w, quality=rng.choice([80, 85, 90, 95]), sampling=rng.choice([420, 420, 444]))
    if kind == 'resize':
        h, w = _log_int(rng, 64, 1200), _log_int(rng, 64, 1200)
        return dict(kind=kind, height=h, width=w, crop_h=rng.randint(h // 2, h), crop_w=rng.randint(w // 2, w),
                    out_h=_log_int(rng, 32, 512), out_w=_log_int(rng, 32, 512))
    if kind == 'serve':
        lo = _log_int(rng, 100, 700)
        return dict(kind=kind, batch=_log_int(rng, 1, 64), short_lo=lo, short_hi=int(lo * rng.uniform(1, 1.6)),
                    quality=rng.choice([80, 85, 90, 95]), sampling=rng.choice([420, 420, 444]),
                    out_h=_log_int(rng, 96, 384), out_w=_log_int(rng, 96, 384), dtype=rng.choice(['f16', 'f32', 'u8']),
                    channels_last=rng.random() < 0.5)
    family = rng.choice(['small', 'train', 'train', 'val', 'hires'])
    case = _loader_case()
    if family == 'small':
        side = _log_int(rng, 24, 96)
        case.update(mode='raw', short_lo=side, short_hi=side, decoder='simple', out_h=side, out_w=side, batches=8,
                    batches_ahead=6, batch=_log_int(rng, 64, 1024), ops=rng.choice(['flip', 'flip,translate', 'flip,translate,cutout']))
    elif family == 'hires':
        lo = _log_int(rng, 800, 1300)
        sampling = rng.choice([420, 444])
        case.update(short_lo=lo, short_hi=int(lo * rng.uniform(1.0, 1.2)), quality=rng.choice([85, 90, 95]), sampling=sampling,
                    scale_lo=rng.choice([0.08, 0.25]), batches=2, batch=_log_int(rng, 8, 64), ops=rng.choice(['flip', 'flip,cutout']))
        case['out_h'] = case['out_w'] = _log_int(rng, 192, 448)
    else:
        lo = _log_int(rng, 120, 480)
        case.update(short_lo=lo, short_hi=int(lo * rng.uniform(1.0, 1.6)), mode=rng.choice(['jpg', 'jpg', 'proportion', 'raw']),
                    quality=rng.choice([80, 85, 90, 95]), sampling=rng.choice([420, 420, 420, 444]), batch=_log_int(rng, 24, 1024),
                    max_side=rng.choice([0, int(1.1 * lo)]), os_cache=rng.random() < 0.8)
        case['out_h'] = case['out_w'] = _log_int(rng, 96, 288)
        if family == 'val':
            case.update(decoder='center', ops='', order='sequential')
        else:
            case.update(ops=rng.choice(['flip', 'flip,cutout', 'flip,translate']), order=rng.choice(['random', 'quasi_random']),
                        colour=rng.random() < 0.25)
    case['dtype'] = 'f32' if case['colour'] else rng.choice(['f16', 'f16', 'f32'])
    case['channels_last'] = case['colour'] or rng.random() < 0.6
    source = _mean_pixels(case) * case['batches']
    output = case['out_h'] * case['out_w'] * case['batches'] * (2 if case['colour'] or case['dtype'] == 'f32' else 1)
    case['batch'] = max(4, min(case['batch'], int(MAX_SOURCE_PIXELS / source), int(MAX_OUTPUT_PIXELS / output)))
    return case


# ---------------------------------------------------------------------------------------- inputs

def _mean_pixels(case):
    """Expected pixels of one stored image of a loader or serve case."""
    short = (case['short_lo'] + case['short_hi']) / 2
    if case.get('decoder') == 'simple':
        return short * short
    long = short * 1.155  # aspect ratio log-uniform in [3/4, 4/3]
    if case.get('max_side') and long > case['max_side']:
        short, long = short * case['max_side'] / long, case['max_side']
    return short * long


def _shape(rng, case):
    short = int(rng.integers(case['short_lo'], case['short_hi'] + 1))
    if case.get('decoder') == 'simple':
        return short, short
    long = int(round(short * math.exp(abs(rng.uniform(math.log(3 / 4), math.log(4 / 3))))))
    if case.get('max_side') and long > case['max_side']:
        short, long = max(1, int(short * case['max_side'] / long)), case['max_side']
    return (short, long) if rng.random() < 0.5 else (long, short)


def _images(rng, seed, shapes):
    """One uint8 [h, w, 3] array per shape, computed on the GPU in groups."""
    dev = torch.device('cuda')
    noise = torch.Generator(device=dev)
    noise.manual_seed(seed)
    out, first = [], 0
    while first < len(shapes):
        last, hm, wm = first, 0, 0
        while last < len(shapes):
            h, w = max(hm, shapes[last][0]), max(wm, shapes[last][1])
            if last > first and h * w * (last - first + 1) > 1 << 23:
                break
            hm, wm, last = h, w, last + 1
        g = last - first
        amp, cx, cy, ph = (torch.from_numpy(rng.uniform(lo, hi, (g, 3, 8))).float().to(dev)
                           for lo, hi in ((8, 32), (-4, 4), (-4, 4), (0, 2 * math.pi)))
        hs = torch.tensor([s[0] for s in shapes[first:last]], device=dev).view(g, 1, 1, 1)
        ws = torch.tensor([s[1] for s in shapes[first:last]], device=dev).view(g, 1, 1, 1)
        x = 2 * math.pi * cx[..., None] * (torch.arange(wm, device=dev) / ws) + ph[..., None]  # [g, 3, 8, w]
        y = 2 * math.pi * cy[..., None] * (torch.arange(hm, device=dev) / hs)                  # [g, 3, 8, h]
        rows = torch.cat([amp[..., None] * y.cos(), amp[..., None] * y.sin()], 2).transpose(2, 3)
        img = torch.matmul(rows, torch.cat([x.sin(), x.cos()], 2))
        img += 128 + 8 * torch.randn(img.shape, device=dev, generator=noise)
        img = img.round_().clamp_(0, 255).to(torch.uint8).permute(0, 2, 3, 1).contiguous().cpu().numpy()
        out += [np.ascontiguousarray(img[k, :h, :w]) for k, (h, w) in enumerate(shapes[first:last])]
        first = last
    return out


def _encoder(case):
    field = make_field(4) if case['sampling'] == 444 else RGBImageField()
    field.jpeg_quality = case['quality']
    return field.encode_jpeg


class _Stored(RGBImageField):
    """Takes samples that are stored already: (mode, height, width, bytes)."""

    def encode(self, destination, sample, malloc):
        destination['mode'], destination['height'], destination['width'], payload = sample
        destination['data_ptr'], storage = malloc(payload.size)
        storage[:] = payload


class _Samples:
    def __init__(self, images, labels):
        self.images, self.labels = images, labels

    def __len__(self):
        return len(self.images)

    def __getitem__(self, k):
        return self.images[k], int(self.labels[k])


def _dataset(case, seed):
    """A .beton of the case's samples in an anonymous in-memory file; returns (file, path)."""
    rng = np.random.default_rng([seed, 1])
    n = case['batch'] * case['batches']
    images = _images(rng, seed, [_shape(rng, case) for _ in range(n)])
    as_jpg = {'jpg': np.ones(n, bool), 'raw': np.zeros(n, bool), 'proportion': rng.random(n) < 0.5}[case['mode']]
    encode = _encoder(case)

    def store(k):
        img = images[k]
        return (0 if as_jpg[k] else 1,) + img.shape[:2] + (encode(img) if as_jpg[k] else img.reshape(-1),)
    with ThreadPoolExecutor() as pool:
        stored = list(pool.map(store, range(n)))
    file = os.fdopen(os.memfd_create('beton'), 'rb')
    path = '/proc/self/fd/%d' % file.fileno()
    DatasetWriter(path, {'image': _Stored(), 'label': IntField()}, num_workers=1).from_indexed_dataset(
        _Samples(stored, rng.integers(0, CLASSES, n)))
    return file, path


def _pipelines(case):
    dev = torch.device('cuda', torch.cuda.current_device())
    size = (case['out_h'], case['out_w'])
    if case['decoder'] == 'simple':
        image = [SimpleRGBImageDecoder()]
    elif case['decoder'] == 'center':
        image = [CenterCropRGBImageDecoder(size, ratio=224 / 256)]
    else:
        image = [RandomResizedCropRGBImageDecoder(size, scale=(case['scale_lo'], 1.0))]
    small = min(size) < 100
    make = {'flip': lambda: RandomHorizontalFlip(), 'translate': lambda: RandomTranslate(padding=2 if small else 8, fill=FILL),
            'cutout': lambda: Cutout(min(size) // 8 if small else min(size) // 6, FILL)}
    image += [make[op]() for op in case['ops'].split(',') if op]
    label = [IntDecoder()]
    if case['colour']:
        image += [RandomBrightness(0.4), RandomContrast(0.4), RandomSaturation(0.4), ImageMixup(0.2, True)]
        label += [LabelMixup(0.2, True), ToTensor(), ToDevice(dev), MixupToOneHot(CLASSES)]
    else:
        label += [ToTensor(), ToDevice(dev), Squeeze()]
    image += [ToTensor(), ToDevice(dev), ToTorchImage(channels_last=case['channels_last']),
              NormalizeImage(MEAN, STD, DTYPES[case['dtype']])]
    return {'image': image, 'label': label}


def _prepare_loader(case, seed):
    gc.collect()  # an earlier loader and its buffers form a cycle
    file, path = _dataset(case, seed)
    loader = Loader(path, batch_size=case['batch'], order=OrderOption[case['order'].upper()], seed=seed,
                    os_cache=case['os_cache'], batches_ahead=case['batches_ahead'], pipelines=_pipelines(case))
    return {'file': file, 'loader': loader}


def _prepare_serve(case, seed):
    rng = np.random.default_rng([seed, 2])
    n = case['batch']
    images = _images(rng, seed, [_shape(rng, case) for _ in range(n)])
    encode = _encoder(case)
    with ThreadPoolExecutor() as pool:
        streams = list(pool.map(encode, images))
    sizes = np.array([s.size for s in streams], np.uint64)
    heights, widths = (np.array([im.shape[a] for im in images], np.uint16) for a in (0, 1))
    params = np.zeros((n, 4), np.int32)  # centre crop of 224 / 256 of the short side
    params[:, 2] = params[:, 3] = (np.minimum(heights, widths).astype(np.int64) * 224 // 256)
    params[:, 0] = (heights.astype(np.int32) - params[:, 2]) // 2
    params[:, 1] = (widths.astype(np.int32) - params[:, 3]) // 2
    dev = torch.device('cuda', torch.cuda.current_device())
    planar = not case['channels_last'] and case['dtype'] != 'u8'
    shape = (n, 3, case['out_h'], case['out_w']) if planar else (n, case['out_h'], case['out_w'], 3)
    table, kind, torch_type = None, L.OUT_U8_NHWC, torch.uint8
    if case['dtype'] != 'u8':
        half = case['dtype'] == 'f16'
        host = ((np.arange(256)[:, None] - MEAN) / STD).astype(DTYPES[case['dtype']])
        table = torch.from_numpy(host).to(dev)
        torch_type = torch.float16 if half else torch.float32
        kind = (L.OUT_F16_NCHW if planar else L.OUT_F16_NHWC) if half else (L.OUT_F32_NCHW if planar else L.OUT_F32_NHWC)
    return {'data': np.concatenate(streams), 'sizes': sizes,
            'offsets': np.concatenate([np.zeros(1, np.uint64), np.cumsum(sizes)[:-1].astype(np.uint64)]),
            'modes': np.zeros(n, np.uint8), 'heights': heights, 'widths': widths, 'params': params, 'table': table,
            'plan': L.make_plan(case['out_h'], case['out_w'], 1, kind, (), table.data_ptr() if table is not None else 0),
            'context': L.Context(dev.index, n_slots=2), 'turn': 0,
            'out': [torch.empty(shape, dtype=torch_type, device=dev) for _ in range(2)]}


def prepare(case, seed):
    if case['kind'] == 'loader':
        state = _prepare_loader(case, seed)
    elif case['kind'] == 'serve':
        state = _prepare_serve(case, seed)
    else:
        h, w = case['height'], case['width']
        image = _images(np.random.default_rng([seed, 3]), seed, [(h, w)])[0]
        if case['kind'] == 'imdecode':
            state = {'stream': _encoder(case)(image), 'out': np.zeros((h, w, 3), np.uint8)}
        else:
            state = {'image': image, 'out': np.zeros((case['out_h'], case['out_w'], 3), np.uint8)}
    state['case'] = case
    return state


# --------------------------------------------------------------------------------------- one pass

def run(state):
    case = state['case']
    if case['kind'] == 'loader':
        return list(state['loader'])
    if case['kind'] == 'serve':
        slot = state['turn']
        state['turn'] = 1 - slot
        context, out = state['context'], state['out'][slot]
        context.stage(slot, state['data'], state['offsets'], state['sizes'], state['modes'], state['heights'],
                      state['widths'], state['plan'], state['params'])
        context.submit(slot, torch.cuda.current_stream().cuda_stream, out.data_ptr())
        return out
    out = state['out']
    if case['kind'] == 'imdecode':
        if L.imdecode(state['stream'], out, case['height'], case['width']) != 0:
            raise RuntimeError('imdecode failed')
    else:
        r0, c0 = (case['height'] - case['crop_h']) // 2, (case['width'] - case['crop_w']) // 2
        L.resize_crop(state['image'], r0, r0 + case['crop_h'], c0, c0 + case['crop_w'], out)
    return out


def work(case):
    """Stored bytes that the result depends on, read once, and the result, written once.  Arithmetic:
    per decoded sample the inverse transform (about 9 integer operations) and per decoded pixel the
    colour conversion (12); per source pixel of a resize a multiply and an add per channel."""
    kind = case['kind']
    if kind == 'resize':
        px = case['crop_h'] * case['crop_w']
        return {'bytes': px * 3 + case['out_h'] * case['out_w'] * 3, 'flops': px * 6}
    density = JPEG_DENSITY[case['sampling'], case['quality']]
    per_pixel = 9 * (3 if case['sampling'] == 444 else 1.5) + 12
    if kind == 'imdecode':
        px = case['height'] * case['width']
        return {'bytes': px * density + px * 3, 'flops': px * per_pixel}
    n = case['batch'] * case.get('batches', 1)
    px = _mean_pixels(case)
    if case.get('decoder') == 'simple':
        used = 1.0
    elif case.get('decoder') == 'rrc':
        used = (1 + case['scale_lo']) / 2
    else:
        used = (224 / 256) ** 2 / 1.1
    jpg = {'jpg': 1.0, 'raw': 0.0, 'proportion': 0.5}[case.get('mode', 'jpg')]
    out_bytes = case['out_h'] * case['out_w'] * 3 * {'u8': 1, 'f16': 2, 'f32': 4}[case['dtype']]
    resize = 0 if case.get('decoder') == 'simple' else 6
    return {'bytes': n * (jpg * px * density + (1 - jpg) * px * used * 3 + out_bytes),
            'flops': n * px * used * (jpg * per_pixel + resize)}


def tolerance(case):
    return 'exact'
