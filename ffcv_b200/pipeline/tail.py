"""Runs of operations behind a fused decoder that become one native call each.

The reference runs colour jitter, mixup and normalisation one closure at a time
(``ffcv/loader/epoch_iterator.py:145-149``); so does :class:`~ffcv_b200.pipeline.graph.Graph` for
operations it does not know.  The runs recognised here are drawn on the host operation by operation,
exactly as their closures draw, and then go to the GPU as a single chain.
"""
import numpy as np
import torch as ch

from ..fields.basics import IntDecoder
from ..transforms.color_jitter import RandomBrightness, RandomContrast, RandomSaturation
from ..transforms.mixup import ImageMixup, LabelMixup, MixupToOneHot, _lambdas
from ..transforms.normalize import NormalizeImage
from ..transforms.ops import ToDevice, ToTensor, ToTorchImage

_JITTERS = (RandomBrightness, RandomContrast, RandomSaturation)
MAX_CHAIN = 8


class PixelChain:
    """[jitter]* [ImageMixup] then, possibly among ToTensor / ToDevice / ToTorchImage, NormalizeImage."""

    def __init__(self, device):
        self.device = device
        self.jitters = []      # (position in the pipeline, operation)
        self.mixup = None
        self.normalize = None
        self.torch_image = False
        self.end = None        # position behind the run
        self.buffer_op = None  # position of the operation whose buffer takes the result (None: in place)
        self.table = None

    @staticmethod
    def match(ops, first, state_shape, device):
        """The chain that starts at ops[first], or None."""
        chain = PixelChain(device)
        k = first
        while k < len(ops) and type(ops[k]) in _JITTERS and len(chain.jitters) < MAX_CHAIN:
            chain.jitters.append((k, ops[k]))
            k += 1
        if k < len(ops) and type(ops[k]) is ImageMixup:
            chain.mixup, chain.buffer_op = ops[k], k
            k += 1
        if not chain.jitters and chain.mixup is None:
            return None
        chain.end = k
        torch_image = False
        while k < len(ops):  # layout operations only count when a normalisation follows
            op = ops[k]
            if type(op) is ToTorchImage and op.channels_last and not op.enable_int16conv and not torch_image:
                torch_image = True
            elif type(op) is NormalizeImage and state_shape[1] != 3:  # (with a width of 3 the layouts look alike)
                chain.normalize, chain.buffer_op, chain.torch_image, chain.end = op, k, torch_image, k + 1
                break
            elif not (type(op) is ToTensor or (type(op) is ToDevice and _same_device(op.device, device))):
                break
            k += 1
        chain.kinds = np.array([op.kind for _, op in chain.jitters], dtype=np.int32)
        if chain.normalize is not None:
            raw = chain.normalize.lookup_table
            chain.table = ch.from_numpy(raw.view(np.int16 if raw.dtype == np.float16 else np.int32).copy()).to(device)
        return chain

    def __call__(self, images, buffer, batch_indices, seed, epoch, batch_ix, pipeline_ix):
        from .graph import shared_context
        (self.jitters[0][1] if self.jitters else self.mixup).check_input(images)
        n, h, w, _ = images.shape
        apply = np.empty((len(self.jitters), n), dtype=np.uint8)
        ratio = np.empty((len(self.jitters), n), dtype=np.float64)
        for row, (k, op) in enumerate(self.jitters):
            op.begin_batch(seed, epoch, batch_ix, pipeline_ix * 64 + k)
            op.draw_into(apply[row], ratio[row])
        lam = None
        if self.mixup is not None:
            lam = _lambdas(self.mixup.alpha, self.mixup.same_lambda, batch_indices, n)
            self.mixup.last_draw = lam
        out = images if buffer is None else buffer[:n].view(n, h, w, 3)
        shared_context(images.device).pixel_chain(ch.cuda.current_stream(images.device).cuda_stream, images.data_ptr(), n, h * w,
                                                  self.kinds, apply, ratio, lam, out.element_size(),
                                                  self.table.data_ptr() if self.table is not None else 0, out.data_ptr())
        return out.permute(0, 3, 1, 2) if self.torch_image else out


class SoftLabels:
    """IntDecoder, LabelMixup, ToTensor, ToDevice, MixupToOneHot: the whole label pipeline of mixup."""
    n_ops = 5

    @staticmethod
    def match(ops):
        if len(ops) < 5 or [type(op) for op in ops[:5]] != [IntDecoder, LabelMixup, ToTensor, ToDevice, MixupToOneHot] or \
                ops[3].device.type != 'cuda':
            return None
        self = SoftLabels()
        self.mixup, self.one_hot = ops[1], ops[4]
        return self

    def __call__(self, column, out, batch_indices):
        from .graph import shared_context
        n = len(batch_indices)
        lam = _lambdas(self.mixup.alpha, self.mixup.same_lambda, batch_indices, n)
        shared_context(out.device).onehot_mix(ch.cuda.current_stream(out.device).cuda_stream, n, self.one_hot.num_classes,
                                              column[batch_indices].astype(np.int32), lam.astype(np.float32), out.data_ptr())
        return out


def _same_device(device, other):
    index = device.index if device.index is not None else ch.cuda.current_device()
    return device.type == other.type and index == other.index

