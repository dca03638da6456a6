"""Lowering of an image pipeline to one GPU launch per batch.

The reference runs ``decoder -> flip -> translate -> cutout`` as numba loops on host arrays, copies
the uint8 batch to the GPU in ``ToDevice`` and normalises it there
(``ffcv/loader/epoch_iterator.py:145-149``).  Here the longest prefix of a pipeline made of
operations that implement :meth:`Operation.fuse` becomes a :class:`FusedImagePlan`: the compressed
(or raw) sample bytes go to the GPU and one call of the native library produces the final tensor.
Operations after the fused prefix run one by one through their ``generate_code`` closures.
"""
import numpy as np
import torch as ch

from .. import libffcv as L
from .sampling import CROP_CENTER, CROP_RANDOM, CROP_WHOLE, batch_seed, gather_batch, prepare_batch


class FusedImagePlan:
    def __init__(self):
        self.decoder = None       # the RGB image decoder opening the pipeline
        self.crop_sampler = None  # operation that draws the crop boxes when it is not the decoder
        self.out_h = self.out_w = None
        self.resize = False
        self.dct_scale = 0        # scale of the JPEG decode (ffcvb_plan.dct_scale): 0 full, -1 by crop box
        self.ops = []             # (native type, arg, fill, operation) in pipeline order
        self.device = None        # set by ToDevice; defaults to the current CUDA device
        self.table = None         # 256 x 3 lookup table of the output type (numpy), or None
        self.torch_image = False  # result presented as (B, C, H, W)
        self.channels_last = True
        self.sealed = False       # no spatial operation may follow (values are no longer uint8)
        self.fused_ops = []

    # ---- called by Operation.fuse implementations
    def set_decoder(self, op, out_h, out_w, resize):
        if self.decoder is not None:
            return False
        self.decoder, self.out_h, self.out_w, self.resize = op, int(out_h), int(out_w), bool(resize)
        return True

    def set_post_crop(self, op, size):
        """A random-resized-crop transform right behind a pass-through decoder is the crop-and-resize
        of the decoder itself."""
        if self.decoder is None or self.resize or self.ops or self.sealed or self.torch_image:
            return False
        self.crop_sampler = op
        self.out_h = self.out_w = int(size)
        self.resize = True
        return True

    def add_spatial(self, native_type, arg, fill, op):
        if self.decoder is None or self.sealed or self.torch_image or len(self.ops) >= L.MAX_OPS:
            return False
        self.ops.append((native_type, int(arg), tuple(int(v) for v in fill), op))
        return True

    def set_table(self, table):
        """table: float16/float32 array [256, 3]; replaces an earlier one (a Convert followed by
        NormalizeImage indexes the normalisation table with the uint8 value)."""
        if self.decoder is None:
            return False
        if self.sealed and self.table is not None and not getattr(self, '_table_is_identity', False):
            return False
        self.table = np.ascontiguousarray(table)
        self.sealed = True
        return True

    def set_identity_table(self, dtype):
        ok = self.set_table(np.repeat(np.arange(256, dtype=dtype)[:, None], 3, axis=1))
        self._table_is_identity = ok
        return ok

    def set_torch_image(self, channels_last):
        if self.decoder is None or self.torch_image:
            return False
        self.torch_image, self.channels_last = True, bool(channels_last)
        return True

    # ---- derived
    @property
    def out_kind(self):
        if self.table is None:
            return L.OUT_U8_NHWC
        planar = self.torch_image and not self.channels_last
        if self.table.dtype == np.float16:
            return L.OUT_F16_NCHW if planar else L.OUT_F16_NHWC
        return L.OUT_F32_NCHW if planar else L.OUT_F32_NHWC

    @property
    def torch_dtype(self):
        if self.table is None:
            return ch.uint8
        return ch.float16 if self.table.dtype == np.float16 else ch.float32

    @property
    def buffer_shape(self):
        if self.torch_image and not self.channels_last and self.table is not None:
            return (3, self.out_h, self.out_w)
        return (self.out_h, self.out_w, 3)

    def needs_repack(self):
        # uint8 output asked for as contiguous NCHW: the kernel writes NHWC, torch repacks
        return self.torch_image and not self.channels_last and self.table is None


def host_plan(ops, field, metadata):
    """The :class:`FusedImagePlan` of the longest fusable prefix of ``ops`` (decoder first), built
    on the host alone: no native context, no GPU.  ``metadata`` is the field's metadata column."""
    plan = FusedImagePlan()
    for op in ops:
        op.accept_field(field)
        op.accept_globals(metadata, None)
        if not op.fuse(plan):
            break
        plan.fused_ops.append(op)
    return plan


def sample_plan_params(plan, md, base_seed, epoch, batch_ix):
    """Parameter table of one batch, ``[n, 4 + 2 * len(plan.ops)]`` int32: the crop box of every
    sample followed by the two values each augmentation draws.  ``md``: the batch's metadata rows.
    Every operation seeds its own stream from (seed, epoch, batch, position in the pipeline)."""
    heights = np.ascontiguousarray(md['height'])
    widths = np.ascontiguousarray(md['width'])
    n = len(md)
    params = np.zeros((n, 4 + 2 * len(plan.ops)), dtype=np.int32)
    crops = np.zeros((n, 4), dtype=np.int32)
    (plan.crop_sampler or plan.decoder).sample_crops(batch_seed(base_seed, epoch, batch_ix, 0), heights, widths, crops)
    params[:, :4] = crops
    for k, (_, _, _, op) in enumerate(plan.ops):
        col = np.zeros((n, 2), dtype=np.int32)
        op.sample_params(batch_seed(base_seed, epoch, batch_ix, k + 1), n, plan.out_h, plan.out_w, col)
        params[:, 4 + 2 * k:6 + 2 * k] = col
    return params


def _native_sampling(plan):
    """The arguments of :func:`prepare_batch` that draw a plan's parameters, or None when the plan
    contains an operation that this module does not know (a subclass draws what it likes)."""
    from ..fields.rgb_image import (CenterCropRGBImageDecoder, RandomResizedCropRGBImageDecoder, SimpleRGBImageDecoder)
    from ..transforms.cutout import Cutout
    from ..transforms.flip import RandomHorizontalFlip
    from ..transforms.random_resized_crop import RandomResizedCrop
    from ..transforms.translate import RandomTranslate
    sampler = plan.crop_sampler or plan.decoder
    scale = ratio = np.zeros(2)
    if type(sampler) in (RandomResizedCropRGBImageDecoder, RandomResizedCrop):
        crop, scale, ratio = CROP_RANDOM, np.array(sampler.scale, dtype=np.float64), np.array(sampler.ratio, dtype=np.float64)
    elif type(sampler) is CenterCropRGBImageDecoder:
        crop, ratio = CROP_CENTER, np.array([sampler.ratio, 0.0], dtype=np.float64)
    elif type(sampler) is SimpleRGBImageDecoder:
        crop = CROP_WHOLE
    else:
        return None
    args = {RandomHorizontalFlip: lambda op: op.flip_prob, RandomTranslate: lambda op: op.padding, Cutout: lambda op: op.crop_size}
    if any(type(op) not in args for (_, _, _, op) in plan.ops):
        return None
    types = np.array([t for (t, _, _, _) in plan.ops], dtype=np.int64)
    values = np.array([float(args[type(op)](op)) for (_, _, _, op) in plan.ops], dtype=np.float64)
    return crop, scale, ratio, types, values, int(plan.out_h), int(plan.out_w)


class FusedImageExecutor:
    """Per-batch driver of a :class:`FusedImagePlan` on one native context."""

    def __init__(self, plan: FusedImagePlan, ctx, metadata, sample_sizes, file_base_fn, base_seed):
        self.plan = plan
        self.ctx = ctx
        self.metadata = metadata
        self.sample_sizes = sample_sizes
        self.file_base_fn = file_base_fn
        self.base_seed = int(base_seed) & 0xFFFFFFFF
        self.device = plan.device if plan.device is not None else ch.device('cuda', ch.cuda.current_device())
        self.table_dev = None
        if plan.table is not None:
            raw = plan.table.view(np.int16 if plan.table.dtype == np.float16 else np.int32)
            self.table_dev = ch.from_numpy(raw.copy()).to(self.device)
        ops = [(t, a, f) for (t, a, f, _) in plan.ops]
        self.native_plan = L.make_plan(plan.out_h, plan.out_w, plan.resize, L.OUT_U8_NHWC if plan.needs_repack()
                                       else plan.out_kind, ops,
                                       self.table_dev.data_ptr() if self.table_dev is not None else 0,
                                       dct_scale=plan.dct_scale)
        self.n_params = 4 + 2 * len(ops)
        # the sample table as columns, and the arrays a batch is prepared in (the native call has taken
        # what it needs when it returns, so one set serves all batches)
        self.columns = (np.ascontiguousarray(metadata['data_ptr'], dtype=np.uint64),
                        np.ascontiguousarray(sample_sizes, dtype=np.uint64),
                        np.ascontiguousarray(metadata['mode'], dtype=np.uint8),
                        np.ascontiguousarray(metadata['height'], dtype=np.uint16),
                        np.ascontiguousarray(metadata['width'], dtype=np.uint16))
        self.sampling = _native_sampling(plan)
        self._arrays = None
        self.last_params = None   # parameter table of the last batch, an array of its own
        self.param_log = None     # set to a list to record (epoch, batch, indices, parameter table) per batch
        self._last_slot = None
        self.riders = []          # other fields' values for the next batch (see Graph.attach_riders)

    @property
    def h2d_bytes(self):
        """Bytes the last batch moved host->device."""
        return 0 if self._last_slot is None else self.ctx.staged_bytes(self._last_slot)

    @property
    def launches(self):
        """Kernels of this library the last batch launched."""
        return 0 if self._last_slot is None else self.ctx.launches(self._last_slot)

    def allocate(self, batch_size, slots):
        p = self.plan
        return [ch.empty((batch_size,) + p.buffer_shape, dtype=p.torch_dtype, device=self.device) for _ in range(slots)]

    def prepare(self, batch_indices, epoch, batch_ix):
        """Everything ffcvb_stage_batch needs for one batch: the rows of the sample table and the
        parameter table, in arrays that the next call overwrites."""
        batch_indices = np.ascontiguousarray(batch_indices, dtype=np.int64)
        n = len(batch_indices)
        if self._arrays is None or len(self._arrays[1]) != n:
            self._arrays = (tuple(np.empty(n, c.dtype) for c in self.columns), np.zeros((n, self.n_params), dtype=np.int32))
            self._staging = L.BatchArrays(*self._arrays[0], self._arrays[1])
        batch, params = self._arrays
        if self.sampling is not None:
            prepare_batch(batch_indices, self.columns, batch, self.base_seed, epoch, batch_ix, *self.sampling, params)
        else:
            gather_batch(batch_indices, self.columns, batch)
            params[:] = sample_plan_params(self.plan, self.metadata[batch_indices], self.base_seed, epoch, batch_ix)
        return params

    def __call__(self, batch_indices, slot, stream_ptr, out, epoch, batch_ix, outputs_free=None):
        params = self.prepare(batch_indices, epoch, batch_ix)
        self.last_params = params.copy()
        if self.param_log is not None:
            self.param_log.append((epoch, batch_ix, np.array(batch_indices), self.last_params))
        n = len(batch_indices)
        if self.riders:
            self.ctx.set_riders(slot, self.riders, n)
            self.riders = []
        # with asynchronous staging this returns while the staging threads still copy the payloads
        self.ctx.stage_arrays(slot, self.file_base_fn(), self._staging, self.native_plan)
        dst = out if len(out) == n else out[:n]
        self.ctx.submit(slot, stream_ptr, dst.data_ptr(), outputs_free)
        self._last_slot = slot
        p = self.plan
        if p.torch_image:
            if p.needs_repack():
                return dst.permute(0, 3, 1, 2).contiguous()
            if p.channels_last:
                return dst.permute(0, 3, 1, 2)
        return dst
