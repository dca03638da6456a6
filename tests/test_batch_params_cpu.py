"""The one-call preparation of a batch draws exactly what the operations draw one by one."""
import numpy as np
import pytest

from ffcv_b200.pipeline import sampling as S


@pytest.mark.parametrize('n', [1, 7, 512])
@pytest.mark.parametrize('crop', [S.CROP_WHOLE, S.CROP_RANDOM, S.CROP_CENTER])
def test_prepare_batch_equals_the_single_draws(n, crop):
    rng = np.random.default_rng(n * 3 + crop)
    total = 600
    columns = (rng.integers(0, 1 << 50, total).astype(np.uint64), rng.integers(1, 1 << 31, total).astype(np.uint64),
               rng.integers(0, 2, total).astype(np.uint8), rng.integers(3, 3000, total).astype(np.uint16),
               rng.integers(3, 3000, total).astype(np.uint16))
    scale, ratio = np.array([0.08, 1.0]), np.array([0.75, 4 / 3])
    ops = [(S.OP_FLIP, 0.5), (S.OP_CUTOUT, 9), (S.OP_TRANSLATE, 4)]
    for trial in range(40):
        indices = rng.integers(0, total, n)
        seed, epoch, batch_ix = int(rng.integers(1 << 32)), trial, int(rng.integers(1 << 20))
        batch = tuple(np.empty(n, c.dtype) for c in columns)
        params = np.full((n, 10), -1, np.int32)
        S.prepare_batch(indices, columns, batch, seed, epoch, batch_ix, crop, scale, ratio, np.array([o for o, _ in ops]),
                        np.array([float(a) for _, a in ops]), 40, 50, params)
        for got, column in zip(batch, columns):
            assert np.array_equal(got, column[indices])
        want = np.zeros((n, 4), np.int32)
        if crop == S.CROP_RANDOM:
            S.sample_random_crops(S.batch_seed(seed, epoch, batch_ix, 0), batch[3], batch[4], scale, ratio, want)
        elif crop == S.CROP_CENTER:
            S.sample_center_crops(batch[3], batch[4], ratio[0], want)
        else:
            want[:, 2], want[:, 3] = batch[3], batch[4]
        assert np.array_equal(params[:, :4], want)
        draws = [lambda s, o: S.sample_flips(s, n, 0.5, o), lambda s, o: S.sample_cutouts(s, n, 40, 50, 9, o),
                 lambda s, o: S.sample_translations(s, n, 4, o)]
        for k, draw in enumerate(draws):
            column = np.zeros((n, 2), np.int32)
            draw(S.batch_seed(seed, epoch, batch_ix, k + 1), column)
            assert np.array_equal(params[:, 4 + 2 * k:6 + 2 * k], column)


def test_last_params_of_a_batch_outlive_it():
    """The parameter table a caller took from the executor is not the array the next batch is prepared in."""
    import torch as ch
    from ffcv_b200.fields.decoders import RandomResizedCropRGBImageDecoder
    from ffcv_b200.pipeline.fusion import FusedImageExecutor, FusedImagePlan
    from ffcv_b200.transforms import RandomHorizontalFlip

    class Recorder:  # in place of the native context
        def __init__(self):
            self.staged = []

        def stage_arrays(self, slot, base, arrays, plan):
            self.staged.append(arrays.arrays[5].copy())

        def submit(self, *args):
            pass

    n = 40
    md = np.zeros(n, dtype=[('mode', 'u1'), ('width', '<u2'), ('height', '<u2'), ('data_ptr', '<u8')])
    md['width'], md['height'] = 300, 200
    plan = FusedImagePlan()
    for op in (RandomResizedCropRGBImageDecoder((32, 32)), RandomHorizontalFlip()):
        assert op.fuse(plan)
    plan.device = ch.device('cpu')
    ctx = Recorder()
    exe = FusedImageExecutor(plan, ctx, md, np.full(n, 1000, np.uint64), lambda: 0, 7)
    exe.param_log = []
    out = exe.allocate(16, 1)[0]
    taken = []
    for b in range(3):
        exe(np.arange(16), 0, 0, out, 0, b)
        taken.append(exe.last_params)
    assert all(np.array_equal(t, s) for t, s in zip(taken, ctx.staged))
    assert all(np.array_equal(t, s) for (_, _, _, t), s in zip(exe.param_log, ctx.staged))
    assert not np.array_equal(taken[0], taken[1]) and not np.array_equal(taken[1], taken[2])
