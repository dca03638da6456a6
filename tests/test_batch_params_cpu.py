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
