"""Loss and gradients of the training step where its kernels' tiles end: rows
around a warp's, a block's and a 256-row slice's, categories around a pass of
31, points without a radial label, against the numpy oracle."""
import numpy as np
import pytest

import hybridmantis_b200.surrogate as sgm
from oracle import sg_oracle as so

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,bins", [(1, 96), (3, 30), (4, 31), (5, 32), (31, 61), (64, 62), (65, 63), (255, 1),
                                       (257, 96), (513, 130)])
def test_loss_and_gradient_at_tile_edges(require_gpu, rows, bins):
    rng = np.random.default_rng(rows)
    f = rng.uniform(-1, 1, (rows, 8)).astype(np.float32)
    ph = np.full(rows, 1000, np.int32)
    det = rng.integers(0, 1001, rows).astype(np.int32)
    rad = rng.integers(0, 40, (rows, bins + 1)).astype(np.uint32)
    rad[:, bins // 2:] *= rng.integers(0, 2, (rows, bins + 1 - bins // 2)).astype(np.uint32)
    rad[::5] = 0  # no radial label
    with sgm.Surrogate(hidden=64, radial_bins=bins, radial_max_um=200.0, batch=640) as s:
        s.set_hull(np.full(8, -1.0), np.full(8, 1.0))
        loss, g = s.loss_grad(f, ph, det, rad)
        want, wg = so.loss_grad(s.params(), 64, f, np.full(8, -1.0), np.full(8, 1.0), ph, det, rad, bins, 200.0)
    # FP32 sums of up to 131 categories and 513 rows of terms of mixed sign
    # beside FP64 ones: 1e-4 of the gradient's norm (BF16 roundings that fall
    # the other way are 2^-9 of single entries)
    assert loss == pytest.approx(want, rel=1e-5)
    assert np.linalg.norm(g - wg) <= 2e-3 * np.linalg.norm(wg)


@pytest.mark.parametrize("rows,bins", [(6, 2), (7, 33), (8, 64), (9, 65), (10, 95), (11, 97)])
def test_loss_and_gradient_around_passes_of_32_edges(require_gpu, rows, bins):
    test_loss_and_gradient_at_tile_edges(None, rows, bins)


@pytest.mark.parametrize("rows", [1, 127, 129, 8193, 37887, 37891, 75780])
def test_predict_at_pass_edges(require_gpu, rows):
    f = np.random.default_rng(rows).uniform(-1, 1, (rows, 8)).astype(np.float32)
    with sgm.Surrogate() as s:
        s.set_hull(np.full(8, -1.0), np.full(8, 1.0))
        out = s.predict(f)
        # rows do not depend on the rows around them
        for a, b in ((0, min(rows, 70)), (max(rows - 70, 0), rows), (37888 - 3, min(rows, 37888 + 40))):
            if a < b:
                assert np.array_equal(out[a:b], s.predict(f[a:b]))
        want, _ = so.forward(s.params(), 256, f[-64:], np.full(8, -1.0), np.full(8, 1.0))
    # the oracle rounds to BF16 where the GPU stores BF16; FP32 sums of 256
    # terms may round an activation the other way (2^-9 of one of 256)
    assert np.abs(out[-64:] - want).max() <= 2e-2 * np.abs(want).max()
