"""The training step's gradient parameter block by parameter block (weights and
biases of each layer), so that a mistake in a small block cannot hide behind the
norm of a large one: a wrong bias column, a dropped row, a category at the wrong
side of a pass."""
import numpy as np
import pytest

import hybridmantis_b200.surrogate as sgm
from oracle import sg_oracle as so

pytestmark = pytest.mark.gpu

NAMES = ("W1", "b1", "W2", "b2", "W3", "b3", "W4", "b4")


@pytest.mark.parametrize("rows,bins,hidden", [(3, 31, 64), (4, 32, 64), (65, 33, 64), (255, 64, 64), (256, 65, 256),
                                              (257, 95, 256), (513, 97, 64), (640, 130, 128)])
def test_gradient_of_every_block(require_gpu, rows, bins, hidden):
    rng = np.random.default_rng(rows + bins)
    f = rng.uniform(-1, 1, (rows, 8)).astype(np.float32)
    ph = np.full(rows, 1000, np.int32)
    det = rng.integers(0, 1001, rows).astype(np.int32)
    rad = rng.integers(0, 40, (rows, bins + 1)).astype(np.uint32)
    rad[::5] = 0  # no radial label
    lo, hi = np.full(8, -1.0), np.full(8, 1.0)
    with sgm.Surrogate(hidden=hidden, radial_bins=bins, radial_max_um=200.0, batch=640) as s:
        s.set_hull(lo, hi)
        loss, g = s.loss_grad(f, ph, det, rad)
        want, wg = so.loss_grad(s.params(), hidden, f, lo, hi, ph, det, rad, bins, 200.0)
    # FP32 sums of up to 131 categories, as relative rounding of the mean loss
    assert loss == pytest.approx(want, rel=131 * 2.0 ** -24)
    # An entry of a layer's gradient that the GPU's FP32 sums put on the other
    # side of a BF16 rounding is 2^-8 of itself off.  Of the output layer's
    # (directly below the loss) fewer than one in 16 are, of the hidden layers',
    # below up to three such roundings, fewer than one in 4: sqrt(1/16) and
    # sqrt(1/4) of 2^-8 of a block's norm.  A row of 640 is 1/640 of a sum that
    # all rows push the same way, and 1/sqrt(640) = 10 x 2^-8 of one where they
    # do not.
    for name, got, ref in zip(NAMES, so.unpack(g, hidden), so.unpack(wg, hidden)):
        bound = (0.25 if name in ("W4", "b4") else 0.5) * 2.0 ** -8
        assert np.linalg.norm(got - ref) <= bound * np.linalg.norm(ref), name
