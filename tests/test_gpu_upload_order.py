"""Uploads of the caller's arrays are in place before the kernels that read them:
calls with other data in turn, the arrays large enough that a copy outlasts the
call that starts it, give what each gives by itself."""
import numpy as np
import pytest

import hybridmantis_b200.surrogate as sgm
from hybridmantis_b200 import xray as xr

pytestmark = pytest.mark.gpu


def _labels(seed, n, bins):
    rng = np.random.default_rng(seed)
    f = rng.uniform(-1, 1, (n, 8)).astype(np.float32)
    det = rng.integers(0, 1001, n).astype(np.int32)
    rad = rng.integers(0, 30, (n, bins + 1)).astype(np.uint32)
    # the radial labels of odd seeds lie in the outer half: far apart losses
    if seed % 2:
        rad[:, :bins // 2] = 0
    return f, np.full(n, 1000, np.int32), det, rad


@pytest.mark.parametrize("bins,n", [(1024, 256), (1024, 2048), (96, 8192)])
def test_loss_of_alternating_batches(require_gpu, bins, n):
    sets = [_labels(s, n, bins) for s in range(4)]
    with sgm.Surrogate(hidden=64, batch=8192, radial_bins=bins, seed=5) as s:
        s.set_hull(np.full(8, -1.0), np.full(8, 1.0))
        first = []
        for k in sets:
            s.loss_grad(*k)
            first.append(s.loss_grad(*k))  # the same data were there before it
        for _ in range(5):
            for k, (loss, grad) in zip(sets, first):
                got, g = s.loss_grad(*k)
                # the rows' losses are added in FP64 in the order blocks end
                assert got == pytest.approx(loss, rel=1e-6)
                assert np.array_equal(g, grad)


def test_training_right_after_new_data(require_gpu):
    sets = [_labels(s, 8192, 96) for s in range(2)]

    def after(k):
        with sgm.Surrogate(hidden=64, batch=512, seed=5) as s:
            for j in (1 - k, k):
                s.set_data(*sets[j], n_val=0)
                s.train(1)
            return s.params()

    for k in (0, 1):
        want = after(k)
        for _ in range(3):
            assert np.array_equal(after(k), want)


def test_learning_rate_right_before_a_step(require_gpu):
    k = _labels(0, 512, 96)
    with sgm.Surrogate(hidden=64, batch=512, lr=1e-3, seed=5) as s:
        s.set_data(*k, n_val=0)
        s.train(1)
        p0 = s.params()
        s.set_lr(1e-30)
        s.train(1)
        assert np.array_equal(s.params(), p0)


def test_cleared_statistics_of_the_front_end(require_gpu):
    with xr.XrayFrontEnd(seed=3) as f:
        src = xr.monoenergetic(25000.0)
        for _ in range(5):
            f.run(src, 200)
            assert f.stats()["histories"] == 200
            f.clear_stats()
            assert f.stats()["histories"] == 0
