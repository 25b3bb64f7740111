"""Gradients of batches of any number of rows where the layers go through the
mma.sync products (more than 256 hidden units, or FD2_SG_GEMM=mma): rows past the
batch, which hold what an earlier, larger batch left there, do not count."""
import numpy as np
import pytest

import hybridmantis_b200.surrogate as sgm
from oracle import sg_oracle as so

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("gemm,hidden", [("", 64), ("mma", 64), ("", 320)])
@pytest.mark.parametrize("rows", [1, 31, 32, 33, 63, 513, 640])
def test_gradient_after_a_larger_batch(require_gpu, monkeypatch, gemm, hidden, rows):
    monkeypatch.setenv("FD2_SG_GEMM", gemm)
    rng = np.random.default_rng(rows)
    n, bins = 640, 40
    f = rng.uniform(-1, 1, (n, 8)).astype(np.float32)
    ph = np.full(n, 1000, np.int32)
    det = rng.integers(0, 1001, n).astype(np.int32)
    rad = rng.integers(0, 40, (n, bins + 1)).astype(np.uint32)
    lo, hi = np.full(8, -1.0), np.full(8, 1.0)
    with sgm.Surrogate(hidden=hidden, radial_bins=bins, radial_max_um=200.0, batch=640) as s:
        s.set_hull(lo, hi)
        s.loss_grad(f, ph, det, rad)  # all rows
        part = (f[:rows], ph[:rows], det[:rows], rad[:rows])
        loss, g = s.loss_grad(*part)
        want, wg = so.loss_grad(s.params(), hidden, f[:rows], lo, hi, *part[1:], bins, 200.0)
    assert loss == pytest.approx(want, rel=1e-5)
    # fewer than one entry in four on the other side of a BF16 rounding (2^-8 of
    # itself); one stale row of 33 is 1/33 of the gradient
    assert np.linalg.norm(g - wg) <= 0.5 * 2.0 ** -8 * np.linalg.norm(wg)
