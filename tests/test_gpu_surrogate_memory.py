"""Device memory of a surrogate's training buffers: the layers' own operands and
partial sums exist only where the layers' weight gradients run side by side."""
import numpy as np
import pytest
import torch

import hybridmantis_b200.surrogate as sgm

pytestmark = pytest.mark.gpu

MIB = 1 << 20


def _used(hidden, batch, bins=96):
    n = 64
    rng = np.random.default_rng(hidden)
    f = rng.uniform(-1, 1, (n, 8)).astype(np.float32)
    args = (f, np.full(n, 100, np.int32), np.full(n, 40, np.int32),
            rng.integers(0, 9, (n, bins + 1)).astype(np.uint32))
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    with sgm.Surrogate(hidden=hidden, batch=batch, radial_bins=bins) as s:
        s.set_hull(np.full(8, -1.0), np.full(8, 1.0))
        loss, g = s.loss_grad(*args)
        used = before - torch.cuda.mem_get_info()[0]
    assert np.isfinite(loss) and np.isfinite(g).all()
    return used


# bytes of a row: inputs and outputs (32 and 64 BF16, 64 FP32), six layers of
# BF16 activations and gradients, labels, target, flag
def _row(hidden, bins=96):
    return 2 * 32 + 2 * 64 + 4 * 64 + 6 * 2 * hidden + 4 * (bins + 1) + 8


@pytest.mark.parametrize("gemm,hidden", [("", 512), ("", 1024), ("mma", 256)])
def test_no_side_buffers_without_side_streams(require_gpu, monkeypatch, gemm, hidden):
    monkeypatch.setenv("FD2_SG_GEMM", gemm)
    _used(hidden, 64)  # modules loaded
    batch = 1 << 16
    params = 2 * hidden * hidden + (32 + 64 + 4) * hidden
    # the rows, 16 planes of the largest layer, parameters in six copies, and
    # what the allocator rounds up
    limit = batch * _row(hidden) + 16 * 4 * hidden * hidden + 6 * 4 * params + 64 * MIB
    assert _used(hidden, batch) <= limit


def test_side_buffers_of_the_layers(require_gpu):
    _used(256, 64)
    batch = 1 << 16
    # four times two operands and a plane for every 256 rows
    side = 4 * (2 * 2 * 256 * batch + batch // 256 * 4 * 256 * 256)
    assert _used(256, batch) <= batch * _row(256) + side + 64 * MIB
