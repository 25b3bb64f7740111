"""MTF calls that leave outputs out: the axes alone come from the line spread
functions, not from the two-dimensional transform.  Sizes around the sums'
bands (64 rows), column tiles (128) and the frequencies of a block (4)."""
import numpy as np
import pytest

import hybridmantis_b200 as hb
from hybridmantis_b200._lib import ptr
from oracle import analysis_oracle as ao

pytestmark = pytest.mark.gpu


def _mtf(img, k, want):
    out = {n: np.full(k, -7.0) for n in ("freq", "x", "y", "r")}
    args = [ptr(out[n]) if n in want else None for n in out]
    return hb.load().fd2_mtf(0, ptr(img), *img.shape, 1.5, k, *args), out


@pytest.mark.parametrize("shape,freqs", [((1, 1), 1), ((2, 3), 2), ((1, 129), 65), ((128, 1), 5), ((63, 33), 31),
                                         ((64, 128), 65), ((65, 127), 4), ((130, 97), 40), ((191, 257), 3)])
@pytest.mark.parametrize("want", [("freq", "x", "y"), ("x",), ("y",), ("freq",), (), ("r",), ("y", "r")])
def test_mtf_with_outputs_left_out(require_gpu, shape, freqs, want):
    img = np.random.default_rng(sum(shape)).gamma(2.0, 3.0, shape)
    st, got = _mtf(img, freqs, want)
    assert st == 0
    # FP64 sums of up to 49,087 positive terms: 1e-16 of the sum each
    for name, ref in zip(("freq", "x", "y", "r"), ao.mtf(img, 1.5, freqs)):
        if name in want:
            assert np.allclose(got[name], ref, rtol=1e-9, atol=1e-12), name
        else:
            assert (got[name] == -7.0).all(), name


@pytest.mark.parametrize("value", [0.0, -2.0, np.nan])
def test_axes_of_an_image_without_signal(require_gpu, value):
    st, out = _mtf(np.full((70, 31), value), 4, ("freq", "x", "y"))
    assert st == 1 and all((o == -7.0).all() for o in out.values())
