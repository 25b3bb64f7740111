"""Which images have signal: the image's sum, added pixel by pixel, is positive
and finite (MTF).  Images whose values cancel make the order of the additions
visible; a refused call leaves its outputs alone."""
import ctypes

import numpy as np
import pytest

import hybridmantis_b200 as hb
from hybridmantis_b200._lib import ptr

pytestmark = pytest.mark.gpu

INVALID = 1


def _mtf(img, k):
    out = [np.full(k, -7.0) for _ in range(4)]
    st = hb.load().fd2_mtf(0, ptr(img), *img.shape, 1.0, k, *[ptr(o) for o in out])
    return st, out


# (37, 53): of these 40 images 10 have sums of other signs row by row
@pytest.mark.parametrize("seed", range(40))
def test_a_cancelling_image_is_decided_pixel_by_pixel(require_gpu, seed):
    img = np.random.default_rng(seed).normal(0.0, 1.0, (37, 53))
    img -= img.mean()
    total = float(np.cumsum(img.ravel())[-1])  # in order
    st, (freq, mx, my, mr) = _mtf(img, 20)
    if total > 0.0:
        assert st == 0
        pad = np.zeros((53, 53))
        pad[:37] = img
        h = np.abs(np.fft.fft2(pad))
        # FP64 sums of 1,961 terms of unit size
        assert np.allclose(mx * total, h[:20, 0], rtol=0.0, atol=1e-11)
        assert np.allclose(my * total, h[0, :20], rtol=0.0, atol=1e-11)
        assert np.array_equal(freq, 1000.0 * np.arange(20) / 53.0)
    else:
        assert st == INVALID
        assert all((o == -7.0).all() for o in (freq, mx, my, mr))


@pytest.mark.parametrize("value", [0.0, -0.0, -1.0, np.nan, np.inf])
def test_an_image_without_signal_is_refused_untouched(require_gpu, value):
    img = np.full((9, 12), value)
    st, out = _mtf(img, 3)
    assert st == INVALID and all((o == -7.0).all() for o in out)
    img = np.full((9, 12), 1.0)
    img[4, 4] = value
    st, out = _mtf(img, 3)
    assert st == (0 if np.isfinite(value) else INVALID)


def _region_mean(imgs, roi, across):
    """Mean signal as fd2_nnps adds it up: pixel t of a region to one of 128
    partial sums, those in a tree, the regions in order."""
    mean = imgs[0] if len(imgs) == 1 else (imgs[0] + imgs[1]) / 2.0
    total = 0.0
    for q in range(across):
        v = mean[:roi, q * roi:(q + 1) * roi].ravel()
        part = np.zeros(128)
        for i in range(0, len(v), 128):
            part[:len(v[i:i + 128])] += v[i:i + 128]
        w = 64
        while w:
            part[:w] += part[w:2 * w]
            w //= 2
        total += float(part[0])
    return total / (float(across) * roi * roi)


# of these 80 stacks 4 have means of other signs with 1,024 partial sums
@pytest.mark.parametrize("seed", range(40))
@pytest.mark.parametrize("n", [1, 2])
def test_cancelling_flat_fields_are_decided_in_a_fixed_order(require_gpu, seed, n):
    imgs = np.random.default_rng(seed).normal(0.0, 1.0, (n, 35, 70))
    imgs -= imgs[:, :33, :66].mean()
    want = _region_mean(imgs, 33, 2)
    m = ctypes.c_double()
    r = np.zeros(17)
    st = hb.load().fd2_nnps(0, ptr(imgs), n, 35, 70, 1.0, 33, 0, 0, 1, 2, 17, None, ptr(r), None,
                            ctypes.byref(m))
    assert st == (0 if want > 0.0 else INVALID)
    if st == 0:
        assert m.value == want
