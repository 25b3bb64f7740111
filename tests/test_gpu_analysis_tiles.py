"""MTF and NNPS where the transform kernels' tiles end (32 rows, 32 column
frequencies, 16 row frequencies, chunks of 32 terms), odd regions, regions
that leave part of the image out, and calls from several threads."""
import threading

import numpy as np
import pytest

from hybridmantis_b200 import analysis
from oracle import analysis_oracle as ao

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape,freqs", [((1, 1), 1), ((2, 3), 2), ((31, 33), 17), ((32, 32), 16), ((33, 31), 17),
                                         ((64, 17), 33), ((17, 129), 65), ((130, 97), 40)])
def test_mtf_at_tile_edges(require_gpu, shape, freqs):
    img = np.random.default_rng(sum(shape)).gamma(2.0, 3.0, shape)
    got = analysis.mtf(img, 1.5, freqs)
    _, mx, my, mr = ao.mtf(img, 1.5, freqs)
    for a, b in ((got["mtf_x"], mx), (got["mtf_y"], my), (got["mtf_r"], mr)):
        assert np.allclose(a, b, rtol=1e-9, atol=1e-12)


@pytest.mark.parametrize("n,roi,rx,ry,x0,y0", [(1, 2, 1, 1, 0, 0), (2, 3, 2, 1, 1, 4), (1, 31, 1, 2, 3, 0),
                                               (3, 32, 2, 2, 0, 1), (2, 33, 1, 1, 30, 2), (5, 64, 1, 1, 0, 0),
                                               (2, 65, 1, 1, 1, 1)])
def test_nnps_at_tile_edges(require_gpu, n, roi, rx, ry, x0, y0):
    imgs = np.random.default_rng(roi).poisson(200.0, (n, 70, 68)).astype(np.float64)
    k = roi // 2 + 1
    got = analysis.nnps(imgs, 2.0, roi, x0, y0, rx, ry, k)
    _, nr, n2, m = ao.nnps(imgs, 2.0, roi, x0, y0, rx, ry, k)
    assert got["mean_signal"] == pytest.approx(m, rel=1e-12)
    # a single image's zero frequency is rounding noise: absolute to the map's scale
    assert np.allclose(got["nnps_2d"], n2, rtol=1e-9, atol=1e-12 * n2.max())
    assert np.allclose(got["nnps_r"], nr, rtol=1e-9, atol=1e-12 * n2.max())


def test_calls_from_several_threads(require_gpu):
    rng = np.random.default_rng(3)
    imgs = [rng.gamma(2.0, 3.0, (90 + i, 70)) for i in range(4)]
    want = [ao.mtf(im, 1.0, 20)[3] for im in imgs]
    bad = []

    def work(i):
        for _ in range(20):
            if not np.allclose(analysis.mtf(imgs[i], 1.0, 20)["mtf_r"], want[i], rtol=1e-9):
                bad.append(i)

    threads = [threading.Thread(target=work, args=(i,)) for i in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad
