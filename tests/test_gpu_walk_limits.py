"""Walks at the edge of what FP32 can hold: columns of a thousandth of a
micrometre and less, where a photon on its column's axis gets a direction that
is no number.  Such a photon still goes down to the sensor; the tallies here are
those of the walk as first written."""
import numpy as np
import pytest

import hybridmantis_b200 as hb

pytestmark = pytest.mark.gpu

FATES = ("detected", "abs_top", "abs_bulk", "lost", "outofcol", "theta1", "capped")
TALLIES = {2e-5: (17, 0, 0, 30, 4753, 0, 0), 1e-4: (3, 0, 0, 4, 4788, 5, 0), 1e-3: (7, 0, 0, 29, 2957, 1807, 0)}


@pytest.mark.parametrize("radius", sorted(TALLIES))
@pytest.mark.parametrize("radial", [0, 9])
def test_fates_in_vanishing_columns(require_gpu, radius, radial):
    n, photons = 60, 40
    p = hb.default_params(num_hist=n)
    p.radius, p.sensor_refl = radius, 0.3
    r = np.random.default_rng(n)
    x = r.uniform(0.1 * p.det_x, 0.9 * p.det_x, n).astype(np.float32)
    y = r.uniform(0.1 * p.det_x, 0.9 * p.det_x, n).astype(np.float32)
    z = (p.det_height * r.uniform(-0.495, 0.495, n)).astype(np.float32)
    with hb.OpticalTransport(p, count_mode=hb.COUNT_GIVEN, seed=8, radial_bins=radial) as t:
        t.submit_events_um(x, y, z, np.full(n, 1e4), np.arange(1, n + 1), np.full(n, photons))
        t.run_sync()
        t.run_sync()
        c = t.counters()
    assert c["generated"] == 2 * n * photons
    assert tuple(c[f] for f in FATES) == TALLIES[radius]
