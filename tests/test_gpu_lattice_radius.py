"""Histories in the square lattice with radii whose square is not an FP32 number.
The wall test of a flight through the gap subtracts the rounded square; fused
into the sum it moved a wall by a last bit, which a column billiard turns into
another history.  The tallies here are those of the lattice kernel as first
written; every launch shape walks the same histories."""
import numpy as np
import pytest

import hybridmantis_b200 as hb

pytestmark = pytest.mark.gpu

# radius (um): detected, absorbed at the top, absorbed in bulk, lost
TALLIES = {0.05: (9538, 7550, 168, 2744), 0.1: (7115, 10733, 394, 1758), 0.2: (6355, 11815, 741, 1089),
           0.3: (7246, 10962, 921, 871)}


@pytest.mark.parametrize("radius", sorted(TALLIES))
@pytest.mark.parametrize("launch", [dict(), dict(ctas_per_sm=3), dict(ctas_per_sm=2),
                                    dict(block_size=320, ctas_per_sm=2)])
def test_square_lattice_of_thin_columns(require_gpu, radius, launch):
    n, photons = 100, 100
    p = hb.default_params(num_hist=n)
    p.radius = radius
    r = np.random.default_rng(n)
    x = r.uniform(0.1 * p.det_x, 0.9 * p.det_x, n).astype(np.float32)
    y = r.uniform(0.1 * p.det_x, 0.9 * p.det_x, n).astype(np.float32)
    z = (p.det_height * r.uniform(-0.495, 0.495, n)).astype(np.float32)
    with hb.OpticalTransport(p, count_mode=hb.COUNT_GIVEN, seed=8, column_grid=1, **launch) as t:
        t.submit_events_um(x, y, z, np.full(n, 1e4), np.arange(1, n + 1), np.full(n, photons))
        t.run_sync()
        t.run_sync()  # and another hundred each
        c = t.counters()
    assert c["generated"] == 2 * n * photons
    assert (c["detected"], c["abs_top"], c["abs_bulk"], c["lost"]) == TALLIES[radius]
