"""Waiting photons parked in shared memory (transport_kernel): the tallies do
not depend on how many photons wait before the warp runs them, on the refill
threshold or on the launch shape.  With fresnel_batch = 1 no photon leaves its
lane; the sizes go from one photon through runs with fewer photons than lanes
and than one refill to several refills per warp."""
import numpy as np
import pytest

import hybridmantis_b200 as hb

pytestmark = pytest.mark.gpu

LAUNCHES = [dict(fresnel_batch=1, refill=1), dict(), dict(fresnel_batch=32, refill=1),
            dict(fresnel_batch=2, refill=32), dict(fresnel_batch=31, refill=3, block_size=64, ctas_per_sm=1),
            dict(fresnel_batch=32, chunk=1, block_size=128, ctas_per_sm=8)]


@pytest.mark.parametrize("grid,radial,geoms", [(0, 0, 1), (1, 0, 1), (2, 0, 1), (0, 24, 1), (0, 0, 3), (0, 24, 3)])
@pytest.mark.parametrize("events,photons", [(1, 1), (3, 11), (40, 1), (977, 37)])
def test_tallies_do_not_depend_on_parking(require_gpu, grid, radial, geoms, events, photons):
    rng = np.random.default_rng(events)
    p = hb.default_params(num_hist=events, det_height=300.0, sensor_refl=0.25)
    g = []
    for k in range(geoms):
        q = hb.params_to_geometry(p)
        q.radius, q.top_absfrac = 5.0 + k, 0.1 * k
        g.append(q)
    args = (rng.uniform(100, 400, events), rng.uniform(100, 400, events), rng.uniform(-149, 149, events),
            np.full(events, 1e4), np.arange(1, events + 1), np.full(events, photons),
            np.arange(events) % geoms if geoms > 1 else None)
    first = None
    for kw in LAUNCHES:
        if grid or radial:
            kw = {k: v for k, v in kw.items() if k != "ctas_per_sm"}
        with hb.OpticalTransport(p, count_mode=hb.COUNT_GIVEN, seed=8, column_grid=grid, radial_bins=radial, **kw) as t:
            if geoms > 1:
                t.set_geometries(g)
            t.submit_events_um(*args)
            t.run_sync()
            got = [t.detected_per_primary()] + ([t.radial()] if radial else [t.prf(k) for k in range(geoms)])
            counts = [{k: v for k, v in t.counters(j).items() if k != "photon_distance"} for j in range(geoms)]
        assert sum(c["generated"] for c in counts) == events * photons
        if first is None:
            first = (got, counts)
        assert all(np.array_equal(a, b) for a, b in zip(first[0], got)), kw
        assert counts == first[1], kw


@pytest.mark.parametrize("grid", [1, 2])
@pytest.mark.parametrize("events,photons", [(1, 1), (151, 701)])
def test_lattice_tallies_do_not_depend_on_the_kernel(require_gpu, grid, events, photons):
    """Each register budget of the lattice kernel walks the same photons."""
    rng = np.random.default_rng(events)
    p = hb.default_params(num_hist=events, det_height=300.0, sensor_refl=0.25)
    args = (rng.uniform(100, 400, events), rng.uniform(100, 400, events), rng.uniform(-149, 149, events),
            np.full(events, 1e4), np.arange(1, events + 1), np.full(events, photons))
    first = None
    for kw in (dict(), dict(ctas_per_sm=4, chunk=3), dict(ctas_per_sm=3), dict(ctas_per_sm=2),
               dict(block_size=320, ctas_per_sm=2)):
        with hb.OpticalTransport(p, count_mode=hb.COUNT_GIVEN, seed=8, column_grid=grid, **kw) as t:
            t.submit_events_um(*args)
            t.run_sync()
            c = t.counters()
            got = (t.detected_per_primary(), t.prf(0), np.array([v for k, v in c.items() if k != "photon_distance"]))
        assert c["generated"] == events * photons
        first = first or got
        assert all(np.array_equal(a, b) for a, b in zip(first, got)), kw
