"""Label mode under every launch shape the options accept: one geometry has one
kernel whatever ctas_per_sm says, several geometries another, and neither the
labels nor the path lengths depend on the shape."""
import os

import numpy as np
import pytest

import hybridmantis_b200 as hb
from hybridmantis_b200 import surrogate as sgm

pytestmark = pytest.mark.gpu

MODEL = os.path.join(os.path.dirname(sgm.__file__), "data", "surrogate_c4.fd2sg")


def _case(geoms, events=977, photons=37):
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
    return p, g, args


def _result(t, geoms):
    counts = [t.counters(k) for k in range(geoms)]
    path = np.array([c.pop("photon_distance") for c in counts])
    return t.radial(), t.detected_per_primary(), counts, path


def _same(a, b, what):
    assert np.array_equal(a[0], b[0]) and np.array_equal(a[1], b[1]), what
    assert a[2] == b[2], what
    # a lane or a CTA adds fewer than 2,000 flights in FP32 (2^-24 of the sum
    # each, at worst all one way), the rest is FP64
    assert np.allclose(a[3], b[3], rtol=2000 * 2.0 ** -24), what


@pytest.mark.parametrize("geoms", [1, 3])
@pytest.mark.parametrize("block", [0, 64])
def test_labels_do_not_depend_on_the_launch_shape(require_gpu, geoms, block):
    p, g, args = _case(geoms)
    first = None
    for ctas in (0, 1, 2, 3, 4, 8):
        with hb.OpticalTransport(p, count_mode=hb.COUNT_GIVEN, seed=8, radial_bins=24, ctas_per_sm=ctas,
                                 block_size=block) as t:
            if geoms > 1:
                t.set_geometries(g)
            t.submit_events_um(*args)
            t.run_sync()
            got = _result(t, geoms)
        assert sum(c["generated"] for c in got[2]) == 977 * 37
        first = first or got
        _same(first, got, (ctas, block))


@pytest.mark.parametrize("geoms", [1, 3])
def test_labels_after_autotuning(require_gpu, geoms):
    p, g, args = _case(geoms)
    with hb.OpticalTransport(p, count_mode=hb.COUNT_GIVEN, seed=8, radial_bins=24) as t:
        if geoms > 1:
            t.set_geometries(g)
        t.submit_events_um(*args)
        t.run_sync()
        want = _result(t, geoms)
        t.autotune()  # tries 256 x 3 and 256 x 2 among others, then clears the tallies
        t.submit_events_um(*args)
        t.run_sync()
        _same(want, _result(t, geoms), "tuned")


@pytest.mark.parametrize("ctas", [1, 2, 3, 4])
def test_audit_does_not_depend_on_the_callers_launch_shape(require_gpu, ctas):
    """The audit's label context takes over the caller's options."""
    es = hb.synth_events(4, 40, 5)
    stats = []
    for k in (0, ctas):
        with sgm.Surrogate() as s, hb.OpticalTransport(es.params, seed=11, ctas_per_sm=k) as t:
            s.load(MODEL)
            t.submit(es)
            stats.append(s.run(t, 0.5))
    assert stats[0]["audit_events"] > 0 and stats[0]["audit_mc_detected"] > 0
    for key in ("audit_events", "audit_mc_detected"):
        assert stats[0][key] == stats[1][key]
