"""Which runs take the reduced grid of a small submission, and which must not."""
import time

import numpy as np
import pytest
import torch

import hybridmantis_b200 as hb

pytestmark = pytest.mark.gpu


def _submit_small(t, es):
    t.submit(es)
    t.run_sync()
    return t.timing()["grid"] // torch.cuda.get_device_properties(0).multi_processor_count


def test_an_ingest_takes_the_full_grid_after_a_small_submission(require_gpu):
    es = hb.synth_events(1, 25, 8)
    x, y, z = es.to_cm()
    with hb.OpticalTransport(es.params, seed=9) as t:
        assert _submit_small(t, es) == 2
        with t.ingest(batch_events=4096) as ing:
            ing.push(x, y, z, es.e_ev.astype(np.float64), es.hist)
            time.sleep(0.2)  # the ingest's first events on the stream are done
            per_sm = t.timing()["grid"] // torch.cuda.get_device_properties(0).multi_processor_count
        assert per_sm == 4


@pytest.mark.parametrize("block,per_sm", [(0, 2), (32, 4), (64, 4), (128, 4), (256, 4)])
def test_a_given_block_size_keeps_the_full_grid(require_gpu, block, per_sm):
    with hb.OpticalTransport(hb.synth_events(1, 25, 8).params, seed=9, block_size=block) as t:
        assert _submit_small(t, hb.synth_events(1, 25, 8)) == per_sm


def test_new_geometries_end_a_tuned_launch_shape(require_gpu):
    es = hb.synth_events(1, 25, 8)
    with hb.OpticalTransport(es.params, seed=9) as t:
        t.submit(es)
        t.autotune(budget_runs=2)  # keeps the shape it starts with, on the full grid
        assert _submit_small(t, es) == 4
        t.set_geometries([hb.params_to_geometry(es.params)])
        assert _submit_small(t, es) == 2
