"""The whole-simulation parity tests on every route of a run.  Their batches have
an SM per simulation, and so take the lone tier alone; here the same cases run as
the parts of larger batches do: on the wide tier alone, on the narrow and wide
tiers side by side, the same in launch order (and over the work queue), and with
large regions on the lone tier beside them."""
import numpy as np
import pytest

import test_gpu_simulation as ts

pytestmark = pytest.mark.gpu

# route of emt6_test_batch_route -> its launches per chunk of steps
_ROUTES = {1: (1,), 2: (1,), 3: (4,), 4: (6,), 5: (6, 7)}


@pytest.fixture(params=sorted(_ROUTES))
def routed(request, monkeypatch):
    """emt6ro.batch.Batch on one route, which checks its launches at each run."""
    from emt6ro import _native as N
    from emt6ro import batch
    per, runs = _ROUTES[request.param], []

    class Routed(batch.Batch):
        chunk = 1200

        def __init__(self, *args, sim_horizon=None, **kw):
            super().__init__(*args, sim_horizon=sim_horizon, **kw)
            N.check(N.lib().emt6_test_batch_route(self._h, request.param))
            self.last = None if sim_horizon is None else int(np.max(sim_horizon))
            self.at = 0

        def set_schedule(self, mode, steps_per_launch=0):
            super().set_schedule(mode, steps_per_launch)
            self.chunk = steps_per_launch or self.chunk

        def reset(self):
            super().reset()
            self.at = 0

        def run(self, nsteps):
            before = self.launches()
            super().run(nsteps)
            starts = range(self.at, self.at + nsteps, self.chunk)
            chunks = sum(self.last is None or t < self.last for t in starts)
            self.at += nsteps
            assert per[0] * chunks <= self.launches() - before <= per[-1] * chunks
            runs.append(chunks)

    monkeypatch.setattr(batch, "Batch", Routed)
    yield request.param
    assert sum(runs) > 0


@pytest.mark.parametrize("case", [
    ts.test_small_batch_bit_exact, ts.test_tumours_against_the_lattice_edge_bit_exact,
    ts.test_empty_and_single_cell_lattices_bit_exact, ts.test_chunked_runs_equal_one_run,
    ts.test_wide_regions_bit_exact, ts.test_33_wide_regions_bit_exact,
    ts.test_35_wide_regions_bit_exact, ts.test_growing_and_shrinking_discs_bit_exact,
    ts.test_ragged_horizons_and_queue, ts.test_graph_replay_and_queue_bit_exact,
    ts.test_reset_gives_fresh_epoch, ts.test_diffused_counter_matches_oracle,
    ts.test_summary_and_timelapse_match_oracle_states, ts.test_one_day_bit_exact],
    ids=lambda f: f.__name__[5:])
def test_case(case, routed, params, oracle):
    case(params, oracle)


@pytest.mark.parametrize("dims", [(40, 47), (54, 60)])
def test_other_lattice_sizes(dims, routed, oracle):
    ts.test_other_lattice_sizes_bit_exact(oracle, dims)


@pytest.mark.parametrize("layouts", [0, 3, 4, 7])
def test_tile_shape_sets(layouts, routed, params, oracle):
    ts.test_every_tile_shape_set_bit_exact(params, oracle, layouts)
