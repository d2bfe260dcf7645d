"""The simulation kernel's register tiles and launch tiers where they end:
regions that just fill or just miss a tile, batches larger than one wave whose
simulations run on both tiers side by side, lists longer than the on-chip
clocks, and cells in every class of the cell loop.  Exact throughout: the
tiles, tiers, schedules and layouts only change where a site is computed, so
nothing is to differ by a bit."""
import numpy as np
import pytest

from test_gpu_units import _diffusion_parity

pytestmark = pytest.mark.gpu

# the tiles' columns and rows per lane; a tile holds 4R x 8C sites
_TILES = [(1, 2), (2, 3), (2, 4), (3, 5), (3, 6), (4, 7), (4, 8), (5, 9), (5, 10), (6, 11),
          (6, 12), (7, 13), (7, 14), (8, 14)]


@pytest.mark.parametrize("tile", range(len(_TILES)))
def test_regions_that_fill_a_tile(tile, params, oracle):
    """One diffusion step on lattices that are one region: as large as the
    tile, one row or column less, one more (the next tile), and flat ones."""
    C, R = _TILES[tile]
    rng = np.random.default_rng(4100 + tile)
    for h, w in [(4 * R, 8 * C), (4 * R - 1, 8 * C), (4 * R, 8 * C - 1), (4 * R + 1, 8 * C),
                 (4 * R, 8 * C + 1), (4 * R, 3), (3, 8 * C)]:
        h, w = min(h, 56), min(w, 62)
        st = np.full((h, w), 2, np.uint8)
        st[1:-1, 1:-1] = rng.random((h - 2, w - 2)) < 0.9
        st[1:-1:max(h - 3, 1), 1:-1:max(w - 3, 1)] = 1  # the corners
        _diffusion_parity(st, rng, params, oracle)


def _tumour(params, r, seed):
    """A disc whose cells are in every phase and class: clocks before, at and
    past the end of their phase or cycle, under repair, first phases longer
    than the cycle."""
    from emt6ro import workloads as wl
    t = wl.disc_tumor(params, r, seed=seed)
    s = t.sites
    rng = np.random.default_rng(seed)
    live = s["state"] == 1
    n = int(live.sum())
    ct = s["cycle_times"][live]
    ct[rng.random(n) < 0.05, 0] = 40.0
    s["cycle_times"][live] = ct
    phase = rng.integers(0, 5, n)
    s["phase"][live] = phase
    s["mode"][live] = rng.integers(0, 4, n)
    end = ct[np.arange(n), phase]
    s["proliferation_time"][live] = np.where(rng.random(n) < 0.1, end, end * rng.random(n))
    hurt = live & (rng.random(s.shape) < 0.2)
    k = int(hurt.sum())
    s["irradiation"][hurt] = rng.integers(1, 17, k).astype(np.float32) * np.float32(0.25)
    s["repair_delay_time"][hurt] = 4.0
    s["time_in_repair"][hurt] = 4.0 * rng.random(k)
    return t


@pytest.mark.parametrize("schedule,layouts", [(0, 7), (1, 7), (2, 7), (3, 0)])
def test_tiers_side_by_side(schedule, layouts, params, oracle):
    """1,400 simulations (more than one wave) of radii 1 to 24 on both tiers:
    the first ones equal the oracle, others equal batches that are one wave,
    whose runs are once short (tiers in turn), once long (side by side)."""
    from emt6ro.batch import Batch
    n, chunks, seed = 1400, [70, 20, 60], 71
    tumors = [_tumour(params, r, 700 + r) for r in (1, 5, 9, 14, 15, 16, 17, 19, 21, 24)]
    protocols = [[(0, 1.5)], [(0, 0.75)], []]
    i = np.arange(n)
    st, sp = (i % 10).astype(np.int32), (i % 3).astype(np.int32)
    hz = np.where(i % 7 == 3, i % 97, 1000).astype(np.uint32)
    b = Batch(params, tumors, protocols, st, sp, sim_horizon=hz, seed=seed)
    b.set_schedule(schedule, 0)
    b.set_layouts(layouts)
    for c in chunks:
        b.run(c)
    counts = b.counts()

    k = 20
    ob = oracle.Batch(oracle.params_copy(params.native), k, seed)
    for j in range(k):
        ob.set(j, tumors[st[j]].sites, b.doses[sp[j]], resolution=300, length=144_000,
               horizon=int(hz[j]))
    ob.run(sum(chunks), nthreads=8)
    assert (counts[:k] == ob.counts()).all()
    for j in range(k):
        assert b.state(j).sites.tobytes() == ob.get(j).tobytes(), j

    for base, parts in ((600, chunks), (1300, [50, 50, 50])):
        m = slice(base, base + 100)
        small = Batch(params, tumors, protocols, st[m], sp[m], sim_horizon=hz[m], seed=seed)
        small.set_index_base(base)
        for c in parts:
            small.run(c)
        assert (small.counts() == counts[m]).all()
        for j in range(0, 100, 9):
            assert small.state(j).sites.tobytes() == b.state(base + j).sites.tobytes(), j


@pytest.mark.parametrize("dims", [(51, 51), (54, 60), (49, 50)])
def test_large_regions_on_every_tier(dims, oracle):
    """Regions of 45 to 56 rows, centred and clipped, with an SM each, as part of
    a batch that is one wave, and of a larger one: the oracle's lattices."""
    from emt6ro import workloads as wl
    from emt6ro.batch import Batch
    params = wl.default_parameters()
    params.native.lattice_height, params.native.lattice_width = dims
    h, w = dims[0] + 2, dims[1] + 2
    tumors = [wl.disc_tumor(params, r, seed=40 + k, center=(h // 2 + dr, w // 2 + dc))
              for k, (r, dr, dc) in enumerate([(21, 0, 0), (22, 0, 1), (23, 0, 0), (24, 0, 0),
                                               (24, 3, -2), (26, -4, 5), (20, 9, 0), (27, 0, 0)])]
    steps, k = 70, len(tumors)
    ob = oracle.Batch(oracle.params_copy(params.native), k, 9)
    batches = [Batch(params, tumors, [[(0, 0.5)]], np.arange(n) % k, np.zeros(n, np.int32), seed=9)
               for n in (k, 300, 700)]
    for j in range(k):
        ob.set(j, tumors[j].sites, batches[0].doses[0], resolution=300, length=144_000)
    ob.run(steps, nthreads=8)
    for b in batches:
        b.run(steps)
        assert (b.counts()[:k] == ob.counts()).all()
        for j in range(k):
            assert b.state(j).sites.tobytes() == ob.get(j).tobytes(), (b.n, j)


@pytest.mark.parametrize("n", [8, 160, 700])
def test_cells_on_a_vacant_far_border_count_for_the_region(n, params, oracle):
    """A lattice whose last row and column are vacant, not mocked: cells divide
    onto them and leave the list at its next rebuild, but stay in the region."""
    from emt6ro import workloads as wl
    from emt6ro.batch import Batch
    tumors = []
    for k, center in enumerate([(50, 50), (51, 26), (26, 51), (51, 12)]):
        t = wl.disc_tumor(params, 6, seed=300 + k, center=center)
        s = t.sites
        s["state"][-1, 1:] = 0
        s["state"][1:, -1] = 0
        live = s["state"] == 1  # divide in the steps before the rebuild at step 128
        rng = np.random.default_rng(k)
        s["phase"][live] = 3
        s["proliferation_time"][live] = (s["cycle_times"][live][:, 3] - 0.17
                                         - 0.04 * rng.random(live.sum()))
        tumors.append(t)
    steps, k = 300, 8
    st = np.arange(n) % 4
    b = Batch(params, tumors, [[]], st, np.zeros(n, np.int32), seed=6)
    b.run(steps)
    ob = oracle.Batch(oracle.params_copy(params.native), k, 6)
    for j in range(k):
        ob.set(j, tumors[st[j]].sites, b.doses[0], resolution=300, length=144_000)
    ob.run(steps, nthreads=8)
    left_out = [np.setdiff1d(np.flatnonzero(ob.get(j)["state"] == 1), ob.occupied_list(j))
                for j in range(k)]
    assert sum(map(len, left_out)) > 10
    assert (b.counts()[:k] == ob.counts()).all()
    for j in range(k):
        assert b.state(j).sites.tobytes() == ob.get(j).tobytes(), j


@pytest.mark.parametrize("dims,radii,n,schedule,launches", [
    ((51, 51), (5, 24, 26, 36), 200, 0, (5, 3)),   # two simulations per SM
    ((51, 51), (20, 22, 23, 24), 260, 2, (5, 3)),  # too many others for the SMs left
    ((51, 51), (5, 12, 17, 20), 200, 2, (4, 1)),   # no large region
    ((51, 51), (5, 24, 26, 36), 400, 0, (4, 1)),   # more per SM
    ((51, 51), (5, 24, 26, 36), 700, 1, (6, 6)),
    ((54, 60), (6, 26, 27, 40), 200, 3, (5, 3)),
    ((54, 60), (6, 26, 27, 40), 400, 0, (5, 3)),   # the largest tile alone
    ((54, 60), (6, 24, 27, 40), 500, 2, (7, 7)),   # four per SM
    ((54, 60), (6, 26, 27, 40), 700, 0, (7, 7)),
    ((54, 60), (6, 26, 27, 40), 700, 1, (7, 7)),
    ((54, 60), (6, 26, 27, 40), 700, 3, (7, 7)),
    ((54, 60), (6, 20, 23, 25), 700, 0, (6, 6))])  # no region of the largest tile
def test_large_regions_in_turns_beside_the_other_tiers(dims, radii, n, schedule, launches, oracle):
    """The lone tier's part of a split launch: launches of a long and a short run,
    and the oracle's lattices."""
    from emt6ro import workloads as wl
    from emt6ro.batch import Batch
    params = wl.default_parameters()
    params.native.lattice_height, params.native.lattice_width = dims
    tumors = [wl.disc_tumor(params, r, seed=80 + r) for r in radii]
    st, k = np.arange(n) % 4, 8
    b = Batch(params, tumors, [[(0, 0.5)]], st, np.zeros(n, np.int32), seed=13)
    b.set_schedule(schedule, 0)
    before, count = b.launches(), []
    for steps in (70, 20):
        b.run(steps)
        count.append(b.launches() - before)
        before = b.launches()
    ob = oracle.Batch(oracle.params_copy(params.native), k, 13)
    for j in range(k):
        ob.set(j, tumors[st[j]].sites, b.doses[0], resolution=300, length=144_000)
    ob.run(90, nthreads=8)
    assert (b.counts()[:k] == ob.counts()).all()
    for j in range(k):
        assert b.state(j).sites.tobytes() == ob.get(j).tobytes(), j
    assert tuple(count) == launches


def test_a_tumour_that_shrank_is_expected_on_the_narrow_tier(params):
    """A disc too large for the narrow tier whose outer cells die of age: from then
    on, its own list and region decide, not the initial tumour's cells."""
    from emt6ro import _native as N
    from emt6ro import workloads as wl
    from emt6ro.batch import Batch
    big, small = (wl.disc_tumor(params, r, seed=5) for r in (23, 6))
    s = big.sites
    rr, cc = np.mgrid[0:53, 0:53]
    outer = (s["state"] == 1) & ((rr - 26) ** 2 + (cc - 26) ** 2 > 36)
    s["proliferation_time"][outer] = s["cycle_times"][outer][:, 4] + 1
    n = 300
    b = Batch(params, [big, small], [[]], np.arange(n) % 2, np.zeros(n, np.int32), seed=2)

    def tiers():
        out = np.zeros(n, np.uint8)
        N.check(N.lib().emt6_test_batch_tiers(b._h, N.ptr(out)))
        return out[:2].tolist()
    assert tiers() == [1, 0]
    b.run(200)
    assert tiers() == [0, 0]
    b.reset()
    assert tiers() == [1, 0]


@pytest.mark.parametrize("dims,radii,n,schedule,launches", [
    ((54, 60), (6, 12, 18, 22), 500, 1, 1),   # wide alone, though not all resident
    ((54, 60), (6, 24, 27, 40), 500, 3, 3),   # the largest tile beside it
    ((51, 51), (6, 24, 26, 36), 200, 0, 1),   # large, but too few steps
    ((51, 51), (6, 12, 18, 22), 608, 1, 1),
    ((54, 60), (6, 12, 18, 22), 700, 1, 6)])
def test_runs_of_single_steps(dims, radii, n, schedule, launches, oracle):
    """Recordings of every step: launches per run and the oracle's lattices."""
    from emt6ro import workloads as wl
    from emt6ro.batch import Batch
    params = wl.default_parameters()
    params.native.lattice_height, params.native.lattice_width = dims
    tumors = [wl.disc_tumor(params, r, seed=60 + r) for r in radii]
    st, k, steps = np.arange(n) % 4, 8, 36
    b = Batch(params, tumors, [[(0, 0.5)]], st, np.zeros(n, np.int32), seed=14)
    b.set_schedule(schedule, 0)
    before = b.launches()
    for _ in range(steps):
        b.run(1)
    assert b.launches() - before == launches * steps
    ob = oracle.Batch(oracle.params_copy(params.native), k, 14)
    for j in range(k):
        ob.set(j, tumors[st[j]].sites, b.doses[0], resolution=300, length=144_000)
    ob.run(steps, nthreads=8)
    for j in range(k):
        assert b.state(j).sites.tobytes() == ob.get(j).tobytes(), j
