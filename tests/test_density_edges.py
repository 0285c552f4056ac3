"""The density pass where its fp16 candidate test and its staged halo are
tightest: pairs just inside and outside the support radius far from a region's
centre, and targets that have drifted out of their brick since the sort.  Lists
are those of the per-target global path, entry by entry."""
import numpy as np
import pytest

from sph_cuda_gb300 import Asph, preset
from statebuild import random_state, reference_geometry, small_config

FTHR = 4.0390625     # the walk's threshold on the fp16 squared distance
CLAMP = 7.9          # a coordinate's largest distance from the region's centre, in cells


def _fp16_r2(a, b):
    """The walk's squared distance of points given in cells from the region's centre."""
    r2 = None
    for k in range(3):
        x, y = (np.clip(p[:, k], -CLAMP, CLAMP).astype(np.float32).astype(np.float16) for p in (a, b))
        d = (x - y).astype(np.float64)   # one fp16 rounding, then fused products
        r2 = (d * d if r2 is None else d * d + r2.astype(np.float64)).astype(np.float16)
    return r2


def _edge_pairs(rng, n, lo, hi, slack):
    """Points with every coordinate between lo and hi cells from the centre, and
    partners further out at a distance of 2 - slack to 2 cells."""
    sign = rng.choice([-1.0, 1.0], (n, 3))
    a = sign * rng.uniform(lo, hi, (n, 3))
    d = np.abs(rng.normal(size=(n, 3)))
    d *= ((2.0 - rng.uniform(0.0, slack, n)) / np.linalg.norm(d, axis=1))[:, None]
    return a, a + sign * d


def test_threshold_passes_every_pair_inside():
    rng = np.random.default_rng(5)
    largest = 0.0
    for lo, hi in ((0.0, 4.0), (3.9, 4.1), (4.0, 5.9), (5.5, 6.5), (6.0, 9.0)):
        a, b = _edge_pairs(rng, 400000, lo, hi, 0.01)
        r2 = _fp16_r2(a, b)
        assert float(r2.max()) <= FTHR
        largest = max(largest, float(r2.max()))
    assert largest > 4.0   # the pairs probe the rounding: a threshold of 4 would drop some


@pytest.mark.gpu
@pytest.mark.parametrize("shape", [0, 1, 2, 3])
@pytest.mark.parametrize("n,drift", [(12000, 0.0), (12000, 0.95), (84672, 0.0), (84672, 0.3)])
def test_pairs_at_the_support_radius(shape, n, drift):
    """3,000 pairs at 1.99 to 2.01 cells whose first point sits in a corner of a
    brick, among uniform points, up to the wide halo's drift later; below and above
    77,824 targets."""
    grid, cell, m = (64, 64, 56), (200.0, 200.0, 50.0), 3000
    p = small_config(lat=(n, 1, 1), grid=grid, box=tuple(g * c for g, c in zip(grid, cell)), sort_every=1)
    rng = np.random.default_rng(11 + shape)
    brick = (8, 8, 8) if shape == 0 else (8, 8, 4) if shape == 1 else (8, 4, 4) if shape == 2 else (4, 4, 4)
    # brick centres with a brick between them and the box's edge
    centre = np.stack([(rng.integers(1, grid[k] // brick[k] - 1, m) + 0.5) * brick[k] for k in range(3)], axis=1)
    sign = rng.choice([-1.0, 1.0], (m, 3))
    a = centre + sign * (0.5 * np.array(brick) - rng.uniform(1e-3, 0.5, (m, 3)))
    d = np.abs(rng.normal(size=(m, 3)))
    d *= (rng.uniform(1.99, 2.01, m) / np.linalg.norm(d, axis=1))[:, None]
    pos = np.concatenate([a, a + sign * d, rng.uniform(0.0, 1.0, (n - 2 * m, 3)) * grid]) * cell
    s = random_state(p, 3, "uniform")
    for k, f in enumerate("xyz"):
        s[f] = pos[:, k].astype(np.float32)
    for f in ("ax", "ay", "az"):
        s[f] = np.zeros(n, np.float32)
    lists = []
    for path in (0, 1):
        with Asph(p) as sim:
            if path == 0:
                sim.set_pair_shape(shape)
            sim.set_pair_path(path)
            dt = sim.control()["dt"]
            for f, c in zip("uvw", cell):
                s[f] = np.full(n, drift * c / dt, np.float32)
            sim.set_state(s)
            sim.sort_build()
            if drift:
                sim.kick_drift_flux()
            sim.density_eos()
            lists.append(sim.neighbours())
    (cnt, lst), (cnt_g, lst_g) = lists
    assert np.array_equal(cnt, cnt_g)
    used = np.arange(lst.shape[0])[:, None] < np.maximum(cnt, 0)[None, :]
    assert np.array_equal(lst[used], lst_g[used])


# Every target moved by the same fraction of a cell along x since the sort: the
# narrow halo (sorts every step or gated, above 77,824 targets) covers those
# that are still in a cell of their brick, the wide one all of them.
@pytest.mark.gpu
@pytest.mark.parametrize("shape,edge", [(0, 8), (1, 8), (2, 8), (3, 4)])
@pytest.mark.parametrize("cadence,n3,narrow", [(0, (48, 42, 42), True), (1, (48, 42, 42), True),
                                               (4, (48, 42, 42), False), (0, (48, 42, 38), False)])
def test_halo_follows_the_cadence_and_the_size(shape, edge, cadence, n3, narrow):
    drift = 0.25
    p = small_config(lat=n3, grid=(48, 40, 40), box=(9600.0, 8000.0, 2000.0), sort_every=cadence)
    s = random_state(p, 7, "uniform")
    with Asph(p) as sim:
        sim.set_pair_shape(shape)
        dt = sim.control()["dt"]
        for f in ("v", "w", "ax", "ay", "az"):
            s[f] = np.zeros(p.n_particles, np.float32)
        s["u"] = np.full(p.n_particles, drift * 200.0 / dt, np.float32)
        sim.set_state(s)
        sim.sort_build()
        sim.kick_drift_flux()
        sim.density_eos()
        deferred = sim.control()["deferred"]
    left = drift / edge * p.n_particles   # uniform positions: the share of a brick within `drift` of its end
    if narrow:
        assert 0.9 * left < deferred < 1.1 * left
    else:
        assert deferred == 0


@pytest.mark.gpu
@pytest.mark.parametrize("shape,brick", [(0, (8, 8, 8)), (1, (8, 8, 4)), (2, (8, 4, 4)), (3, (4, 4, 4))])
def test_gated_sorts_above_the_wide_halos_size(shape, brick):
    """The displacement-gated cadence on the narrow halo, steps after the last sort:
    lists of the global path, and no more targets deferred than can have left
    their brick.  A sort comes after about 0.3 cells of the fastest particle's way, the
    last step's own way comes on top (below 0.2 cells at these speeds)."""
    p = reference_geometry(48, 44, 40)
    assert p.sort_every == 0 and p.n_particles > 77824
    s = random_state(p, 13, "jitter", speed=8.0)
    with Asph(p) as sim:
        sim.set_pair_shape(shape)
        sim.set_state(s)
        sim.sort_build()
        sim.step(1)
        between = 0
        for _ in range(12):
            sorts = sim.control()["sort_count"]
            sim.step(1)
            c = sim.control()
            stayed = np.prod([1.0 - min(1.0, 0.5 / b) for b in brick])
            assert c["deferred"] <= (1.0 - stayed) * p.n_particles
            if c["sort_count"] != sorts:
                continue
            between += 1
            snap = sim.snapshot()
            lists = []
            for path in (0, 1):
                sim.set_pair_path(path)
                sim.density_eos()
                lists.append(sim.neighbours())
                sim.restore(snap)
            snap.close()
            sim.set_pair_path(0)
            (cnt, lst), (cnt_g, lst_g) = lists
            assert np.array_equal(cnt, cnt_g)
            used = np.arange(lst.shape[0])[:, None] < np.maximum(cnt, 0)[None, :]
            assert np.array_equal(lst[used], lst_g[used])
        assert between >= 3


@pytest.mark.gpu
@pytest.mark.parametrize("n,grid,narrow", [(30000, (100, 100, 100), True), (30000, (64, 64, 64), False)])
def test_wide_halo_only_while_the_bricks_are_resident_together(n, grid, narrow):
    """Few targets on a grid of many bricks: the halo to stage is then most of the pass."""
    drift = 0.25
    p = small_config(lat=(n, 1, 1), grid=grid, box=tuple(g * c for g, c in zip(grid, (200.0, 200.0, 50.0))), sort_every=1)
    s = random_state(p, 9, "uniform")
    for f in ("u", "v", "w", "ax", "ay", "az"):
        s[f] = np.zeros(n, np.float32)
    with Asph(p) as sim:
        s["u"][:] = drift * 200.0 / sim.control()["dt"]
        sim.set_state(s)
        sim.sort_build()
        sim.kick_drift_flux()
        sim.density_eos()
        deferred = sim.control()["deferred"]
    left = drift / 8 * n   # uniform positions: the share of an 8-cell edge within `drift` of its end
    if narrow:
        assert 0.85 * left < deferred < 1.15 * left   # five standard deviations of a count of 938
    else:
        assert deferred == 0
