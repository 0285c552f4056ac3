"""The brick density pass finds its candidates with an fp16 test that may only
pass too many: its lists are those of the per-target global path, entry by
entry, and its densities agree to the float rounding of the sums."""
import numpy as np
import pytest

from sph_cuda_gb300 import Asph
from statebuild import random_state, reference_geometry, small_config

pytestmark = pytest.mark.gpu


def _wide(lat=(20, 20, 20), **kw):
    """8:1 cells (160 m x 20 m) far from the origin of a large box, where a float position is coarsest in cells."""
    return small_config(lat=lat, grid=(60, 14, 100), box=(9600.0, 2240.0, 2000.0), **kw)


CASES = {
    # the narrowest grid that has bricks, odd slot counts, empty rows
    "narrow_sparse": (lambda: small_config(lat=(13, 11, 9), grid=(14, 14, 17), box=(2800.0, 2800.0, 850.0)), "uniform"),
    # one and two particles per cell: the smaller bricks, more than one round of targets
    "one_per_cell": (lambda: reference_geometry(24, 22, 20), "jitter"),
    "two_per_cell": (lambda: small_config(lat=(32, 28, 32), grid=(24, 24, 25), box=(4800.0, 4800.0, 1250.0)), "uniform"),
    # clustered: long rows, queues that drain many times, split regions
    "clustered": (lambda: small_config(lat=(40, 40, 20), grid=(40, 40, 40), box=(8000.0, 8000.0, 2000.0)), "cluster"),
    # pairs across the periodic edge, whose raw distances are a box length
    "anisotropic_wide": (lambda: _wide(), "jitter"),
    # more than 77,824 targets, one block of 512 threads per SM:
    # sorted every step the narrow halo, which drifted targets leave; every fourth step the wide one
    "narrow_halo": (lambda: small_config(lat=(48, 42, 42), grid=(48, 42, 40), box=(9600.0, 8400.0, 2000.0),
                                         sort_every=1), "jitter"),
    "wide_halo": (lambda: small_config(lat=(48, 42, 42), grid=(48, 42, 40), box=(9600.0, 8400.0, 2000.0),
                                       sort_every=4), "jitter"),
}


def _density(p, s, path, drift):
    sim = Asph(p)
    sim.set_pair_path(path)
    sim.set_state(s)
    sim.sort_build()
    if drift:   # the table is one drift old, as in a step
        sim.kick_drift_flux()
    sim.density_eos()
    cnt, lst = sim.neighbours()
    st = sim.get_state(("rho", "x"))
    sim.close()
    return cnt, lst, st


@pytest.mark.parametrize("drift", [False, True])
@pytest.mark.parametrize("name", sorted(CASES))
def test_lists_equal_the_global_path(name, drift):
    make, layout = CASES[name]
    p = make()
    s = random_state(p, 31, layout, speed=25.0)
    cnt, lst, st = _density(p, s, 0, drift)
    cnt_g, lst_g, st_g = _density(p, s, 1, drift)
    assert np.array_equal(st["x"], st_g["x"])
    assert np.array_equal(cnt, cnt_g)
    used = np.arange(lst.shape[0])[:, None] < np.maximum(cnt, 0)[None, :]
    assert np.array_equal(lst[used], lst_g[used])
    # rho = S1 / S2 of at most a few hundred positive terms: n 2^-24 relative for
    # each sum at the very worst, 1e-5 for 200 terms
    assert np.max(np.abs(st["rho"] - st_g["rho"]) / st_g["rho"]) < 1e-5
