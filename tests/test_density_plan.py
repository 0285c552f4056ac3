"""The density pass's launch plan, formed on the host (no GPU needed)."""
import pytest

import hostbuild


@pytest.fixture(scope="module")
def plan(tmp_path_factory):
    return hostbuild.build("plan", tmp_path_factory.mktemp("plan"), fake=False)


@pytest.mark.parametrize("n", [1, 60, 64, 125, 1000])
@pytest.mark.parametrize("grid", [(20, 20, 40), (14, 14, 5), (100, 100, 100)])
def test_sparse_grids_have_a_plan(plan, grid, n):
    """Fewer particles than one per brick still make a launch of whole warps."""
    r = hostbuild.run(plan, *grid, n)
    assert r.returncode == 0, "exit %d" % r.returncode
    assert -1 <= int(r.stdout) <= 3


@pytest.mark.parametrize("grid,n,shape", [
    # sparse: smaller bricks would be no better filled, only more
    ((100, 100, 100), 3000, 0), ((100, 100, 100), 30000, 0), ((100, 100, 100), 150000, 0), ((160, 160, 160), 40960, 0),
    # few bricks: smaller ones until every SM has four
    ((64, 64, 64), 7864, 1), ((40, 40, 40), 28800, 3),
    # dense: smaller ones while they leave more warps resident
    ((133, 133, 200), 2097152, 0), ((128, 128, 128), 2097152, 1),
])
def test_shape_for_the_density_of_the_grid(plan, grid, n, shape):
    r = hostbuild.run(plan, *grid, n)
    assert r.returncode == 0 and int(r.stdout) == shape
