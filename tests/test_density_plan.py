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
