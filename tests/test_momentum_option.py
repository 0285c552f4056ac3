"""The targets-per-thread option of the momentum pass and the launch it gives
(formed on the host, no GPU needed)."""
import pytest

import hostbuild


@pytest.fixture(scope="module")
def launch(tmp_path_factory):
    prog = hostbuild.build("momentum_launch", tmp_path_factory.mktemp("momentum"))

    def f(*args):
        r = hostbuild.run(prog, *args)
        assert r.returncode == 0, "exit %d" % r.returncode
        return tuple(int(v) for v in r.stdout.split())
    return f


@pytest.mark.parametrize("n", [16400, 65536, 311296, 311297, 475136, 2097152])
def test_setting_the_value_that_was_read_keeps_the_launch(launch, n):
    default = launch(n)
    assert launch(n, "r") == default
    assert launch(n, 4, 0) == default
    assert launch(n, 4, 2) == default   # 2 is the default


@pytest.mark.parametrize("n", [16400, 475136])
@pytest.mark.parametrize("tpt", [1, 4])
def test_other_values_are_taken_as_they_are(launch, n, tpt):
    assert launch(n, tpt) == (tpt, tpt)
    assert launch(n, tpt, "r") == (tpt, tpt)
