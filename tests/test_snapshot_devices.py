"""Snapshots between GPUs of one process (the CUDA runtime replaced by a
stand-in on the host, no GPU needed)."""
import pytest

import hostbuild

PARTS = 13   # field groups and the control block


@pytest.fixture(scope="module")
def exchange(tmp_path_factory):
    prog = hostbuild.build("snapshot", tmp_path_factory.mktemp("snapshot"))

    def f(*devices):
        r = hostbuild.run(prog, *devices)
        assert r.returncode == 0, "exit %d" % r.returncode
        return tuple(int(v) for v in r.stdout.split())
    return f


@pytest.mark.parametrize("dev", [0, 1])
def test_one_gpu_takes_one_launch(exchange, dev):
    assert exchange(dev, dev, dev, dev, dev)[:4] == (1, 0, 1, 0)


# the current device while each is made or called: context, snapshot, save, second context, restore
@pytest.mark.parametrize("devices", [(0, 1, 0, 0, 0), (0, 0, 1, 0, 1), (0, 1, 1, 1, 0), (1, 0, 0, 0, 1)])
def test_another_gpu_takes_copies(exchange, devices):
    """A kernel cannot read or write another GPU's memory, and cannot be launched
    on a stream of a GPU that is not current; copies can."""
    assert exchange(*devices) == (0, PARTS, 0, PARTS, 1)


def test_restoring_on_a_second_gpu(exchange):
    launches_save, copies_save, launches_restore, copies_restore, _ = exchange(0, 0, 0, 1, 1)
    assert (launches_save, copies_save) == (1, 0)
    assert (launches_restore, copies_restore) == (0, PARTS)
