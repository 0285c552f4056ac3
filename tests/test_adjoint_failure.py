"""The adjoint's backward when it fails half way (the CUDA runtime replaced by a
stand-in on the host, no GPU needed)."""
import pytest

import hostbuild
from sph_cuda_gb300 import abi


@pytest.mark.parametrize("given", [1, 2, 4, 7])
def test_seeds_are_the_callers_again_when_backward_returns(given, tmp_path):
    """Page-locked seeds are read by the GPU: a failing backward returns only
    after its copies of them have ended."""
    r = hostbuild.run(hostbuild.build("backward", tmp_path), given)
    assert r.returncode == 0, r.stderr
    status, made, unfinished = (int(v) for v in r.stdout.split())
    assert status == abi.ASPH_ERR_CUDA
    assert made == bin(given).count("1")
    assert unfinished == 0
