"""The key sort at the edges of its tiles: sizes around one tile, a whole number
of tiles, and where the tile size changes, with few distinct keys (one digit
holds most of a tile) and with many."""
import ctypes

import numpy as np
import pytest

from sph_cuda_gb300 import abi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bits,distinct", [(8, 3), (24, 1 << 24), (30, 1 << 30)])
@pytest.mark.parametrize("n", [1, 31, 1023, 1024, 1025, 152 * 1024, 152 * 1024 + 1, 200 * 2048 + 7,
                               abi.NOALLOC_MAX_KEYS - 1])
def test_sorted_keys_and_permutation(n, bits, distinct):
    torch = pytest.importorskip("torch")
    lib = abi.load_library()
    keys = np.random.default_rng(n + bits).integers(0, distinct, n, dtype=np.uint32)
    dk = torch.from_numpy(keys.view(np.int32)).cuda()
    out = [torch.full((n,), -1, dtype=torch.int32, device="cuda") for _ in range(2)]
    rc = lib.asph_sort_keys_noalloc(ctypes.c_void_p(dk.data_ptr()), ctypes.c_void_p(out[0].data_ptr()),
                                    ctypes.c_void_p(out[1].data_ptr()), n, bits,
                                    ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert rc == abi.ASPH_OK, lib.asph_last_error()
    perm = np.argsort(keys, kind="stable")
    assert np.array_equal(out[1].cpu().numpy().view(np.uint32), perm.astype(np.uint32))
    assert np.array_equal(out[0].cpu().numpy().view(np.uint32), keys[perm])
