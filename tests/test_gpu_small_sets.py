"""Small sets: the sort by counting (up to a tile of 4096 keys) against a stable sort, around its block,
tile and range limits and with many equal keys; and the one-block scan of the output offsets (up to
16,384 entries) against the owned vertices counted from the stores."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2, 3, 63, 64, 65, 1000, 4095, 4096, 4097, 8192])
@pytest.mark.parametrize("distinct", [1, 7, 1 << 62])
def test_sort_is_stable(n, distinct):
    import torch
    import apo_b200
    lib = apo_b200.load_library()
    rng = np.random.default_rng(n)
    keys = rng.integers(0, distinct, n, dtype=np.int64)
    values = rng.permutation(n).astype(np.int32)
    k, v = torch.from_numpy(keys).cuda(), torch.from_numpy(values).cuda()
    scratch = torch.empty(lib.apo2_radix_sort_scratch_bytes(n), dtype=torch.uint8, device="cuda")
    apo_b200._check(lib.apo2_radix_sort_pairs(k.data_ptr(), v.data_ptr(), n, scratch.data_ptr(), ctypes.c_void_p(0)))
    torch.cuda.synchronize()
    order = np.argsort(keys, kind="stable")
    assert np.array_equal(k.cpu().numpy(), keys[order])
    assert np.array_equal(v.cpu().numpy(), values[order])


@pytest.mark.parametrize("n", [2047, 2048, 2049, 16383, 16384, 16385])
def test_output_offsets(n):
    import apo_b200
    from apo_b200 import generators
    algo = apo_b200.AlgorithmGPU(generators.uniform_random(n, 10.0 * n ** (1 / 3) / 2.15, 0.5, 2.0, n))
    algo.build()
    nb = algo.debug_array("vertex_nb").astype(np.int64)
    status = algo.debug_array("status")
    rec = algo.debug_array("vertices").reshape(-1, 4)[:, :3].astype(np.int64)
    cell = np.repeat(np.arange(n), nb)
    own = (cell <= rec[:, 0]) & (rec < n).all(axis=1) & (status[cell] != 0xff)
    ix = algo.debug_array("indices")
    expected = np.concatenate([ix[cell[own]][:, None], ix[rec[own]]], axis=1)
    assert np.array_equal(algo.toHost().verticesId.reshape(-1, 4), expected)
    algo.close()
