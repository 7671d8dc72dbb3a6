"""The radix sort at the sizes where it goes from one form to another: pairs per thread of the
one-launch passes (4,096 pairs each), the largest input they take, tiles of the launches beyond it.
Whole numbers: equal to a stable host sort."""
import ctypes

import numpy as np
import pytest

import akuaengine_gb300 as ak
from akuaengine_gb300 import LambdaCorrParams, PBFConfig
from test_gpu_parity import assert_grid_equal, assert_records_bitexact, run_gpu, run_oracle
from test_gpu_walk_edges import first_of_block

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 31, 4095, 4096, 4097, 8192, 8193, 16384, 16385, 32768, 32769, 65536,
                               65537, 69632, 69633])
@pytest.mark.parametrize("bits", [1, 9, 10, 11, 19, 22, 23, 32])
def test_sort_pairs_edges(cuda_lib, n, bits):
    """Random keys with bits above `bits`, runs of equal keys among them, arrays that start off
    a 16-byte boundary."""
    import torch

    rng = np.random.default_rng(n * 64 + bits)
    keys = rng.integers(0, 1 << 32, size=n, dtype=np.uint64).astype(np.uint32)
    keys[n // 3: n // 2] = keys[0]
    payload = rng.permutation(n).astype(np.uint32)
    order = np.argsort(keys & np.uint32((1 << bits) - 1), kind="stable")
    dev = [torch.zeros(n + 1, dtype=torch.int32, device="cuda") for _ in range(4)]
    for t, host in zip(dev, (keys, payload)):
        t[1:] = torch.from_numpy(host.view(np.int32)).cuda()
    ptr = [ctypes.c_void_p(t.data_ptr() + 4) for t in dev]
    torch.cuda.synchronize()
    rc = cuda_lib.akua_sort_pairs_noalloc(ptr[0], ptr[1], ptr[2], ptr[3], n, bits, None)
    assert rc == 0, ak._abi.status_string(rc)
    torch.cuda.synchronize()
    assert np.array_equal(dev[2][1:].cpu().numpy().view(np.uint32), keys[order])
    assert np.array_equal(dev[3][1:].cpu().numpy().view(np.uint32), payload[order])


@pytest.mark.parametrize("n", [4096, 4097, 16384, 16385, 65536, 65537])
def test_step_order_at_sort_edges(cuda_lib, n):
    """Two steps (the second sorts the first one's order) on both sides of the lines, against the
    oracle."""
    sc = first_of_block(n, seed=n)
    cfg, corr = PBFConfig(), LambdaCorrParams()
    g, ge = run_gpu(sc, cfg, corr, 2, ak.OPT_EXACT_MATH)
    o, oe = run_oracle(sc, cfg, corr, 2)
    assert_grid_equal(ge, oe, cfg.maxNeighbours)
    assert_records_bitexact(g, o)


@pytest.mark.parametrize("n", [262143, 262144, 262145, 266241])
@pytest.mark.parametrize("bits", [8, 9, 20, 27])
def test_sort_pairs_around_64_tiles(cuda_lib, n, bits):
    """Up to 64 tiles a pass's scatter adds the tiles' counts up itself, beyond them the scan does: 64
    tiles but for a pair, 64, 65 (an uneven split of the scan's work) and 66 of one pair; passes of
    8, 9 and 10 bits."""
    test_sort_pairs_edges(cuda_lib, n, bits)


@pytest.mark.parametrize("n", [262144, 262145])
def test_step_order_around_64_tiles(cuda_lib, n):
    """The order of two steps on both sides of that line, against the oracle."""
    test_step_order_at_sort_edges(cuda_lib, n)
