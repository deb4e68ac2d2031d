"""hp_dt_noalloc in one launch: the last block to finish reduces the others'
partial minima.  The minimum over the cells equals, bit for bit, the minimum
over calls of at most one block each, at the edges of a block, of the
reduction's strides and with more calls than there are block counters."""
import ctypes

import numpy as np
import pytest

from hydraphase import cases, lib

pytestmark = pytest.mark.gpu
BLOCK = 256


@pytest.fixture(scope="module")
def state():
    import torch
    sp = cases.shock_bubble(n=23, alpha_min=0.1)
    reps = 4                                   # 292,008 cells: over 1024 blocks
    rng = np.random.default_rng(5)
    cn = np.tile(sp.cu, (1, reps)) * (1.0 + 1e-3 * rng.random((1, reps * sp.mesh.neles)))
    dl = rng.uniform(0.01, 0.02, cn.shape[1])
    return torch, torch.from_numpy(np.ascontiguousarray(cn)).cuda(), torch.from_numpy(dl).cuda(), sp.params(cfl=0.3)


def _dt(state, start, n, out):
    torch, cn, dl, p = state
    rc = lib().hp_dt_noalloc(cn.data_ptr() + 8 * start, cn.shape[1], dl.data_ptr() + 8 * start, n, ctypes.byref(p),
                             out.data_ptr(), torch.cuda.current_stream().cuda_stream)
    assert rc == 0
    return out


@pytest.mark.parametrize("n", [1, 31, 255, 256, 257, 4 * 256 * 256 - 1, 4 * 256 * 256 + 257])
def test_blocks_reduce_to_the_minimum_of_single_block_calls(state, n):
    torch, cn, dl, p = state
    whole = _dt(state, 0, n, torch.zeros(1, dtype=torch.float64, device="cuda"))
    parts = torch.full((-(-n // BLOCK),), np.nan, dtype=torch.float64, device="cuda")
    for k in range(parts.numel()):             # up to 1,026 calls
        _dt(state, k * BLOCK, min(BLOCK, n - k * BLOCK), parts[k:])
    assert whole.item() == parts.min().item() and whole.item() > 0
    again = _dt(state, 0, n, torch.zeros(1, dtype=torch.float64, device="cuda"))
    assert again.item() == whole.item()
