"""Scans and ascending emission of the compression at the edges of their blocks: one group, a whole block of 4096 groups
and one more, rows of one column and dense ones, against a plain restatement with numpy (all column ids are below the
final table length here, so the order is ascending)."""
import numpy as np
import pytest
import torch

from sspmm_b200 import ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("V", [8, 16])
@pytest.mark.parametrize("vec_rows,K,density", [(1, 8, 0.7), (3, 2000, 0.9), (2, 500, 1.0), (40, 33, 0.8), (4095, 6, 0.6), (4096, 6, 0.6),
                                                (4097, 6, 0.6), (9000, 6, 0.5)])
def test_ascending_groups(lib, V, vec_rows, K, density):
    rng = np.random.default_rng(vec_rows + V)
    M = vec_rows * V - 3                                  # the last vector row is not full
    dense = rng.random((M, K)) < density
    vals = rng.uniform(-1, 1, (M, K)).astype(np.float16)
    row_ptr = np.concatenate([[0], np.cumsum(dense.sum(1))]).astype(np.int32)
    col = dense.nonzero()[1].astype(np.int32)
    d = lambda a: torch.from_numpy(a).cuda()
    ptr, vc, vv, _ = ops.svc(d(row_ptr), d(col), d(vals[dense]), M, K, V)
    pad = np.zeros((vec_rows * V, K), dtype=bool)
    pad[:M] = dense
    full = np.zeros((vec_rows * V, K), dtype=np.float16)
    full[:M] = np.where(dense, vals, np.float16(0))
    has = pad.reshape(vec_rows, V, K).any(1)
    want_ptr = np.concatenate([[0], np.cumsum(has.sum(1))])
    assert np.array_equal(ptr.cpu().numpy(), want_ptr)
    r, c = has.nonzero()
    assert np.array_equal(vc.cpu().numpy(), c)
    assert np.array_equal(vv.cpu().numpy().reshape(-1, V), full.reshape(vec_rows, V, K)[r, :, c])
