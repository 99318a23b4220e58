"""Diagonal tiles of the Cholesky and projected-inverse sweeps on the GPU:
one dense front of two column blocks whose second has from 1 to 64 columns,
pivots far from 1 (outside the range of the fast pivots), and a failing pivot
at every kind of position, against LAPACK."""
import numpy as np
import pytest
import torch

import chompack_b200 as cp
from chompack_b200 import _native as N, cbase, grids
from helpers import assert_blocks_close

pytestmark = pytest.mark.gpu


def dense(n, seed=3):
    A = grids.random_lower(n, 1.0, seed=seed)
    s = cp.symbolic(A)
    assert s.Nsn == 1
    X = (cp.cspmatrix(s, device="cpu") + A).blkval.numpy().reshape(n, n, order="F")
    return s, np.tril(X) + np.tril(X, -1).T


def values(s, M):
    return torch.from_numpy(np.tril(M).ravel(order="F").copy()).cuda()


@pytest.mark.parametrize("last", [1, 7, 8, 9, 15, 16, 17, 24, 31, 33, 48, 49, 63, 64])
@pytest.mark.parametrize("scale", [1.0, 1e-302, 1e302])
def test_factor_and_inverse(last, scale):
    s, M = dense(64 + last)
    X = cp.cspmatrix(s, blkval=values(s, M * scale))
    cp.cholesky(X)
    L = np.linalg.cholesky(M)
    assert_blocks_close(s, X.blkval.cpu().numpy() / np.sqrt(scale), L.ravel(order="F"))
    if scale == 1.0:
        cp.projected_inverse(X)
        assert_blocks_close(s, X.blkval.cpu().numpy(), np.tril(np.linalg.inv(M)).ravel(order="F"))


@pytest.mark.parametrize("bad", [0, 1, 7, 8, 9, 15, 16, 40, 63, 64, 71, 72, 90])
def test_failing_pivot(bad):
    s, M = dense(91)
    M[bad, bad] = -1.0
    v = values(s, M)
    plan = s.plan(v.device.index)
    info = cbase._run_and_status(plan, N.OP_CHOLESKY, lambda ws, nb, st: N.cholesky(plan.handle, v.data_ptr(), ws, nb,
                                                                                   st))
    assert info == bad + 1
