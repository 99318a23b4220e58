"""Fronts of at most 64 rows as one task each (cholesky, projected_inverse),
bundles off: a front of nn columns and na separators under a root of na + 3
columns, at the edges of the 8- and 16-column blocks, against the oracle; a
failing pivot in either front."""
import numpy as np
import pytest
import torch

import chompack_b200 as cp
from chompack_b200 import _native as N, cbase, grids
from helpers import assert_blocks_close
from oracle import oracle

pytestmark = pytest.mark.gpu

SIZES = [(1, 1), (2, 40), (1, 60), (7, 9), (8, 8), (9, 55), (15, 17), (16, 16), (16, 48), (17, 44), (24, 33),
         (31, 33), (32, 32), (33, 31), (40, 24), (47, 17), (48, 16), (49, 15), (50, 14), (57, 7), (60, 1), (63, 1)]


def two_fronts(nn, na, extra=3):
    n = nn + na + extra
    r, c = np.tril_indices(n, -1)
    keep = (c >= nn) | (r < nn + na)
    A = grids.spd_from_lower_pattern(n, r[keep], c[keep], nn + 100 * na)
    s = cp.symbolic(A)
    assert [int(x) for x in np.diff(s.snptr)] == [nn, na + extra]
    s.plan().set_option("subtrees", 0)
    return s, (cp.cspmatrix(s, device="cpu") + A).blkval.numpy()


@pytest.mark.parametrize("nn,na", SIZES)
def test_factor_and_inverse(nn, na):
    s, x = two_fronts(nn, na)
    ref = x.copy()
    X = cp.cspmatrix(s, blkval=torch.from_numpy(x.copy()).cuda())
    assert oracle.cholesky(s, ref) == 0
    cp.cholesky(X)
    assert_blocks_close(s, X.blkval.cpu().numpy(), ref)
    X.blkval.copy_(torch.from_numpy(ref))
    assert oracle.projected_inverse(s, ref) == 0
    cp.projected_inverse(X)
    assert_blocks_close(s, X.blkval.cpu().numpy(), ref)


@pytest.mark.parametrize("nn,na,k,bad", [(9, 30, 0, 0), (9, 30, 0, 8), (40, 20, 0, 39), (40, 20, 1, 0), (5, 50, 1, 52),
                                         (17, 40, 1, 16)])
def test_failing_pivot(nn, na, k, bad):
    s, x = two_fronts(nn, na)
    nj = int(s.sncolptr[k + 1] - s.sncolptr[k])
    x[int(s.blkptr[k]) + bad * (nj + 1)] = -1.0
    v = torch.from_numpy(x).cuda()
    plan = s.plan(v.device.index)
    info = cbase._run_and_status(plan, N.OP_CHOLESKY, lambda ws, nb, st: N.cholesky(plan.handle, v.data_ptr(), ws, nb,
                                                                                   st))
    assert info == bad + 1


@pytest.mark.parametrize("scale", [1e-302, 1e302])
def test_pivots_far_from_one(scale):
    s, x = two_fronts(20, 30)
    ref = x.copy()
    assert oracle.cholesky(s, ref) == 0
    X = cp.cspmatrix(s, blkval=torch.from_numpy(x * scale).cuda())
    cp.cholesky(X)
    got = X.blkval.cpu().numpy()
    nj, nn = 50, 20
    # diagonal blocks scale with the root, the rows below them not at all
    b = got[:nj * nn].reshape(nn, nj)
    b[:, :nn] /= np.sqrt(scale)
    got[nj * nn:] /= np.sqrt(scale)
    assert_blocks_close(s, got, ref)
