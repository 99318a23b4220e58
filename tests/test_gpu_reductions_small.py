"""dot and the weights of `dot` on patterns of many small supernodes, whose
entries are searched for one by one, and at the sizes where the pieces' length
changes, against numpy."""
import numpy as np
import pytest
import torch

import chompack_b200 as cp
from chompack_b200 import grids
from chompack_b200.autograd import _sym_weight
from test_gpu_reductions import close, weights

pytestmark = pytest.mark.gpu


def leaves(count, cols, sep, root):
    """`count` leaves of `cols` columns, each over the first `sep` columns of
    a dense root."""
    E, at = [], count * cols
    for v in range(count):
        c = list(range(v * cols, (v + 1) * cols)) + list(range(at, at + sep))
        E += [(a, b) for a in c for b in c if a > b and b < at]
    E += [(a, b) for a in range(at, at + root) for b in range(at, a)]
    I, J = np.array(E).T
    return grids.spd_from_lower_pattern(at + root, I, J, count)


@pytest.mark.parametrize("count,cols,sep,root", [(1, 1, 1, 1), (50, 1, 2, 9), (85, 1, 2, 2), (600, 1, 1, 70),
                                                 (40, 5, 10, 300), (300, 7, 5, 700), (30, 9, 9, 1500)])
def test_many_small_supernodes(count, cols, sep, root):
    s = cp.symbolic(leaves(count, cols, sep, root))
    rng = np.random.default_rng(count)
    x, y = (rng.standard_normal(int(s.blkptr[-1])) for _ in range(2))
    w = weights(s)
    X, Y = (cp.cspmatrix(s, blkval=torch.from_numpy(v).cuda()) for v in (x, y))
    close(cp.dot(X, Y), x, y, w)
    assert np.array_equal(_sym_weight(s, X.blkval, -0.5).cpu().numpy(), -0.5 * w * x)


@pytest.mark.parametrize("side", [10, 60, 200])
def test_unmerged_grid(side):
    A = grids.grid2d(side, seed=0)
    s = cp.symbolic(A, p=cp.amd.order(A))
    x = np.random.default_rng(side).standard_normal(int(s.blkptr[-1]))
    X = cp.cspmatrix(s, blkval=torch.from_numpy(x).cuda())
    close(cp.dot(X, X), x, x, weights(s))
