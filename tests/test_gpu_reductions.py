"""dot, the batched dot and the weights of `dot` on the GPU, over pieces of
the block values: blocks smaller and larger than a piece (4096 entries) and
ending on its edges, single blocks and merged plans, against numpy."""
import numpy as np
import pytest
import torch

import chompack_b200 as cp
from chompack_b200 import grids
from chompack_b200.autograd import _sym_weight

pytestmark = pytest.mark.gpu


def weights(s):
    w = np.empty(int(s.blkptr[-1]))
    for k in range(s.Nsn):
        nn = int(s.snptr[k + 1] - s.snptr[k])
        nj = int(s.sncolptr[k + 1] - s.sncolptr[k])
        r, c = np.arange(nj)[:, None], np.arange(nn)[None, :]
        w[int(s.blkptr[k]):int(s.blkptr[k + 1])] = np.where(r > c, 2.0, np.where(r == c, 1.0, 0.0)).ravel(order="F")
    return w


def pattern(kind, size):
    A = grids.random_lower(size, 1.0, seed=1) if kind == "dense" else \
        grids.grid2d(size) if kind == "grid2d" else grids.grid3d(size)
    return cp.symbolic(A, p=cp.amd.order(A), merge_function=cp.merge_size_fill(8, 8) if kind == "grid3d" else None)


def close(got, x, y, w):
    # a sum of N products in any order is within N 2^-53 of the sum of their sizes
    t = x * y * w
    assert abs(got - t.sum()) <= 2.0 * t.size * 2.0 ** -53 * np.abs(t).sum()


CASES = [("dense", 1), ("dense", 63), ("dense", 64), ("dense", 65), ("dense", 200), ("grid2d", 1), ("grid2d", 37),
         ("grid3d", 9)]


@pytest.mark.parametrize("kind,size", CASES)
def test_dot_and_weights(kind, size):
    s = pattern(kind, size)
    rng = np.random.default_rng(size)
    x, y = (rng.standard_normal(int(s.blkptr[-1])) for _ in range(2))
    w = weights(s)
    X, Y = (cp.cspmatrix(s, blkval=torch.from_numpy(v).cuda()) for v in (x, y))
    close(cp.dot(X, Y), x, y, w)
    assert np.array_equal(_sym_weight(s, X.blkval, -0.5).cpu().numpy(), -0.5 * w * x)


def test_batched_dot_cuts_at_the_matrices():
    ss = [pattern(*c) for c in CASES] + [pattern("grid2d", 3)] * 3
    B = cp.batch(ss)
    rng = np.random.default_rng(5)
    x, y = (rng.standard_normal(B.size) for _ in range(2))
    xd, yd = torch.from_numpy(x).cuda(), torch.from_numpy(y).cuda()
    got = B.dot(xd, yd).cpu().numpy()
    for m, s in enumerate(ss):
        a, b = B.offsets[m], B.offsets[m + 1]
        close(got[m], x[a:b], y[a:b], weights(s))
    w = np.concatenate([weights(s) for s in ss])
    assert np.array_equal(B.sym_weight(xd, 3.0).cpu().numpy(), 3.0 * w * x)
