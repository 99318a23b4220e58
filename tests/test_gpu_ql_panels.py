"""Householder panels of the factored updates on the GPU: completion with
factored updates on three-level patterns whose panels have from one to 70
columns and heights on both sides of every change of the panel's layout
(128, 256 and 512 rows), against the oracle."""
import numpy as np
import pytest
import torch

import chompack_b200 as cp
from chompack_b200 import grids
from helpers import assert_blocks_close
from oracle import oracle

pytestmark = pytest.mark.gpu


def three_levels(na, n2, n1=3, nchild=2, nmid=4, seed=0):
    """Root: a dense block of na + 5; a middle front with na separators; a
    child whose separators are n1 columns of the middle front and n2 of the
    root's, the first and the last of them included."""
    rng = np.random.default_rng(seed)
    root = nchild + nmid
    n = root + na + 5
    sep = np.arange(root, root + na)
    inner = rng.choice(np.arange(1, na - 1), size=n2 - 2, replace=False) if n2 > 2 else np.zeros(0, int)
    sub = sep[np.unique(np.concatenate([[0], inner, [na - 1]])[:max(n2, 1)].astype(int))]
    E = set()

    def clique(v):
        for a in v:
            for b in v:
                if a > b:
                    E.add((int(a), int(b)))
    clique(list(range(nchild)) + list(range(nchild, nchild + n1)) + list(sub))
    clique(list(range(nchild, root)) + list(sep))
    clique(range(root, n))
    I, J = np.array(sorted(E)).T
    return grids.spd_from_lower_pattern(n, I, J, seed)


@pytest.mark.parametrize("na,n2", [(20, 1), (90, 2), (127, 8), (128, 9), (129, 63), (130, 64), (255, 16), (256, 30),
                                   (257, 17), (300, 70), (511, 8), (512, 20), (514, 25), (700, 12)])
def test_factored_completion(na, n2):
    A = three_levels(na, n2)
    s = cp.symbolic(A)
    X = cp.cspmatrix(s, device="cpu") + A
    ref = X.blkval.numpy().copy()
    assert oracle.cholesky(s, ref) == 0
    assert oracle.projected_inverse(s, ref) == 0
    Y = cp.cspmatrix(s, blkval=torch.from_numpy(ref.copy()).cuda())
    assert oracle.completion(s, ref, True) == 0
    cp.completion(Y, factored_updates=True)
    assert_blocks_close(s, Y.blkval.cpu().numpy(), ref)
