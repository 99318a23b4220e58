"""Traces of a solve in list order: a task's start stamp is not before the end
of any task it waits for, narrow products (which wait inside the task)
included."""
import numpy as np
import pytest
import torch

import chompack_b200 as cp
from chompack_b200 import _native as N, trace
from helpers import problem

pytestmark = pytest.mark.gpu

SLACK = 2000  # ns: the granularity of the global timer, and the stamps' order


@pytest.mark.parametrize("trans", ["N", "T"])
def test_narrow_products_start_when_their_dependencies_are_met(trans):
    A, s = problem("grid3d", 16, merge=(32, 32), seed=0)
    L = cp.cspmatrix(s) + A
    cp.cholesky(L)
    plan = s.plan(0)
    plan.set_schedule("static")
    B = torch.randn(8, s.n, dtype=torch.float64, device="cuda")
    cp.trsm(L, B.clone().t(), trans=trans)
    tasks, waits, tr = trace.record(plan, N.OP_TRSM, lambda: cp.trsm(L, B.clone().t(), trans=trans), 8,
                                    int(trans == "T"))
    narrow = np.flatnonzero((tasks["op"] == 0) & (tasks["aux"][:, 0] == 1))
    assert len(narrow) > 100
    members = {}
    for i, g in enumerate(tasks["group"]):
        members.setdefault(int(g), []).append(i)
    for i in narrow:
        w0 = int(tasks["wait_off"][i])
        for cid, target in waits[w0:w0 + int(tasks["nwait"][i])]:
            prod = [int(cid)] if cid < len(tasks) else members[int(cid)]
            if target == len(prod):
                assert tr[i, 1] >= tr[prod, 2].max() - SLACK, (i, prod)
