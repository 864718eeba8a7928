"""The FMM's passes over few and many boxes per level.

Columns of a few thousand ions have many levels of a handful of boxes (taken in
one launch by the upward and downward passes), balls jump from 64 boxes to
hundreds, and source-only ions leave boxes, branches and whole levels without
targets.  Bounds: the force error against the FP64 oracle that each order is
held to elsewhere (p 4: 5e-3, 6: 2.5e-4, 8: 1e-5, 10: 2e-6 at separation 2;
targets that stay targets get the same accelerations, to 1e-6, when the other
ions turn into sources only).
"""
import numpy as np
import pytest

import oracle_py as O
import plume
import solveit_gpu as sv
from gpu_util import rel_l2

pytestmark = pytest.mark.gpu

EPS20 = 1e-20
BOUND = {4: 5e-3, 6: 2.5e-4, 8: 1e-5, 10: 2e-6}


def make(kind, n):
    return plume.make_ball(n, 2e-9 * n ** 0.4, n) if kind == "ball" else plume.make_plume(n, n * 1e-10, n)


def run(st, **kw):
    with sv.ForceMethod(softening2=EPS20, method=sv.FMM, fmm_ws=2, **kw) as fm:
        fm.upload(st)
        fm.accel(out=False)
        return fm.accel()


@pytest.mark.parametrize("p", [4, 6, 8, 10])
@pytest.mark.parametrize("kind,n", [("column", 1500), ("column", 12000), ("ball", 3000), ("ball", 30000)])
def test_levels(kind, n, p):
    st = make(kind, n)
    tg = np.arange(0, n, max(1, n // 1000))
    a = run(st, fmm_order=p)
    assert rel_l2(a[tg], O.direct_f64(st, EPS20, targets=tg), st["status"][tg]) < BOUND[p]


@pytest.mark.parametrize("kind,n", [("column", 12000), ("ball", 30000)])
def test_few_targets(kind, n):
    st = make(kind, n)
    full = run(st, fmm_order=8)
    few = dict(st, status=np.full(n, 2, np.int32))
    few["status"][[7, n // 2, n - 1]] = 1
    a = run(few, fmm_order=8)
    t = few["status"] == 1
    assert rel_l2(a[t], full[t], few["status"][t]) < 1e-6
    assert not np.any(a[~t])
