"""The tensor-core M2L's class passes over few and many boxes per block.

The bucketed translations are the same set whatever boxes a block takes, so
the accelerations agree with the FP32 rotation kernel's to the two paths'
bound (3e-6) on plumes of a few boxes, of hundreds of well-filled boxes
(4 boxes per block) and of thousands of thin ones, and in a forest.
"""
import numpy as np
import pytest

import plume
import solveit_gpu as sv
from gpu_util import rel_l2

pytestmark = pytest.mark.gpu

EPS20 = 1e-20


@pytest.mark.parametrize("p", [6, 8])
@pytest.mark.parametrize("st", [("ball", 700, 60e-9), ("ball", 40000, 180e-9), ("column", 150000, 20e-6)],
                         ids=["few", "filled", "thin"])
def test_classes_match_rotation_kernel(st, p):
    kind, n, size = st
    s = plume.make_ball(n, size, 31) if kind == "ball" else plume.make_plume(n, size, 31)
    out = []
    for tc in (1, -1):
        with sv.ForceMethod(softening2=EPS20, method=sv.FMM, fmm_order=p, fmm_ws=2, fmm_m2l_tc=tc) as fm:
            fm.upload(s)
            fm.accel(out=False)  # the first evaluation sizes the tensor-core room
            out.append(fm.accel())
            assert fm.stats().m2l_tc == (1 if tc == 1 else 0)
    assert rel_l2(out[0], out[1], s["status"]) < 3e-6


def test_forest_classes_match_rotation_kernel():
    states = [plume.make_ball(n, 1.5e-7, 60 + n) for n in (9000, 20000, 12345)]
    st = np.concatenate([s["status"] for s in states])
    out = []
    for tc in (1, -1):
        with sv.ForceMethod(softening2=EPS20, fmm_order=6, fmm_ws=2, fmm_m2l_tc=tc) as fm:
            fm.upload_batch(states, [sv.FMM] * 3, [sv.SYM_NONE, sv.SYM_ROTATIONAL, sv.SYM_NONE])
            fm.accel(out=False)
            out.append(fm.accel())
    assert rel_l2(out[0], out[1], st) < 3e-6
