"""A batch's direct plumes do not depend on the FMM plumes beside them.

The direct kernel's FP32 offsets are as precise as its blocks of consecutive
targets are compact, so its plumes are ordered down to the last Morton level,
however shallow the forest's order is.  The same plumes alone in a batch, and
beside balls (a shallow forest) or long columns (a deep one): the accelerations
agree to the order of FP64 atomic additions (1e-12), also where an ion far ahead
of its plume makes the plume's cube large.
"""
import numpy as np
import pytest

import oracle_py as O
import plume
import solveit_gpu as sv
from gpu_util import rel_l2

pytestmark = pytest.mark.gpu

EPS20 = 1e-20


def ahead(n, d, seed):
    st = plume.make_plume(n, n * 2.5e-10, seed)
    if d:
        st["x"][-1] = (0.3 * d, -0.2 * d, d)
    return st


@pytest.mark.parametrize("beside", ["balls", "columns"])
def test_direct_plumes_beside_a_forest(beside):
    direct = [ahead(8000, 1e-4, 1), ahead(8000, 1e-3, 2), ahead(3001, 0.0, 3)]
    if beside == "balls":
        fmm = [plume.make_ball(20000, 1e-7, 4), plume.make_ball(9001, 1e-7, 5)]
    else:
        fmm = [plume.make_plume(40000, 10e-6, 6)]
    with sv.ForceMethod(softening2=EPS20, fmm_order=6, fmm_ws=2) as fm:
        fm.upload_batch(direct, [sv.DIRECT] * 3, [sv.SYM_NONE, sv.SYM_NONE, sv.SYM_ROTATIONAL])
        alone = fm.accel()
    with sv.ForceMethod(softening2=EPS20, fmm_order=6, fmm_ws=2) as fm:
        fm.upload_batch(fmm[:1] + direct + fmm[1:], [sv.FMM] + [sv.DIRECT] * 3 + [sv.FMM] * (len(fmm) - 1),
                        [sv.SYM_NONE] * 3 + [sv.SYM_ROTATIONAL] + [sv.SYM_NONE] * (len(fmm) - 1))
        a = [fm.accel(), fm.accel()]
    first = fmm[0]["q"].size
    for b in a:
        o = 0
        for k, st in enumerate(direct):
            n = st["q"].size
            own, beside_a = alone[o:o + n], b[first + o:first + o + n]
            assert rel_l2(beside_a, own, st["status"]) < 1e-12
            o += n
        # and the FMM plumes themselves (order 6)
        ref = O.direct_f64(fmm[0], EPS20, targets=np.arange(0, first, 16))
        assert rel_l2(b[:first:16], ref, fmm[0]["status"][::16]) < 2.5e-4
