"""The M2L's weight that a batch takes before tuning: by the shape of its plumes.

Plumes that fill their cubes take 800, columns 200, large columns 400 (measured beside
the rule); a weight that the caller sets stays, over re-planning and further evaluations.
Accelerations meet the batch's order-6 bound either way.
"""
import numpy as np
import pytest

import oracle_py as O
import plume
import solveit_gpu as sv
from gpu_util import rel_l2

pytestmark = pytest.mark.gpu

EPS20 = 1e-20


def column(n, seed):
    return plume.make_plume(n, 1e-6, seed)


def ball(n, seed):
    return plume.make_ball(n, 3e-9 * n ** 0.4, seed)


@pytest.mark.parametrize("kinds,weight", [((ball, ball), 800), ((column, column), 200), ((ball, ball, column), 800),
                                          ((column, column, ball), 200)], ids=["balls", "columns", "balls+", "columns+"])
def test_untuned_weight(kinds, weight):
    n = 12000
    states = [k(n, 30 + i) for i, k in enumerate(kinds)]
    with sv.ForceMethod(softening2=EPS20, fmm_order=6, fmm_ws=2) as fm:
        fm.upload_batch(states, [sv.FMM] * len(states), [sv.SYM_NONE] * len(states))
        a = fm.accel()
        assert fm.batch_info().m2l_weight == weight
        tg = np.arange(0, n, 16)
        for k, st in enumerate(states):
            assert rel_l2(a[k * n:(k + 1) * n][tg], O.direct_f64(st, EPS20, targets=tg), st["status"][tg]) < 2.5e-4
        fm.set_tuning(400, 2048)
        for _ in range(2):
            fm.accel(out=False)
            assert fm.batch_info().m2l_weight == 400


def test_large_columns():
    states = [column(22000, 50 + i) for i in range(2)]
    with sv.ForceMethod(softening2=EPS20, fmm_order=4, fmm_ws=2) as fm:
        fm.upload_batch(states, [sv.FMM] * 2, [sv.SYM_ROTATIONAL] * 2)
        fm.accel(out=False)
        assert fm.batch_info().m2l_weight == 400
