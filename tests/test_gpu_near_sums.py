"""The near field's FP32 sums take at most 32 sources before a compensated addition.

One target with a strong neighbour and 2,000 weak sources that all pull the same
way, each with a force of 2^-26 of the neighbour's: below half a unit in the last
place, a weak force is lost when it is added to an FP32 sum that holds the strong
one, and kept by the compensated additions.  A sum of 32 sources runs in two halves
of 16, so at most 15 are lost; the result's own rounding to FP32 is worth up to 4.
The positions are multiples of 2^-45 m, so that every offset is exact in FP32, and
the neighbour's own force, with the error of its reciprocal square root, is taken
off by an evaluation with uncharged weak sources.
"""
import numpy as np
import pytest

import oracle_py as O
import plume
import solveit_gpu as sv

pytestmark = pytest.mark.gpu

EPS20 = 1e-20


def accel(st, ws):
    # a cube of about one leaf box of level 2: the near field alone
    with sv.ForceMethod(softening2=EPS20, method=sv.FMM, fmm_order=4, fmm_ws=ws, fmm_root_scale=1.875,
                        fmm_leaf_target=4096) as fm:
        fm.upload(st)
        a = fm.accel()
        assert fm.stats().cell_interactions == 0
    return a


@pytest.mark.parametrize("ws", [1, 2])
@pytest.mark.parametrize("weak", [300, 2000])
def test_weak_sources_beside_a_strong_one(weak, ws):
    n = weak + 4
    side = 2.0 ** -23 * 1.0001
    grid = lambda v: np.round(np.asarray(v) * 2.0 ** 45) * 2.0 ** -45
    rng = np.random.default_rng(weak)
    st = plume.make_plume(n, 1e-6, weak)
    x = np.empty((n, 3))
    x[0], x[1] = 0.0, side                                # the cube's corners, uncharged
    x[2] = grid(np.full(3, 0.1 * side))                   # the target
    x[3] = x[2] - grid(np.full(3, 6e-10))                 # its neighbour: first in the order, and pushing as the weak
    x[4:] = grid(x[2] + (0.7 + 0.02 * rng.random((weak, 1))) * side + 0.004 * side * rng.random((weak, 3)))
    st["x"] = x
    st["status"][:] = 2
    st["status"][2] = 1
    unit = 2.0 ** -26 / (np.sum((x[3] - x[2]) ** 2) + EPS20)
    st["q"] = np.zeros(n)
    st["q"][2:4] = 1.0
    alone = accel(st, ws)
    st["q"][4:] = -unit * np.sum((x[4:] - x[2]) ** 2, axis=1)  # attracting: the same direction as the neighbour's push
    a = accel(st, ws)
    ref0 = O.direct_f64(dict(st, q=np.where(np.arange(n) < 4, st["q"], 0.0)), EPS20, targets=np.array([2]))[0]
    ref = O.direct_f64(st, EPS20, targets=np.array([2]))[0]
    want, got = ref - ref0, a[2] - alone[2]
    lost = weak * (1.0 - got / want)
    assert np.all(np.abs(lost) < 20), lost
