"""The near field's pair count: targets times their near sources, on every path.

A cube of about one leaf box of level 2 makes every box a near box of every other, so
the count is the number of targets times the number of sources exactly, without
images and with image copies; source-only, ignored and uncharged ions are no
targets.
"""
import numpy as np
import pytest

import plume
import solveit_gpu as sv

pytestmark = pytest.mark.gpu

EPS20 = 1e-20


def cube(n, seed, centred):
    st = plume.make_plume(n, 1e-6, seed)
    rng = np.random.default_rng(seed)
    side = 2.0 ** -23 * 1.0001
    x = rng.random((n, 3)) * side
    x[0], x[-1] = 0.0, side
    if centred:  # on the rotation axis: the images fall into the same cube
        x[:, :2] -= side / 2
    st["x"] = np.ascontiguousarray(x)
    st["status"] = rng.choice(np.array([1, 2, 0], np.int32), n, p=[0.6, 0.3, 0.1])
    st["status"][[0, -1]] = 2
    st["q"] = rng.choice([0.0, 1.0, 2.0], n, p=[0.1, 0.6, 0.3])
    return st


def numbers(st):
    return int(((st["status"] == 1) & (st["q"] != 0)).sum()), int(np.isin(st["status"], (1, 2)).sum())


@pytest.mark.parametrize("ws", [1, 2])
@pytest.mark.parametrize("sym", [sv.SYM_NONE, sv.SYM_ROTATIONAL], ids=["none", "rotational"])
@pytest.mark.parametrize("n", [9, 257, 3001])
def test_single_plume(n, sym, ws):
    st = cube(n, 40 + n, sym == sv.SYM_ROTATIONAL)
    with sv.ForceMethod(softening2=EPS20, method=sv.FMM, symmetry=sym, fmm_order=4, fmm_ws=ws, fmm_root_scale=1.875,
                        fmm_leaf_target=4096) as fm:
        fm.upload(st)
        fm.accel()
        s = fm.stats()
    t, src = numbers(st)
    assert s.cell_interactions == 0
    assert s.pair_interactions == t * src * (4 if sym == sv.SYM_ROTATIONAL else 1)

