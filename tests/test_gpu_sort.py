"""The Morton order of small plumes (one chunk, chunks and ranks) against the radix passes' order.

At theta 0 the Barnes-Hut walk opens every cell, and the FMM's depth, lists and
near field follow the sorted keys, so a slot lost or doubled by the order shows
as a wrong force.  Sizes are the edges of a chunk (1024), whole and short last
chunks, the largest ranked plume and one past it; positions repeat (equal keys),
statuses leave inactive particles at the end of the order.
"""
import numpy as np
import pytest

import oracle_py as O
import plume
import solveit_gpu as sv
from gpu_util import rel_l2

pytestmark = pytest.mark.gpu

EPS20 = 1e-20


def state(n, seed):
    st = plume.make_plume(n, max(1e-7, n * 2e-10), seed)
    rng = np.random.default_rng(seed)
    k = n // 7
    if k:  # equal positions: equal keys in different chunks
        st["x"][rng.permutation(n)[:k]] = st["x"][rng.integers(0, n, k)]
    st["status"] = rng.choice(np.array([1, 2, 0, -1], np.int32), n, p=[0.85, 0.05, 0.05, 0.05])
    st["status"][0] = 1
    return st


# the Barnes-Hut walk sums its pairs in FP32, so its bound holds up to a few thousand of them
@pytest.mark.parametrize("n,method,prec,tol",
                         [(n, sv.DIRECT, sv.FP64, 1e-12)
                          for n in (1, 2, 31, 1023, 1024, 1025, 2048, 4095, 5121, 33333)] +
                         [(n, sv.BARNES_HUT, sv.MIXED, 2e-6)
                          for n in (1, 2, 31, 1023, 1024, 1025, 2048, 4095, 5121)])
def test_small_orders(n, method, prec, tol):
    st = state(n, 900 + n)
    tg = np.arange(0, n, max(1, n // 1500))
    ref = O.direct_f64(st, EPS20, targets=tg)
    with sv.ForceMethod(softening2=EPS20, method=method, precision=prec, theta=0.0, leaf_size=16) as fm:
        fm.upload(st)
        a = fm.accel()
        b = fm.accel()  # the second order takes the tree's own number of key levels
    assert rel_l2(a[tg], ref, st["status"][tg]) < tol
    assert rel_l2(b[tg], ref, st["status"][tg]) < tol
    assert not np.any(a[st["status"] != 1])


@pytest.mark.parametrize("n", [65536, 131072, 131073])
def test_fmm_at_the_ranked_limit(n):
    st = plume.make_plume(n, n * 5e-11, n)
    tg = np.arange(0, n, 512)
    ref = O.direct_f64(st, EPS20, targets=tg)
    with sv.ForceMethod(softening2=EPS20, method=sv.FMM, fmm_order=8, fmm_ws=2) as fm:
        fm.upload(st)
        fm.accel(out=False)
        a = fm.accel()
    assert rel_l2(a[tg], ref, st["status"][tg]) < 1e-5
