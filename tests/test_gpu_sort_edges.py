"""The order of small plumes at its kernels' own edges.

Up to 1,024 particles one CTA sorts, up to 8,192 chunks of 256 and up to 32,768 chunks of
1,024 are ranked against each other, above that radix passes sort.  Whole and short
last chunks, both sides of each change, equal keys in different chunks, inactive
particles behind them.  A slot lost or doubled shows in the FP64 direct sum (1e-12;
it sorts above 8,192 particles), a wrong place in the FMM, whose boxes are runs
of sorted slots (order 8: 1e-5 on sampled targets).
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
    k = n // 7  # equal positions
    st["x"][rng.permutation(n)[:k]] = st["x"][rng.integers(0, n, k)]
    st["status"] = rng.choice(np.array([1, 2, 0, -1], np.int32), n, p=[0.85, 0.05, 0.05, 0.05])
    st["status"][0] = 1
    return st


@pytest.mark.parametrize("method,prec,tol", [(sv.DIRECT, sv.FP64, 1e-12), (sv.FMM, sv.MIXED, 1e-5)],
                         ids=["direct", "fmm"])
@pytest.mark.parametrize("n", [1024, 1025, 1280, 1281, 8191, 8192, 8193, 9216, 9217, 32767, 32768, 32769])
def test_edges(n, method, prec, tol):
    st = state(n, 300 + n)
    tg = np.arange(0, n, max(1, n // 1500))
    ref = O.direct_f64(st, EPS20, targets=tg)
    with sv.ForceMethod(softening2=EPS20, method=method, precision=prec, fmm_order=8, fmm_ws=2) as fm:
        fm.upload(st)
        a = fm.accel()
        b = fm.accel()  # the FMM's second order takes its tree's own number of key levels
    for v in (a, b):
        assert rel_l2(v[tg], ref, st["status"][tg]) < tol
        assert not np.any(v[st["status"] != 1])
