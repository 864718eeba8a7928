"""What a method asks of its sort holds for every evaluation, the one that allocates or grows
the sorted buffers among them.

The direct sum up to 8,192 particles (images counted) asks for its sources first
instead of the Morton order: one launch instead of three, so the launch counts of
an evaluation show which was taken.  Bound on the relative L2 in mixed precision:
5e-6 (coordinates to 2^-25 of offsets of up to ~60 nm, neighbours ~2 nm apart,
r^-3 triples a relative error); 1e-12 in FP64.
"""
import numpy as np
import pytest

import oracle_py as O
import plume
import solveit_gpu as sv
from gpu_util import rel_l2

pytestmark = pytest.mark.gpu

EPS20 = 1e-20
BOUND = {sv.MIXED: 5e-6, sv.FP64: 1e-12}


def state(n, seed):
    st = plume.make_plume(n, max(2e-8, n * 2.4e-10), seed)
    rng = np.random.default_rng(seed)
    st["q"] = rng.choice([1.0, 2.0, 3.0], n)
    st["status"] = rng.choice(np.array([1, 2, 0, -1], np.int32), n, p=[0.7, 0.2, 0.05, 0.05])
    st["status"][: n // 3] = 0
    st["status"][n // 2] = 1
    st["x"] += np.array([1e-3, -2e-3, 5e-3])
    return st


def evaluate(fm, n, ref, st, bound):
    before = fm.launches
    a = fm.accel()
    assert rel_l2(a, ref, st["status"]) < bound
    assert not np.any(a[st["status"] != 1])
    return fm.launches - before


@pytest.mark.parametrize("prec", [sv.MIXED, sv.FP64], ids=["mixed", "fp64"])
def test_first_and_later_evaluations(prec):
    counts = {}
    for n in (3, 257, 8191, 8192, 8193):
        st = state(n, 50 + n)
        ref = O.direct_f64(st, EPS20)
        with sv.ForceMethod(softening2=EPS20, method=sv.DIRECT, precision=prec) as fm:
            fm.upload(st)
            counts[n] = [evaluate(fm, n, ref, st, BOUND[prec]) for _ in range(3)]
    for n, c in counts.items():
        assert c[0] == c[1] == c[2], (n, c)
    # bounds, chunks and ranks where the Morton order is taken, one launch otherwise
    assert counts[8191] == counts[8192] == counts[257]
    assert counts[8193][0] == counts[8192][0] + 2


def test_a_larger_plume_after_a_small_one():
    with sv.ForceMethod(softening2=EPS20, method=sv.DIRECT) as fm:
        counts = []
        for n in (300, 5000, 8192, 8192):
            st = state(n, 80 + n)
            fm.upload(st)
            counts.append(evaluate(fm, n, O.direct_f64(st, EPS20), st, BOUND[sv.MIXED]))
    assert len(set(counts)) == 1, counts


@pytest.mark.parametrize("prec", [sv.MIXED, sv.FP64], ids=["mixed", "fp64"])
@pytest.mark.parametrize("sym,edge", [("rotational", 4096), ("translational", 2730)])
def test_images(sym, edge, prec):
    """The edge with images: n^2 times their number up to 8,192^2."""
    counts = []
    for n in (edge, edge + 1):
        st = state(n, 90 + n)
        st["x"] -= np.array([1e-3, -2e-3, 5e-3])
        if sym == "rotational":
            ref = O.direct_f64(st, EPS20, sym=1)
            kw = dict(symmetry=sv.SYM_ROTATIONAL)
        else:
            ref = O.direct_f64(st, EPS20, sym=2, img_off=O.trans_images(1, (1, 1, 0)) * np.array([2e-6, 2e-6, 0.0]))
            kw = dict(symmetry=sv.SYM_TRANSLATIONAL, sym_axes=(1, 1, 0), sym_levels=1, domain_size=(2e-6, 2e-6, 0.0))
        with sv.ForceMethod(softening2=EPS20, method=sv.DIRECT, precision=prec, **kw) as fm:
            fm.upload(st)
            c = [evaluate(fm, n, ref, st, BOUND[prec]) for _ in range(2)]
        assert c[0] == c[1], (n, c)
        counts.append(c[0])
    assert counts[1] == counts[0] + 2, counts
