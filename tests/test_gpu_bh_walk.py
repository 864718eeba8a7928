"""The Barnes-Hut walk's batches of cells, its bounded stack and its image split.

At theta 0 every cell is opened, so the walk visits the whole tree (the largest
stack it can need) and equals the direct sum to FP32 accumulation: 2e-6 per
particle up to a few thousand sources, as the walk is held to elsewhere.  Trees:
a column, tight clusters in a large box (deep, narrow), repeated positions
(leaves at the finest level that no split can empty); 8, 16 and 32 targets per
warp by size; single-particle and large leaves; both kinds of images.  At theta
0.5 the accepted cells and pairs are counted per target and do not depend on
how targets share warps.
"""
import numpy as np
import pytest

import oracle_py as O
import plume
import solveit_gpu as sv
from gpu_util import rel_l2

pytestmark = pytest.mark.gpu

EPS20 = 1e-20


def make(kind, n):
    st = plume.make_plume(n, max(1e-7, n * 2e-10), 17 + n)
    rng = np.random.default_rng(n)
    if kind == "clusters":
        centres = rng.random((5, 3)) * 1e-4
        st["x"] = centres[rng.integers(0, 5, n)] + rng.normal(size=(n, 3)) * 1e-8
    elif kind == "repeated":
        k = n // 3
        st["x"][:k] = st["x"][k:2 * k]
        st["x"][2 * k:2 * k + 90] = st["x"][0]
    st["status"] = rng.choice(np.array([1, 2, 0], np.int32), n, p=[0.85, 0.1, 0.05])
    st["status"][0] = 1
    return st


@pytest.mark.parametrize("leaf", [1, 16, 64])
@pytest.mark.parametrize("kind", ["column", "clusters", "repeated"])
@pytest.mark.parametrize("n", [3, 40, 1500, 5000])
def test_theta_zero_is_the_direct_sum(n, kind, leaf):
    if kind == "repeated" and n < 300:
        pytest.skip("the repeated positions need a few hundred particles")
    st = make(kind, n)
    ref = O.direct_f64(st, EPS20)
    with sv.ForceMethod(softening2=EPS20, method=sv.BARNES_HUT, theta=0.0, leaf_size=leaf) as fm:
        fm.upload(st)
        a = fm.accel()
        s = fm.stats()
    assert s.cell_interactions == 0
    src = np.isin(st["status"], (1, 2)).sum()
    assert s.pair_interactions == (st["status"] == 1).sum() * (src - 1)
    assert rel_l2(a, ref, st["status"]) < 2e-6


@pytest.mark.parametrize("sym", [sv.SYM_ROTATIONAL, sv.SYM_TRANSLATIONAL], ids=["rotational", "translational"])
@pytest.mark.parametrize("n", [40, 1300])
def test_theta_zero_images(n, sym):
    st = make("column", n)
    img = O.trans_images(1, (1, 1, 0)) * np.array([2e-6, 2e-6, 0.0]) if sym == sv.SYM_TRANSLATIONAL else None
    ref = O.direct_f64(st, EPS20, sym=sym, img_off=img)
    with sv.ForceMethod(softening2=EPS20, method=sv.BARNES_HUT, theta=0.0, leaf_size=8, symmetry=sym,
                        sym_axes=(1, 1, 0), sym_levels=1, domain_size=(2e-6, 2e-6, 0.0)) as fm:
        fm.upload(st)
        a = fm.accel()
    assert rel_l2(a, ref, st["status"]) < 2e-6


def test_counts_do_not_depend_on_the_warp_split():
    """The same particles alone (8 targets per warp) and as targets among sources in a larger evaluation's rule."""
    n = 6000
    st = make("column", n)
    counts = []
    for keep in (n, 700):  # all inbound ions as targets, then a part of them
        s2 = dict(st, status=np.where((st["status"] == 1) & (np.arange(n) >= keep), 2, st["status"]).astype(np.int32))
        with sv.ForceMethod(softening2=EPS20, method=sv.BARNES_HUT, theta=0.5, leaf_size=16) as fm:
            fm.upload(s2)
            counts.append((fm.accel(), fm.stats()))
    t = (st["status"] == 1) & (np.arange(n) < 700)
    assert rel_l2(counts[1][0][t], counts[0][0][t], st["status"][t]) < 2e-6
