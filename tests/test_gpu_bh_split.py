"""The Barnes-Hut walk gives the same cells, pairs and forces with 8, 16 and 32 targets per warp.

The walk takes 32 targets per warp from 32 such warps per SM on, 16 from 8, else 8;
every image counts.  38,000 ions without images take 8; images a kilometre away put the
same plume above the other two lines, and each of them adds exactly one accepted cell
per target, the root.  Sampled targets against the FP64 oracle hold the
multipole error of theta 0.5 (2e-2 relative L2 per particle).
"""
import numpy as np
import pytest

import oracle_py as O
import plume
import solveit_gpu as sv
from gpu_util import rel_l2

pytestmark = pytest.mark.gpu

EPS20 = 1e-20


@pytest.mark.parametrize("leaf", [1, 16])
def test_counts_and_forces(leaf):
    n = 38000
    st = plume.make_plume(n, 6e-6, 5)
    rng = np.random.default_rng(5)
    st["status"] = rng.choice(np.array([1, 2, 0], np.int32), n, p=[0.85, 0.14, 0.01])
    targets = int((st["status"] == 1).sum())
    got = []
    for axes in ((0, 0, 0), (1, 0, 0), (1, 1, 0)):
        images = 3 ** sum(axes)
        kw = dict(symmetry=sv.SYM_TRANSLATIONAL, sym_axes=axes, sym_levels=1, domain_size=(1e3, 1e3, 1e3))
        with sv.ForceMethod(softening2=EPS20, method=sv.BARNES_HUT, theta=0.5, leaf_size=leaf,
                            **(kw if images > 1 else {})) as fm:
            fm.upload(st)
            for _ in range(2):  # the second order takes the tree's own number of key levels
                a = fm.accel()
                s = fm.stats()
                got.append((a, s.cell_interactions - (images - 1) * targets, s.pair_interactions))
    for a, cells, pairs in got[1:]:
        assert (cells, pairs) == got[0][1:]
        # the same cells and pairs, the order of the FP32 sums apart
        assert rel_l2(a, got[0][0], st["status"]) < 2e-6
    tg = np.arange(0, n, 40)
    assert rel_l2(got[0][0][tg], O.direct_f64(st, EPS20, targets=tg), st["status"][tg]) < 2e-2


@pytest.mark.parametrize("n,sym", [(40001, sv.SYM_ROTATIONAL), (160001, sv.SYM_NONE)], ids=["images", "plain"])
def test_widest_split_against_the_oracle(n, sym):
    """32 targets per warp, ragged: every cell opened near the target, a small opening angle elsewhere."""
    st = plume.make_plume(n, n * 1.5e-10, 9)
    tg = np.arange(0, n, n // 400)
    with sv.ForceMethod(softening2=EPS20, method=sv.BARNES_HUT, theta=0.1, leaf_size=16, symmetry=sym) as fm:
        fm.upload(st)
        a = fm.accel()
    ref = O.direct_f64(st, EPS20, targets=tg, sym=1 if sym == sv.SYM_ROTATIONAL else 0)
    assert rel_l2(a[tg], ref, st["status"][tg]) < 1e-3
