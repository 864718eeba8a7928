"""The near field's split of a leaf box's targets over chunks, groups and CTAs.

A cube a little wider than a power of two under the largest root scale spans
about one leaf box of level 2, so every box is a near box of every other and
the FMM is the near field alone: it has to meet the mixed direct sum's bound
(2e-6 per-particle relative L2 against the FP64 oracle) whatever a box holds:
one target, odd counts, counts around the chunk and group sizes, more than one
chunk per box, uniform and mixed charges, sources that are no targets.
"""
import numpy as np
import pytest

import oracle_py as O
import plume
import solveit_gpu as sv
from gpu_util import rel_l2

pytestmark = pytest.mark.gpu

EPS20 = 1e-20


def cube(n, seed):
    st = plume.make_plume(n, 1e-6, seed)
    side = 2.0 ** -23 * 1.0001
    x = np.random.default_rng(seed).random((n, 3)) * side
    x[0], x[-1] = 0.0, side
    st["x"] = np.ascontiguousarray(x)
    return st


@pytest.mark.parametrize("mixed", [False, True])
@pytest.mark.parametrize("ws", [1, 2])
@pytest.mark.parametrize("n", [2, 9, 63, 257, 1021, 2311, 9000])
def test_near_field_alone(n, ws, mixed):
    st = cube(n, 77 + n)
    if mixed:
        rng = np.random.default_rng(n)
        st["q"] = rng.choice([1.0, 2.0, -1.0], n)
        st["status"] = rng.choice(np.array([1, 2], np.int32), n, p=[0.8, 0.2])
        st["status"][0] = 1
    ref = O.direct_f64(st, EPS20)
    with sv.ForceMethod(softening2=EPS20, method=sv.FMM, fmm_order=4, fmm_ws=ws, fmm_root_scale=1.875,
                        fmm_leaf_target=4096) as fm:
        fm.upload(st)
        a = fm.accel()
        s = fm.stats()
    assert s.cell_interactions == 0 and s.pair_interactions >= float((st["status"] == 1).sum()) * n
    assert rel_l2(a, ref, st["status"]) < 2e-6


def test_forest_near_field_alone():
    """The same through the forest's work queue: several plumes, one of them with many chunks per box."""
    states = [cube(n, 500 + n) for n in (8200, 30, 12000)]
    with sv.ForceMethod(softening2=EPS20, fmm_order=10, fmm_ws=2) as fm:
        fm.upload_batch(states, [sv.FMM] * 3, [sv.SYM_NONE] * 3)
        a = fm.accel()
    o = 0
    for st in states:
        n = st["q"].size
        assert rel_l2(a[o:o + n], O.direct_f64(st, EPS20), st["status"]) < 1e-5
        o += n


@pytest.mark.parametrize("mixed", [False, True])
@pytest.mark.parametrize("ws", [1, 2])
@pytest.mark.parametrize("n", [1, 40, 129, 700, 3001])
def test_images_leave_the_targets_lanes(n, ws, mixed):
    """Boxes of image copies and targets together: the targets alone are gathered (one or
    several rounds of 128 particles, one or several chunks), the images and source-only
    particles pull.  The cube sits on the rotation axis, so that every box holds all four
    quadrants' copies."""
    st = cube(max(n, 2), 900 + n)
    st["x"][:, :2] -= 2.0 ** -24
    if n == 1:
        st["status"][1:] = 2
    if mixed:
        rng = np.random.default_rng(n)
        st["q"] = rng.choice([1.0, 2.0, -1.0], st["q"].size)
        st["status"][1:] = rng.choice(np.array([1, 2], np.int32), st["q"].size - 1, p=[0.5, 0.5])
    ref = O.direct_f64(st, EPS20, sym=1)
    with sv.ForceMethod(softening2=EPS20, method=sv.FMM, symmetry=sv.SYM_ROTATIONAL, fmm_order=4, fmm_ws=ws,
                        fmm_root_scale=1.875, fmm_leaf_target=4096) as fm:
        fm.upload(st)
        a = fm.accel()
        s = fm.stats()
    assert s.cell_interactions == 0
    assert rel_l2(a, ref, st["status"]) < 2e-6
    assert not np.any(a[st["status"] != 1])


@pytest.mark.parametrize("sizes", [(8200, 30, 12000), (9001,), (20011, 8193)])
def test_forest_work_list(sizes):
    """The forest's list of work items, largest first: plumes of very different density, every
    other one with image copies, source-only particles among them.  Order 10 keeps the far field
    below the bound wherever the levels fall."""
    states = []
    for k, n in enumerate(sizes):
        st = plume.make_plume(n, (0.4e-6, 3e-6)[k % 2], 40 + n)
        st["status"][3::7] = 2
        states.append(st)
    syms = [(sv.SYM_ROTATIONAL, sv.SYM_NONE)[k % 2] for k in range(len(sizes))]
    with sv.ForceMethod(softening2=EPS20, fmm_order=10, fmm_ws=2) as fm:
        fm.upload_batch(states, [sv.FMM if n > 1000 else sv.DIRECT for n in sizes], syms)
        a = fm.accel()
    o = 0
    for st, sym in zip(states, syms):
        n = st["q"].size
        ref = O.direct_f64(st, EPS20, sym=1 if sym == sv.SYM_ROTATIONAL else 0)
        assert rel_l2(a[o:o + n], ref, st["status"]) < 1e-5
        assert not np.any(a[o:o + n][st["status"] != 1])
        o += n
