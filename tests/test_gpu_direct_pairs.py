"""The direct sum's pair kernels: every unordered pair of particle blocks once.

Against the FP64 oracle at the edges of a lane tile (32), of a block (64 below
2,048 particles, 256 above), even and odd block counts, the change of block
size, uniform and mixed charges, source-only and ignored particles, few
targets, no softening, and the symmetry images (the reaction on the travelling
particle turned or shifted back).  Bounds on the per-particle relative L2: 1e-12 in FP64;
in mixed precision 5e-6: coordinates are rounded to 2^-25 of offsets of up to
~60 nm (2e-15 m), nearest neighbours are ~2 nm apart and r^-3 triples a relative
error (3e-6), the FP32 sums adding a few 1e-7.
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


def state(n, mixed, seed):
    st = plume.make_plume(n, max(2e-8, n * 2.4e-10), seed)
    if mixed:
        rng = np.random.default_rng(seed)
        st["q"] = rng.choice([1.0, 2.0, 3.0], n)
        st["status"] = rng.choice(np.array([1, 2, 0, -1], np.int32), n, p=[0.7, 0.2, 0.05, 0.05])
        st["status"][0] = 1
    return st


def accel(st, **kw):
    with sv.ForceMethod(method=sv.DIRECT, **kw) as fm:
        fm.upload(st)
        return fm.accel()


@pytest.mark.parametrize("prec", [sv.MIXED, sv.FP64], ids=["mixed", "fp64"])
@pytest.mark.parametrize("charges", ["uniform", "mixed"])
@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 64, 65, 129, 193, 2047, 2048, 2049, 2305, 4097])
def test_block_edges(n, charges, prec):
    st = state(n, charges == "mixed", 300 + n)
    a = accel(st, softening2=EPS20, precision=prec)
    assert rel_l2(a, O.direct_f64(st, EPS20), st["status"]) < BOUND[prec]
    assert not np.any(a[st["status"] != 1])


@pytest.mark.parametrize("prec", [sv.MIXED, sv.FP64], ids=["mixed", "fp64"])
@pytest.mark.parametrize("n", [70, 2500])
def test_few_targets_and_no_softening(n, prec):
    st = state(n, False, 7)
    st["status"][:] = 2
    st["status"][[0, n // 2, n - 1]] = 1
    a = accel(st, softening2=0.0, precision=prec)
    assert rel_l2(a, O.direct_f64(st, 0.0), st["status"]) < BOUND[prec]


@pytest.mark.parametrize("prec", [sv.MIXED, sv.FP64], ids=["mixed", "fp64"])
@pytest.mark.parametrize("n", [45, 700, 2100])
@pytest.mark.parametrize("sym", ["rotational", "translational"])
def test_images(sym, n, prec):
    st = state(n, True, 40 + n)
    if sym == "rotational":
        ref = O.direct_f64(st, EPS20, sym=1)
        kw = dict(symmetry=sv.SYM_ROTATIONAL)
    else:
        ref = O.direct_f64(st, EPS20, sym=2, img_off=O.trans_images(1, (1, 1, 0)) * np.array([2e-6, 2e-6, 0.0]))
        kw = dict(symmetry=sv.SYM_TRANSLATIONAL, sym_axes=(1, 1, 0), sym_levels=1, domain_size=(2e-6, 2e-6, 0.0))
    a = accel(st, softening2=EPS20, precision=prec, **kw)
    assert rel_l2(a, ref, st["status"]) < BOUND[prec]


@pytest.mark.parametrize("n", [64, 97, 1024])
def test_fp64_tiles_of_equal_charges(n):
    """Charges that differ between regions only: pairs of tiles with one charge take the
    sum without them, pairs of tiles with two do not; source-only and ignored particles mixed in."""
    st = state(n, False, 90 + n)
    st["q"] = np.where(st["x"] < np.median(st["x"]), 2.0, -1.0)
    st["status"][5::17] = 2
    st["status"][7::19] = 0
    a = accel(st, softening2=EPS20, precision=sv.FP64)
    assert rel_l2(a, O.direct_f64(st, EPS20), st["status"]) < BOUND[sv.FP64]


@pytest.mark.parametrize("prec", [sv.MIXED, sv.FP64], ids=["mixed", "fp64"])
@pytest.mark.parametrize("n", [3, 255, 257, 8191, 8192, 8193])
def test_sources_first(n, prec):
    """Around the size up to which the sources are only put before the other particles: the first
    particles and others in between are none, the plume lies far from the origin, and its blocks
    spread over all of it."""
    st = state(n, True, 600 + n)
    st["status"][: n // 3] = 0
    st["status"][n // 2] = 1
    st["x"] += np.array([1e-3, -2e-3, 5e-3])
    a = accel(st, softening2=EPS20, precision=prec)
    assert rel_l2(a, O.direct_f64(st, EPS20), st["status"]) < BOUND[prec]
    assert not np.any(a[st["status"] != 1])


@pytest.mark.parametrize("n", [4096, 4097])
def test_sources_first_with_images(n):
    """The same at the size of the four quadrants (an image counts as a particle's pairs do)."""
    st = state(n, True, 700 + n)
    st["status"][:5] = 0
    a = accel(st, softening2=EPS20, precision=sv.MIXED, symmetry=sv.SYM_ROTATIONAL)
    assert rel_l2(a, O.direct_f64(st, EPS20, sym=1), st["status"]) < BOUND[sv.MIXED]
