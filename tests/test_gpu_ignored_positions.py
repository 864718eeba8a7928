"""Particles that take no part may be anywhere: lost ions far away do not change the others' forces.

The mixed direct sum and the adjoint take FP32 coordinates from an origin per block of
particles, and an ignored particle must not become one.  Half of the ions are lost and
sit up to some kilometres off; the others' forces meet the mixed direct sum's bound
(5e-6 relative L2: coordinates to 2^-25 of offsets of up to ~60 nm, neighbours
~2 nm apart, r^-3 triples a relative error), and the gradients those of the FP64
adjoint (1e-4).  Sizes take the sources-first order (two block sizes) and the Morton order.
"""
import ctypes as C

import numpy as np
import pytest

import oracle_py as O
import plume
import solveit_gpu as sv
from gpu_util import rel_l2

pytestmark = pytest.mark.gpu

EPS20 = 1e-20


def state(n, far=1e3):
    st = plume.make_plume(n, max(1e-7, n * 2.5e-10), 60 + n)
    rng = np.random.default_rng(n)
    off = rng.random(n) < 0.5
    off[n // 2] = False
    st["status"][off] = np.where(rng.random(off.sum()) < 0.5, 0, -1)
    st["x"][off] = rng.normal(size=(off.sum(), 3)) * far
    return st


@pytest.mark.parametrize("sym", [sv.SYM_NONE, sv.SYM_ROTATIONAL], ids=["none", "rotational"])
@pytest.mark.parametrize("n", [300, 700, 3001, 9001])
def test_forces(n, sym):
    st = state(n)
    ref = O.direct_f64(st, EPS20, sym=1 if sym == sv.SYM_ROTATIONAL else 0)
    with sv.ForceMethod(softening2=EPS20, method=sv.DIRECT, symmetry=sym) as fm:
        fm.upload(st)
        for _ in range(2):
            a = fm.accel()
            assert rel_l2(a, ref, st["status"]) < 5e-6
            assert not np.any(a[st["status"] != 1])


@pytest.mark.parametrize("n", [700, 9001])
def test_allocation_free_forces(n):
    torch = pytest.importorskip("torch")
    st = state(n)
    L = sv.load()
    L.sv_direct_accel_noalloc.restype = C.c_int
    d = [torch.as_tensor(np.ascontiguousarray(st[k]), device="cuda:0") for k in ("x", "q", "m", "status")]
    out = torch.empty((n, 3), dtype=torch.float64, device="cuda:0")
    rc = L.sv_direct_accel_noalloc(C.c_int64(n), *[C.c_void_p(t.data_ptr()) for t in d], C.c_double(EPS20),
                                   C.c_double(sv.default_params().k_const), C.c_void_p(out.data_ptr()),
                                   C.c_void_p(torch.cuda.current_stream(0).cuda_stream))
    assert rc == 0
    assert rel_l2(out.cpu().numpy(), O.direct_f64(st, EPS20), st["status"]) < 5e-6


@pytest.mark.parametrize("n", [400, 9001])
def test_gradients(n):
    st = state(n)
    rng = np.random.default_rng(n)
    live = (st["status"] == 1)[:, None]
    gx, gv = rng.normal(size=(n, 3)) * live, rng.normal(size=(n, 3)) * 1e-12 * live
    out = []
    for prec in (sv.FP64, sv.MIXED):
        with sv.ForceMethod(softening2=EPS20, method=sv.DIRECT, precision=prec, efield=(0.0, 0.0, 1e8)) as fm:
            fm.upload(st)
            fm.adjoint_forward(2, 1e-13, 0.0, 1)
            out.append(fm.adjoint_backward(gx, gv))
    for a, b in zip(*out):
        assert np.linalg.norm(a - b) <= 1e-4 * np.linalg.norm(a)
