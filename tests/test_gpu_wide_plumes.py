"""Plumes of tight clusters over metres: the mixed pair sums keep the FP64 positions' differences.

FP32 hi + lo parts resolve 2^-49 of a particle's distance from the plume's origin; from
1/32 m on the pair kernels keep a third part, all bits of the position, in the caller's
order (up to 8,192 particles) as in the Morton order, for clusters that fill whole
blocks and for clusters that alternate in the caller's order.  What is left is
the FP32 pair arithmetic: 2e-6 relative L2 per particle, the mixed direct sum's bound;
gradients within 1e-5 of the FP64 adjoint's (five powers of the distance, a few
steps).  Distances on both sides of the rule.
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


def clusters(n, k, size, d, alternate, seed=3):
    st = plume.make_plume(n, 1e-6, seed)
    rng = np.random.default_rng(seed)
    centres = (rng.random((k, 3)) - 0.5) * 2 * d
    which = np.arange(n) % k if alternate else np.arange(n) * k // n
    st["x"] = np.ascontiguousarray(centres[which] + rng.normal(size=(n, 3)) * size)
    return st


@pytest.mark.parametrize("charges", ["uniform", "mixed"])
@pytest.mark.parametrize("alternate", [False, True], ids=["grouped", "alternating"])
@pytest.mark.parametrize("n,k,size,d", [(300, 3, 1e-8, 10.0), (2048, 4, 1e-8, 10.0), (2500, 5, 1e-7, 10.0),
                                        (2048, 4, 1e-8, 0.012), (2048, 4, 1e-8, 0.05), (16384, 8, 1e-8, 1.0),
                                        (16384, 8, 1e-8, 10.0), (16384, 64, 1e-8, 10.0), (40000, 8, 1e-8, 10.0)])
def test_forces(n, k, size, d, alternate, charges):
    st = clusters(n, k, size, d, alternate)
    if charges == "mixed":
        rng = np.random.default_rng(n)
        st["q"] = rng.choice([1.0, 2.0], n)
        st["status"] = rng.choice(np.array([1, 2, 0], np.int32), n, p=[0.8, 0.1, 0.1])
        st["status"][0] = 1
    tg = np.arange(0, n, max(1, n // 2000))
    ref = O.direct_f64(st, EPS20, targets=tg)
    with sv.ForceMethod(softening2=EPS20, method=sv.DIRECT) as fm:
        fm.upload(st)
        for _ in range(2):
            assert rel_l2(fm.accel()[tg], ref, st["status"][tg]) < 2e-6


@pytest.mark.parametrize("sym", ["rotational", "translational"])
@pytest.mark.parametrize("n", [1200, 5000])
def test_images(sym, n):
    st = clusters(n, 4, 1e-8, 5.0, True)
    st["q"][::3] = 2.0
    kw, io = dict(symmetry=sv.SYM_ROTATIONAL), None
    if sym == "translational":
        io = O.trans_images(1, (1, 1, 0)) * np.array([2e-6, 2e-6, 0.0])
        kw = dict(symmetry=sv.SYM_TRANSLATIONAL, sym_axes=(1, 1, 0), sym_levels=1, domain_size=(2e-6, 2e-6, 0.0))
    ref = O.direct_f64(st, EPS20, sym=1 if io is None else 2, img_off=io)
    with sv.ForceMethod(softening2=EPS20, method=sv.DIRECT, **kw) as fm:
        fm.upload(st)
        for _ in range(2):
            assert rel_l2(fm.accel(), ref, st["status"]) < 2e-6


@pytest.mark.parametrize("n", [2048, 16384])
def test_allocation_free_forces(n):
    torch = pytest.importorskip("torch")
    st = clusters(n, 8, 1e-8, 10.0, False)
    L = sv.load()
    L.sv_direct_accel_noalloc.restype = C.c_int
    d = [torch.as_tensor(np.ascontiguousarray(st[k]), device="cuda:0") for k in ("x", "q", "m", "status")]
    out = torch.empty((n, 3), dtype=torch.float64, device="cuda:0")
    rc = L.sv_direct_accel_noalloc(C.c_int64(n), *[C.c_void_p(t.data_ptr()) for t in d], C.c_double(EPS20),
                                   C.c_double(sv.default_params().k_const), C.c_void_p(out.data_ptr()),
                                   C.c_void_p(torch.cuda.current_stream(0).cuda_stream))
    assert rc == 0
    tg = np.arange(0, n, max(1, n // 2000))
    assert rel_l2(out.cpu().numpy()[tg], O.direct_f64(st, EPS20, targets=tg), st["status"][tg]) < 2e-6


@pytest.mark.parametrize("n,d", [(600, 10.0), (9000, 1.0)])
def test_gradients(n, d):
    st = clusters(n, 4, 3e-8, d, True)
    st["v"][:] = 0.0
    rng = np.random.default_rng(n)
    gx, gv = rng.normal(size=(n, 3)), rng.normal(size=(n, 3)) * 1e-13
    out = []
    for prec in (sv.FP64, sv.MIXED):
        with sv.ForceMethod(softening2=EPS20, method=sv.DIRECT, precision=prec) as fm:
            fm.upload(st)
            fm.adjoint_forward(2, 1e-14, 0.0, 1)
            out.append(fm.adjoint_backward(gx, gv)[:2])
    for a, b in zip(*out):
        assert np.linalg.norm(a - b) <= 1e-5 * np.linalg.norm(a)
