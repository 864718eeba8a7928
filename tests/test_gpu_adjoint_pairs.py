"""The adjoint's pair kernels and its kept segment against a dense FP64 reverse sweep.

The reference walks the same leapfrog steps and their transposes in numpy.
Sizes are the edges of a lane tile (32) and of a block (128), with uniform and
mixed charges, source-only and ignored particles and ions injected on the way.
Bounds: 1e-9 for the FP64 adjoint (summation order over a few steps), 1e-4 for
the mixed one (the bound it is held to against the FP64 adjoint).  A second
backward pass, and one after the state was replaced by itself, re-run every
segment and have to give what the first gave.
"""
import numpy as np
import pytest

import oracle_py as O
import plume
import solveit_gpu as sv

pytestmark = pytest.mark.gpu

EPS2, DT, EZ = 1e-20, 1e-13, 1e8


def state(n, mixed):
    st = plume.make_plume(n, max(4e-8, n * 1e-9), 8000 + n)
    if mixed:
        rng = np.random.default_rng(n)
        st["q"] = rng.choice([1.0, 2.0], n)
        st["status"] = rng.choice(np.array([1, 2, 0], np.int32), n, p=[0.7, 0.2, 0.1])
        st["status"][0] = 1
        st["t_inj"][n // 2:] = rng.random(n - n // 2) * 3 * DT
    return st


def reference(st, steps, gx, gv):
    K, q, m, t_inj, w = O.k_const(), st["q"], st["m"], st["t_inj"], st["status"]
    move = (w == 1) | (w == 2)
    c = O.e_over_amu() * q / m

    def pairs(x):
        d = x[:, None] - x[None]
        return d, (d * d).sum(2) + EPS2

    x, v, tape = st["x"].copy(), st["v"].copy(), []
    for s in range(steps):
        ts = s * DT
        h1 = np.clip(ts + DT / 2 - t_inj, 0, DT / 2) * move
        xh = x + h1[:, None] * v
        win = t_inj <= ts + DT / 2
        tgt, src = (w == 1) & win, move & win
        k = np.clip(ts + DT - t_inj, 0, DT) * tgt
        d, r2 = pairs(xh)
        a = (K * q / m * tgt)[:, None] * ((q * src)[None] * r2 ** -1.5)[:, :, None].__mul__(d).sum(1)
        a[:, 2] += c * EZ
        v = v + k[:, None] * a
        h2 = np.clip(ts + DT - t_inj, 0, DT / 2) * move
        x = xh + h2[:, None] * v
        tape.append((h1, xh, tgt, src, k, h2))
    lx, lv = gx(x, v).copy(), gv(x, v).copy()
    fx, fv = lx.copy(), lv.copy()
    lE = np.zeros(3)
    for h1, xh, tgt, src, k, h2 in reversed(tape):
        lv = lv + h2[:, None] * lx
        la = k[:, None] * lv
        lE += ((c * (w == 1))[:, None] * la).sum(0)
        u = (K * q / m * tgt)[:, None] * la
        qs = q * src
        d, r2 = pairs(xh)
        wv = qs[None, :, None] * u[:, None] - qs[:, None, None] * u[None]
        lx = lx + (wv * r2[:, :, None] ** -1.5 - 3 * ((d * wv).sum(2) * r2 ** -2.5)[:, :, None] * d).sum(1)
        lv = lv + h1[:, None] * lx
    return (lx, lv, lE), fx, fv


def gx_of(x, v):
    g = np.zeros_like(x)
    g[:, :2] = x[:, :2] / np.sqrt(x[:, 0] ** 2 + x[:, 1] ** 2)[:, None]
    return g


def gv_of(x, v):
    return v * 1e-14


@pytest.mark.parametrize("prec,tol", [(sv.FP64, 1e-9), (sv.MIXED, 1e-4)], ids=["fp64", "mixed"])
@pytest.mark.parametrize("mixed", [False, True], ids=["uniform", "mixed"])
@pytest.mark.parametrize("n,every", [(1, 1), (2, 2), (31, 1), (33, 5), (127, 2), (129, 3), (257, 2), (400, 1)])
def test_against_dense_reverse(n, every, mixed, prec, tol):
    st = state(n, mixed)
    steps = 4
    ref, fx, fv = reference(st, steps, gx_of, gv_of)
    with sv.ForceMethod(softening2=EPS2, precision=prec, efield=(0.0, 0.0, EZ)) as fm:
        fm.upload(st)
        fm.adjoint_forward(steps, DT, 0.0, every)
        got = fm.adjoint_backward(fx, fv)
        again = fm.adjoint_backward(fx, fv)
        x, v, _ = fm.download()
        fm.update_state(x, v)
        third = fm.adjoint_backward(fx, fv)
    for g, a, t, r in zip(got, again, third, ref):
        assert np.linalg.norm(g - r) <= tol * np.linalg.norm(r)
        # the same sums, their order over the GPU apart
        assert np.linalg.norm(a - g) <= 1e-11 * np.linalg.norm(g)
        assert np.linalg.norm(t - g) <= 1e-11 * np.linalg.norm(g)
