"""The work that a SOLVEiT user has this framework do, as timed cases.

Each case goes through the public entry points (the Python binding of the C
ABI, solveit-code_gb300/solveit_gpu.py) on seeded synthetic plumes
(solveit-code_gb300/plume.py).  Four kinds of pass:

  drop_in  one call of the reference's ForceCalculationMethod, as the adapter
           makes it every step: the reference's float4 arrays up
           (sv_upload_ref32), one force evaluation, the acceleration added
           into the caller's float4 array (sv_add_accel_ref32);
  run      a trajectory segment: positions and velocities set from the
           program's page-locked arrays, a few leapfrog steps on the device, the
           state read back (in the reference's float4 arrays; in FP64 for the
           plain FP64 path);
  batch    the same for many independent plumes in one context;
  adjoint  forward rollout, loss gradient at the final state, backward
           rollout; the gradients in the float32 of a torch program's parameters.
"""
import ctypes as C
import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "solveit-code_gb300")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import plume  # noqa: E402
import solveit_gpu as sv  # noqa: E402

EPS2 = 1e-20      # softening 1e-10 m, squared
EZ = 1e8          # uniform field, V/m
DT = 1e-13        # s
DOMAIN = 2e-6     # period of the translational variant in x and y, m
METHOD = {"direct": sv.DIRECT, "bh": sv.BARNES_HUT, "fmm": sv.FMM}
SYM = {"none": sv.SYM_NONE, "rotational": sv.SYM_ROTATIONAL, "translational": sv.SYM_TRANSLATIONAL}


def _case(**kw):
    c = dict(kind="drop_in", method="direct", precision="mixed", sym="none", n=1024, length=1e-6, shape="column",
             statuses="inbound", inject=False, steps=1, theta=0.5, leaf=16, order=8, ws=2, near=0, root_scale=1.0,
             levels=1, plumes=0, every=1)
    c.update(kw)
    return c


def listed():
    return [
        # the smallest plumes of a study, early in the injection: the call's own latency
        _case(name="drop_in_direct_n256", n=256),
        # an ordinary direct force call on a ragged count, with ions that only act as sources or have left
        _case(name="drop_in_direct_n30011", n=30011, length=7e-6, statuses="mixed"),
        # the finite periodic lattice, 81 images, by the direct sum
        _case(name="drop_in_direct_periodic_n3001", n=3001, sym="translational", levels=2),
        # the plain FP64 path: the reference's own direct leapfrog at N = 4096
        _case(name="run_direct_fp64_n4096", kind="run", precision="fp64", n=4096, steps=10),
        # the Barnes-Hut leapfrog at its configured size
        _case(name="run_bh_n65536", kind="run", method="bh", n=65536, length=10e-6, steps=4),
        # Barnes-Hut as a force call in the 4-fold rotational sector, odd count
        _case(name="drop_in_bh_rotational_n9973", method="bh", n=9973, length=2e-6, sym="rotational", theta=0.7,
              leaf=8),
        # the library's default FMM (the reference's interaction lists) as a force call
        _case(name="drop_in_fmm_ws1_n20011", method="fmm", n=20011, length=2e-6, ws=1),
        # a plume that has expanded in all three dimensions, ions still being injected
        _case(name="run_fmm_ball_n131101", kind="run", method="fmm", n=131101, shape="ball", length=3e-7, order=6,
              near=2, inject=True, steps=3),
        # the headline: one million ions, p = 8, below 1e-5 force error
        _case(name="run_fmm_n1m", kind="run", method="fmm", n=1 << 20, length=50e-6, root_scale=1.375, steps=4),
        # many realisations at once: direct below 8192 ions, FMM above, every other one rotational
        _case(name="batch_24_plumes", kind="batch", method="fmm", plumes=24, n=24000, order=6, near=2, steps=2),
        # gradients of a short rollout, checkpointed
        _case(name="adjoint_n4096", kind="adjoint", n=4096, steps=8, every=4),
        # gradients at the configured plume size, FP32 pairs
        _case(name="adjoint_n16384", kind="adjoint", n=16384, steps=4, every=2),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    k = rng.choice(["small", "direct", "direct", "images", "fp64", "bh", "bh_sym", "fmm", "fmm", "fmm_run", "batch",
                    "adjoint"])
    if k == "small":
        return _case(n=_log(rng, 64, 4096), sym=rng.choice(["none", "rotational"]),
                     statuses=rng.choice(["inbound", "mixed"]))
    if k == "direct":
        n = _log(rng, 2000, 60000)
        return _case(kind=rng.choice(["drop_in", "run"]), n=n, length=n * 2.4e-10, steps=rng.choice([1, 2, 3]),
                     statuses=rng.choice(["inbound", "mixed"]), inject=rng.random() < 0.3,
                     sym=rng.choice(["none", "none", "rotational"]) if n < 30000 else "none")
    if k == "images":
        return _case(n=_log(rng, 500, 4000), sym="translational", levels=rng.choice([1, 2]))
    if k == "fp64":
        return _case(kind=rng.choice(["run", "run", "drop_in"]), precision="fp64", n=_log(rng, 300, 6000),
                     steps=rng.randint(2, 10))
    if k == "bh":
        n = _log(rng, 1500, 70000)
        return _case(kind=rng.choice(["drop_in", "run"]), method="bh", n=n, length=n * 1.5e-10,
                     theta=rng.choice([0.4, 0.5, 0.6, 0.8]), leaf=rng.choice([4, 8, 16, 24]),
                     steps=rng.choice([1, 2, 4]), statuses=rng.choice(["inbound", "mixed"]))
    if k == "bh_sym":
        return _case(method="bh", n=_log(rng, 1000, 16000), theta=rng.choice([0.5, 0.7]), leaf=rng.choice([8, 16]),
                     sym=rng.choice(["rotational", "translational"]), levels=1)
    if k == "fmm":
        n = _log(rng, 3000, 200000)
        return _case(method="fmm", n=n, length=n * 1e-10, order=rng.choice([4, 6, 8, 10]), ws=rng.choice([1, 2]),
                     root_scale=rng.choice([1.0, 1.25, 1.5]), statuses=rng.choice(["inbound", "mixed"]),
                     sym=rng.choice(["none", "none", "rotational"]))
    if k == "fmm_run":
        n = _log(rng, 20000, 1 << 20)
        ball = n < 300000 and rng.random() < 0.5
        return _case(kind="run", method="fmm", n=n, shape="ball" if ball else "column",
                     length=3e-9 * n ** 0.4 if ball else n * 5e-11, order=rng.choice([6, 8]),
                     near=rng.choice([0, 2]), root_scale=rng.choice([1.0, 1.375, 1.625]), steps=rng.choice([1, 2, 3]),
                     inject=rng.random() < 0.3)
    if k == "batch":
        return _case(kind="batch", method="fmm", plumes=rng.randint(3, 24), n=_log(rng, 4000, 24000),
                     order=rng.choice([4, 6, 8]), near=rng.choice([0, 2]), steps=rng.choice([1, 2]))
    return _case(kind="adjoint", precision=rng.choice(["mixed", "mixed", "fp64"]), n=_log(rng, 300, 6000),
                 steps=rng.randint(2, 6), every=rng.randint(1, 4))


# ------------------------------------------------------------------ inputs --
def _plume(c, n, seed):
    if c["shape"] == "ball":
        st = plume.make_ball(n, c["length"], seed)
    else:
        st = plume.make_plume(n, c["length"], seed)
    rng = np.random.Generator(np.random.PCG64(seed + 104729))
    if c["statuses"] == "mixed":  # source-only, out-of-bounds and crashed ions among the inbound ones
        st["status"] = rng.choice(np.array([1, 2, 0, -1], np.int32), n, p=[0.9, 0.05, 0.03, 0.02])
    if c["inject"]:  # the last tenth of the ions enters during the segment
        late = n // 10
        st["t_inj"][n - late:] = np.sort(rng.random(late)) * c["steps"] * DT
    if c["sym"] == "rotational":
        # the simulated sector is the first quadrant
        st["x"][:, :2] = np.abs(st["x"][:, :2])
    return st


def _sizes(c, seed):
    """Plume sizes of a batch, about c["n"] each on average."""
    rng = np.random.Generator(np.random.PCG64(1000003))  # the study's plan: the same for every realisation
    return [int(k) for k in rng.integers(1024, 2 * c["n"] - 1024, c["plumes"])]


def _params(c):
    kw = dict(softening2=EPS2, efield=(0.0, 0.0, EZ), method=METHOD[c["method"]],
              precision=sv.FP64 if c["precision"] == "fp64" else sv.MIXED, theta=c["theta"], leaf_size=c["leaf"],
              fmm_order=c["order"], fmm_ws=c["ws"], fmm_near=c["near"], fmm_root_scale=c["root_scale"])
    if c["kind"] != "batch":
        kw["symmetry"] = SYM[c["sym"]]
    if c["sym"] == "translational":
        kw.update(sym_axes=(1, 1, 0), sym_levels=c["levels"], domain_size=(DOMAIN, DOMAIN, 0.0))
    return kw


def _pinned(a):
    t = torch.empty(a.shape, dtype=torch.from_numpy(a[:1]).dtype, pin_memory=True)
    out = t.numpy()
    out[...] = a
    return out


def _batch_plan(c, seed):
    sizes = _sizes(c, seed)
    states = [_plume(c, k, 1000 * (seed % 100000) + i) for i, k in enumerate(sizes)]
    methods = [sv.DIRECT if k < 8192 else sv.FMM for k in sizes]
    syms = [sv.SYM_ROTATIONAL if i % 2 == 0 else sv.SYM_NONE for i in range(len(sizes))]
    return states, methods, syms


def prepare(case, seed):
    c = case
    s = {"c": c, "fm": sv.ForceMethod(**_params(c))}
    fm = s["fm"]
    if c["kind"] == "batch":
        states, methods, syms = _batch_plan(c, seed)
        cat, counts = plume.concat(states)
        s["pin"] = {k: _pinned(cat[k]) for k in ("x", "v", "q", "m", "status", "t_inj")}
        s["counts"] = counts
        s["methods"] = np.array(methods, np.int32)
        s["syms"] = np.array(syms, np.int32)
        s["n"] = int(counts.sum())
        s["pos4"], s["vel4"], _, _ = plume.to_ref32(cat)
        return s
    st = _plume(c, c["n"], seed)
    s["n"] = c["n"]
    s["pos4"], s["vel4"], s["acc4"], s["t_inj"] = plume.to_ref32(st)
    if c["kind"] == "drop_in":
        return s
    fm.upload(st)
    s["x"], s["v"] = _pinned(st["x"]), _pinned(st["v"])
    if c["kind"] == "run" and c["precision"] == "fp64":
        s["xo"], s["vo"], s["so"] = _pinned(st["x"]), _pinned(st["v"]), _pinned(st["status"])
    return s


# -------------------------------------------------------------------- pass --
def _ptr(a):
    return a.ctypes.data_as(C.c_void_p)


def _ok(fm, rc):
    if rc != 0:
        raise sv.SolveitError(fm.L.sv_last_error(fm.h).decode())


def run(state):
    c, fm = state["c"], state["fm"]
    if c["kind"] == "drop_in":
        acc4 = state["acc4"]
        acc4[:, :3] = 0.0  # the integrator zeroes the accelerations before the call
        fm.upload_ref32(state["pos4"], state["vel4"], acc4, state["t_inj"])
        fm.accel(out=False)
        return {"acc4": fm.add_accel_ref32(acc4)}
    if c["kind"] == "run":
        fm.update_state(state["x"], state["v"])
        fm.leapfrog(c["steps"], DT, 0.0)
        if c["precision"] == "fp64":
            _ok(fm, fm.L.sv_download(fm.h, _ptr(state["xo"]), _ptr(state["vo"]), _ptr(state["so"])))
            return {"x": state["xo"], "v": state["vo"], "status": state["so"]}
        _ok(fm, fm.L.sv_download_ref32(fm.h, _ptr(state["pos4"]), _ptr(state["vel4"])))
        return {"pos4": state["pos4"], "vel4": state["vel4"]}
    if c["kind"] == "batch":
        p = state["pin"]
        _ok(fm, fm.L.sv_upload_batch(fm.h, len(state["counts"]), _ptr(state["counts"]), _ptr(state["methods"]),
                                     _ptr(state["syms"]), _ptr(p["x"]), _ptr(p["v"]), _ptr(p["q"]), _ptr(p["m"]),
                                     _ptr(p["status"]), _ptr(p["t_inj"])))
        fm.leapfrog(c["steps"], DT, 0.0)
        _ok(fm, fm.L.sv_download_ref32(fm.h, _ptr(state["pos4"]), _ptr(state["vel4"])))
        return {"pos4": state["pos4"], "vel4": state["vel4"]}
    # adjoint: L = 1e3 x mean transverse radius (m) of the final state
    n = state["n"]
    fm.update_state(state["x"], state["v"])
    fm.adjoint_forward(c["steps"], DT, 0.0, c["every"])
    x, v, _ = fm.download()
    gx, gv = np.zeros_like(x), np.zeros_like(v)
    gx[:, :2] = 1e3 / n * x[:, :2] / np.sqrt(x[:, 0] ** 2 + x[:, 1] ** 2)[:, None]
    dx, dv, de = fm.adjoint_backward(gx, gv)
    out = {k: torch.from_numpy(g).float() for k, g in (("dx0", dx), ("dv0", dv), ("dE", de))}
    if c["precision"] == "fp64":
        out.update(x=x, v=v)
    return out


# -------------------------------------------------------------------- work --
def _images(c):
    return {"none": 1, "rotational": 4, "translational": (3 ** c["levels"]) ** 2}[c["sym"]]


def _force_flops(method, c, n, images):
    """Algorithmic operations of one force evaluation: 20 per pair (or accepted cell) and the expansions'."""
    if method == "direct":
        return 20.0 * n * n * images
    if method == "bh":
        # accepted cells and leaf pairs per target: a few hundred at theta 0.5, growing with log n and 1 / theta^2
        return 20.0 * n * images * (6.0 * math.log2(max(n, 2)) / c["theta"] ** 2 + 2.0 * c["leaf"])
    # near field: 3^3 or 5^3 boxes of ~32 ions where the plume is resolved; thin columns fill a fraction of them
    near = {("ball", 1): 27, ("ball", 2): 93 if c["near"] == 2 else 125}.get((c["shape"], c["ws"]), 27 if c["ws"] == 1 else 67)
    p = c["order"]
    return n * (20.0 * 32 * near + 32.0 * (p * (p + 1) // 2)) * (1 if images == 1 else 2)


def work(case):
    c = case
    if c["kind"] == "batch":
        flops, n = 0.0, 0
        for i, k in enumerate(_sizes(c, 0)):
            flops += _force_flops("direct" if k < 8192 else "fmm", c, k, 4 if i % 2 == 0 else 1)
            n += k
        return {"bytes": float(n * (24 + 24 + 8 + 8 + 4 + 8 + 32)), "flops": flops * c["steps"]}
    n = c["n"]
    f = _force_flops(c["method"], c, n, _images(c))
    if c["kind"] == "drop_in":
        return {"bytes": float(n * (16 + 16 + 16 + 4 + 16)), "flops": f}
    if c["kind"] == "run":
        return {"bytes": float(n * (48 + (52 if c["precision"] == "fp64" else 32))), "flops": f * c["steps"]}
    # forward and the transposed Jacobian sum (about 45 operations per pair) of every step
    return {"bytes": float(n * (48 * 4 + 24)), "flops": c["steps"] * n * float(n) * (20 + 45)}


# ------------------------------------------------------------------- exact --
_E, _AMU, _EPS0 = np.float32(1.6021766e-19), np.float32(1.66053904e-27), np.float32(8.85419e-12)
_K = float(np.float32(_E * _E)) / (4 * math.pi * float(_EPS0) * float(_AMU))
_EOA = float(np.float32(_E / _AMU))
_MASS = {0: 111.0, 1: 309.0}


def _shifts(c):
    if c["sym"] == "rotational":
        return [("rot", g) for g in range(4)]
    if c["sym"] == "translational":
        h = 3 ** c["levels"] // 2
        return [("off", (i * DOMAIN, j * DOMAIN)) for i in range(-h, h + 1) for j in range(-h, h + 1)]
    return [("rot", 0)]


def _accel64(x, q, m, tgt, src, shifts):
    """The direct sum in FP64: acceleration of the particles of mask tgt from those of mask src, zero elsewhere."""
    a = torch.zeros_like(x)
    it = torch.nonzero(tgt).squeeze(1)
    xs, qs = x[src], q[src]
    rows = max(1, (1 << 25) // max(1, xs.shape[0]))
    for kind, g in shifts:
        ys = xs.clone()
        if kind == "off":
            ys[:, 0] += g[0]
            ys[:, 1] += g[1]
        else:
            for _ in range(g):
                ys = torch.stack([-ys[:, 1], ys[:, 0], ys[:, 2]], 1)
        for r in range(0, it.shape[0], rows):
            k = it[r:r + rows]
            d = [x[k, e][:, None] - ys[None, :, e] for e in range(3)]
            r2 = d[0] * d[0] + d[1] * d[1] + d[2] * d[2] + EPS2
            w = qs / (r2 * torch.sqrt(r2))
            a[k] += torch.stack([(w * d[e]).sum(1) for e in range(3)], 1)
    return a * (_K * q / m)[:, None]


def _leapfrog64(x, v, q, m, st, t_inj, steps, shifts, accel=None):
    tgt_all, act = st == 1, (st == 1) | (st == 2)
    field = torch.tensor([0.0, 0.0, EZ], dtype=torch.float64, device=x.device)
    h = 0.5 * DT
    for k in range(steps):
        ts = k * DT
        x = x + v * (torch.clamp(ts + h - t_inj, 0.0, h) * act)[:, None]
        win = t_inj <= ts + h
        a = _accel64(x, q, m, tgt_all & win, act & win, shifts) if accel is None else accel(x, q, m)
        a = a + _EOA * (q / m)[:, None] * field
        v = v + a * (torch.clamp(ts + DT - t_inj, 0.0, DT) * (tgt_all & win))[:, None]
        x = x + v * (torch.clamp(ts + DT - t_inj, 0.0, h) * act)[:, None]
    return x, v


def _dense(x, q, m):
    """The same sum over all pairs at once, differentiable (the self pair contributes nothing)."""
    d = x[:, None, :] - x[None, :, :]
    r2 = (d * d).sum(2) + EPS2
    w = q[None, :] / (r2 * torch.sqrt(r2))
    return (w[:, :, None] * d).sum(1) * (_K * q / m)[:, None]


def _to64(st):
    g = {k: torch.from_numpy(np.asarray(st[k], np.float64)).cuda() for k in ("x", "v", "q", "m", "t_inj")}
    g["status"] = torch.from_numpy(np.asarray(st["status"])).cuda()
    return g


def _vec4(x, w):
    return torch.cat([x, w[:, None]], 1).cpu().numpy()


def exact(case, seed):
    c = case
    if c["kind"] == "batch":
        states, _, syms = _batch_plan(c, seed)
        if sum(float(len(s["q"])) ** 2 * (4 if y else 1) for s, y in zip(states, syms)) * c["steps"] > 1.2e11:
            return None
        pos, vel = [], []
        for s, y in zip(states, syms):
            g = _to64(s)
            sh = [("rot", k) for k in range(4 if y == sv.SYM_ROTATIONAL else 1)]
            x, v = _leapfrog64(g["x"], g["v"], g["q"], g["m"], g["status"], g["t_inj"], c["steps"], sh)
            pos.append(_vec4(x, g["q"]))
            vel.append(_vec4(v, torch.from_numpy(s["species"].astype(np.float64)).cuda()))
        return {"pos4": np.concatenate(pos), "vel4": np.concatenate(vel)}
    n = c["n"]
    if float(n) * n * _images(c) * c["steps"] > 6e10:
        return None
    st = _plume(c, n, seed)
    if c["kind"] == "drop_in":
        pos4, vel4, acc4, t_inj = plume.to_ref32(st)
        g = _to64(dict(x=pos4[:, :3], v=vel4[:, :3], q=pos4[:, 3], m=st["m"], t_inj=t_inj, status=st["status"]))
        a = _accel64(g["x"], g["q"], g["m"], g["status"] == 1, (g["status"] == 1) | (g["status"] == 2), _shifts(c))
        return {"acc4": _vec4(a, g["status"].double())}
    g = _to64(st)
    if c["kind"] == "adjoint":
        if float(n) * n * c["steps"] > 1.1e9:
            return None
        x0, v0 = g["x"].requires_grad_(), g["v"].requires_grad_()
        e = torch.zeros(3, dtype=torch.float64, device=x0.device, requires_grad=True)

        def accel(x, q, m):
            return _dense(x, q, m) + _EOA * (q / m)[:, None] * e

        x, v = _leapfrog64(x0, v0, g["q"], g["m"], g["status"], g["t_inj"], c["steps"], None, accel)
        loss = 1e3 * torch.sqrt(x[:, 0] ** 2 + x[:, 1] ** 2).mean()
        dx, dv, de = (t.cpu() for t in torch.autograd.grad(loss, [x0, v0, e]))
        out = {"dx0": dx, "dv0": dv, "dE": de}
        if c["precision"] == "fp64":
            out.update(x=x.detach().cpu().numpy(), v=v.detach().cpu().numpy())
        return out
    x, v = _leapfrog64(g["x"], g["v"], g["q"], g["m"], g["status"], g["t_inj"], c["steps"], _shifts(c))
    if c["precision"] == "fp64":
        return {"x": x.cpu().numpy(), "v": v.cpu().numpy(), "status": None}
    return {"pos4": _vec4(x, g["q"]), "vel4": _vec4(v, torch.from_numpy(st["species"].astype(np.float64)).cuda())}
