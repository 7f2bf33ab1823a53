"""Performance cases of the operator path: what its users run, from the smallest calls to C2, C3 and C4 at full size.

A case is a dict of plain values; `prepare` builds the handle and uploads what a program has in hand, `run` is one pass
through the public entry points, `work` the bytes and operations it cannot do without, `exact` the same outputs from
plain torch in 64 bits. Kinds:

  dg    a coupled ocean run: `steps` mode-split steps, then the state staged to the host (output every `steps` steps).
        A mixed-precision run holds its 3D state in 32 bits, and its output file is written in 32 bits too.
  ens   an uneven ensemble advanced together, then every member's state read back
  amr   DG3DIntegration on a directionally refined mesh: `steps` LSRK45 steps, then the state read back; with 0 steps
        one compute_rhs of a host field, the reference's own call
  bz    a bathymetry smoothing solve (PCG to 1e-10)
  cnn   one forward and backward of the learned preconditioner's network on a batch of crops
"""
from __future__ import annotations

import math

import numpy as np
import torch

from drifter_b200 import configs
from drifter_b200.amr import DG3DIntegration
from drifter_b200.bezier import BezierSmoother
from drifter_b200.cnn import CNN
from drifter_b200.dg import DGConfig, Ensemble, OceanModel

DEV = "cuda"
F64 = torch.float64
LSRK_A = (0.0, -0.4178904745, -1.192151694643, -1.697784692471, -1.514183444257)
LSRK_B = (0.1496590219993, 0.3792103129999, 0.8229550293869, 0.6994504559488, 0.1530572479681)
CH = (16, 32, 32, 32, 16)  # the network's channels
AMR_DT = 1e-4  # the benchmark's step on these meshes
NSUB = 20  # barotropic subcycles per step, in every configuration


# ------------------------------------------------------------------------------------------ cases
def _dg(name, nx, ny, nz, order, precision, steps, flux="lf", tide=False, baroclinic=False):
    return dict(name=name, kind="dg", nx=nx, ny=ny, nz=nz, order=order, precision=precision, steps=steps, flux=flux,
                tide=tide, baroclinic=baroclinic)


def listed():
    return [
        # C1: a small closed basin in FP64, where launches and their gaps count; its run is 100 steps
        _dg("dg_c1_fp64", 16, 16, 4, 3, "fp64", 100),
        # a small odd-sized tidal basin at a low order with another barotropic flux: a quick-look run
        _dg("dg_small_hllc", 23, 17, 5, 2, "mixed", 50, flux="hllc", tide=True),
        # C2's physics on a quarter of its columns: a regional model
        _dg("dg_regional_mixed", 64, 64, 16, 4, "mixed", 40, tide=True),
        # C2 at full size, the headline run
        _dg("dg_c2_mixed", 128, 128, 16, 4, "mixed", 60, tide=True),
        # ragged sizes with the baroclinic pressure gradient on
        _dg("dg_baroclinic_mixed", 45, 38, 12, 4, "mixed", 15, baroclinic=True),
        # an FP64 run with every term on, as used to check a mixed-precision one
        _dg("dg_baroclinic_fp64", 48, 40, 16, 4, "fp64", 15, tide=True, baroclinic=True),
        # C5: uneven members stepped together
        dict(name="ens_c5_mixed", kind="ens", members=24, nmin=16, nmax=40, zmin=4, zmax=8, order=3,
             precision="mixed", steps=200),
        # C3 at full size: 256 x 256 base columns refined towards a coastline
        dict(name="amr_c3", kind="amr", nb=256, order=3, flux="lf", mode="complete", steps=100),
        # a small refined mesh at another order and flux
        dict(name="amr_small", kind="amr", nb=45, order=2, flux="upwind", mode="complete", steps=100),
        # C4 at full size with the cheapest preconditioner
        dict(name="bz_c4_jacobi", kind="bz", n=512, precond="jacobi"),
        # a smaller chart with the reference's own preconditioner
        dict(name="bz_mg", kind="bz", n=192, precond="mg"),
        # one training batch of the learned preconditioner
        dict(name="cnn_batch", kind="cnn", batch=16, crop=48),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["dg", "dg", "dg", "dg", "ens", "amr", "amr", "bz", "bz", "cnn"])
    if kind == "dg":
        order, prec = rng.randint(1, 5), rng.choice(["mixed", "mixed", "fp64"])
        nx, ny, nz = _log(rng, 8, 96), _log(rng, 8, 96), _log(rng, 2, 16)
        bar = rng.random() < 0.3
        # steps for a pass within the listed ones' cost
        nodes = nx * ny * nz * (order + 1) ** 3 * (2 if prec == "fp64" else 1) * (2 if bar else 1)
        steps = max(4, min(15 if bar else 60, int(3e8 / nodes)))
        return dict(kind="dg", nx=nx, ny=ny, nz=nz, order=order, precision=prec, steps=steps,
                    flux=rng.choice(["lf", "lf", "hllc", "roe"]), tide=rng.random() < 0.5, baroclinic=bar)
    if kind == "ens":
        nmin = _log(rng, 8, 16)
        return dict(kind="ens", members=rng.randint(3, 20), nmin=nmin, nmax=nmin + rng.randint(4, 22), zmin=2,
                    zmax=rng.randint(3, 8), order=rng.randint(2, 4), precision=rng.choice(["mixed", "mixed", "fp64"]),
                    steps=rng.randint(20, 50))
    if kind == "amr":
        order = rng.randint(1, 4)
        rhs = rng.random() < 0.2  # the reference's call has its own face set (no conforming faces)
        return dict(kind="amr", nb=_log(rng, 16, 256 if order < 4 else 128), order=order,
                    flux=rng.choice(["lf", "upwind", "central"]), mode="reference" if rhs else "complete",
                    steps=0 if rhs else rng.randint(10, 60))
    if kind == "bz":
        return dict(kind="bz", n=_log(rng, 8, 512), precond=rng.choice(["jacobi", "jacobi", "none"])) \
            if rng.random() < 0.7 else dict(kind="bz", n=2 ** rng.randint(3, 6) * rng.choice([3, 4, 5]), precond="mg")
    return dict(kind="cnn", batch=rng.randint(1, 16), crop=rng.randint(12, 64))


# ------------------------------------------------------------------------------------------ inputs
def _lgl(order):
    """LGL nodes, weights and differentiation matrix."""
    from numpy.polynomial import legendre as L
    P = L.Legendre.basis(order)
    x = np.concatenate([[-1.0], np.sort(P.deriv().roots().real), [1.0]]) if order > 1 else np.array([-1.0, 1.0])
    for _ in range(3):  # polish the roots of P'
        if order > 1:
            x[1:-1] -= P.deriv()(x[1:-1]) / P.deriv(2)(x[1:-1])
    w = 2.0 / (order * (order + 1) * P(x) ** 2)
    return x, w, _diff(x)


def _diff(x):
    c = np.array([np.prod([x[i] - x[k] for k in range(len(x)) if k != i]) for i in range(len(x))])
    D = np.array([[0.0 if i == j else c[i] / (c[j] * (x[i] - x[j])) for j in range(len(x))] for i in range(len(x))])
    return D - np.diag(D.sum(1))


def _lagrange(nodes, pts):
    """Lagrange basis on `nodes` at `pts`: [len(pts), len(nodes)]."""
    return np.array([[np.prod([(p - nodes[k]) / (nodes[j] - nodes[k]) for k in range(len(nodes)) if k != j])
                      for j in range(len(nodes))] for p in pts])


def _t(a):
    return torch.as_tensor(np.asarray(a), dtype=F64, device=DEV)


def _basin(nx, ny, nz, order, precision, flux, tide, baroclinic, seed):
    """A seeded basin: depth, wind, and a smooth moving, stratified initial state (device tensors [ny, nx, (nz,) k, j, i])."""
    rng = np.random.default_rng([seed, 11])
    el = 200e3 / 128 if nx * ny > 1024 else 100e3 / 16  # element size of C2 / C1
    Lx, Ly = nx * el, ny * el
    eos = {} if baroclinic else dict(alpha=0.0, beta=0.0)
    cfg = DGConfig(nx=nx, ny=ny, nz=nz, order=order, Lx=Lx, Ly=Ly, precision=precision, flux2d=flux,
                   bc=("tide" if tide else "wall", "wall", "wall", "wall"), tide_amp=1.0 if tide else 0.0,
                   Tref_s=configs.C2_T_SURFACE, Tref_dz=configs.C2_T_DZ, **eos)
    x = _t(_lgl(order)[0])
    ax = lambda n, d: ((torch.arange(n, dtype=F64, device=DEV)[:, None] + 0.5 * (x[None] + 1)) * d)  # noqa: E731
    X = ax(nx, el)[None, :, None, :]
    Y = ax(ny, el)[:, None, :, None]
    sg = -1 + ax(nz, 1.0 / nz)[None, None, :, :, None, None]
    # a gentle, slow shelf sea with the pressure gradient on (the sigma-coordinate error of steep flanks
    # grows in time), seamounts over a 500 m basin without it
    base, amp, wid, speed = (200.0, 40.0, 0.3, 0.02) if baroclinic else (500.0, 450.0, 0.1, 0.2)
    h = torch.full((ny, nx, order + 1, order + 1), base, dtype=F64, device=DEV)
    for _ in range(8):
        a, s = rng.uniform(0.2, 1.0) * amp / 2, rng.uniform(0.5, 1.0) * wid * min(Lx, Ly)
        h = h - a * torch.exp(-((X - rng.uniform(0, Lx)) ** 2 + (Y - rng.uniform(0, Ly)) ** 2) / (2 * s * s))
    h = h.clamp(min=50.0)
    k, ph = rng.uniform(0.6, 1.6, 6) * 2 * np.pi, rng.uniform(0, 2 * np.pi, 6)
    eta = 0.25 * speed * torch.sin(k[0] * X / Lx + ph[0]) * torch.cos(k[1] * Y / Ly + ph[1])
    H = (h + eta)[:, :, None, None]
    X3, Y3 = X[:, :, None, None], Y[:, :, None, None]
    u = speed * torch.sin(k[2] * X3 / Lx + ph[2]) * torch.cos(k[3] * Y3 / Ly + ph[3]) * (1 + 0.5 * sg)
    v = speed * torch.cos(k[4] * X3 / Lx + ph[4]) * torch.sin(k[5] * Y3 / Ly + ph[5]) * (1 + 0.3 * sg)
    front = torch.tanh(2 * torch.sin(k[0] * X3 / Lx + k[5] * Y3 / Ly))
    T = configs.C2_T_SURFACE + configs.C2_T_DZ * (eta[:, :, None, None] + sg * H) + 2.5 * speed * front * (1 + sg)
    S = 35.0 + 0.5 * speed * front * (1 + sg) + 0 * H
    q = [(f * H).contiguous() for f in (u, v, T, S)]
    tau, ang = rng.uniform(0.05, 0.15), rng.uniform(0, 2 * np.pi)
    f2 = torch.full_like(h, 1e-4)
    c = math.sqrt(cfg.g * float(h.max())) + 1.0
    dt = NSUB * 0.3 * el * 0.5 * float(x[1] - x[0]) / c
    return dict(cfg=cfg, h=h, f=f2, taux=torch.full_like(h, tau * math.cos(ang)),
                tauy=torch.full_like(h, tau * math.sin(ang)), q=q, eta=eta.contiguous(), dt=dt)


def _dg_basin(c, seed):
    return _basin(c["nx"], c["ny"], c["nz"], c["order"], c["precision"], c["flux"], c["tide"], c["baroclinic"], seed)


def _members(c, seed):
    """The members' meshes vary with the ensemble, not with the seed; bathymetry, wind and state do."""
    rng = np.random.default_rng(5)
    size = [[int(v) for v in (rng.integers(c["nmin"], c["nmax"] + 1), rng.integers(c["nmin"], c["nmax"] + 1),
                              rng.integers(c["zmin"], c["zmax"] + 1))] for _ in range(c["members"])]
    return [_basin(*s, c["order"], c["precision"], "lf", False, False, seed * 1000 + i) for i, s in enumerate(size)]


def _np(t):
    return t.reshape(-1).cpu().numpy()


def _host(b):
    return dict(cfg=b["cfg"], **{k: _np(b[k]) for k in ("h", "f", "taux", "tauy")})


def _amr_inputs(c, seed):
    """The configuration's own mesh (a seeded coastline); the field and its velocity vary with the seed."""
    i = configs.c3(c["nb"], c["order"])
    rng = np.random.default_rng([seed, 2])
    k, ph = rng.uniform(1, 4, 3), rng.uniform(0, 2 * np.pi, 3)
    lo, d = i["mesh"]["box"][:, :3], np.diff(i["mesh"]["box"].reshape(-1, 2, 3), axis=1)[:, 0]
    x = 0.5 * (_lgl(c["order"])[0] + 1)
    f = [np.sin(2 * np.pi * k[a] * (lo[:, a, None] + x * d[:, a, None]) + ph[a]) for a in range(3)]
    U = f[0][:, None, None, :] * f[1][:, None, :, None] * (1.5 + f[2])[:, :, None, None]
    return dict(order=c["order"], mesh=i["mesh"], U=np.ascontiguousarray(U.reshape(len(U), -1)),
                a=rng.uniform(0.2, 1.0, 3) * rng.choice([-1.0, 1.0], 3))


def _bz_inputs(c, seed):
    n = c["n"]
    return configs.c4(n=n, L=100.0 * n, seed=seed % (1 << 30))


def _cnn_inputs(c, seed):
    rng = np.random.default_rng([seed, 3])
    X, T = (np.zeros((c["batch"], c["crop"], c["crop"], 16)) for _ in range(2))
    X[..., :9], T[..., :9] = rng.standard_normal((2, c["batch"], c["crop"], c["crop"], 9))
    # weights [co][tap][ci] and bias per layer, at their usual scale
    w = [(rng.standard_normal(9 * i * o) * math.sqrt(2 / (9 * i)), 0.1 * rng.standard_normal(o)) for i, o in zip(CH, CH[1:])]
    return X, T, np.concatenate([a for l in w for a in l])


# ------------------------------------------------------------------------------------------ prepare and run
FIELDS = ("Hu", "Hv", "HT", "HS", "eta", "HU", "HV")


def _dg_sizes(cfg):
    return [cfg.n3] * 4 + [cfg.n2] * 3


def prepare(case, seed):
    c = case
    if c["kind"] == "dg":
        b = _dg_basin(c, seed)
        cfg = b["cfg"]
        m = OceanModel(**_host(b))
        m.upload_state([_np(a) for a in b["q"]], _np(b["eta"]))
        # pinned output buffers, kept over the run
        out = {k: torch.empty(n, dtype=F64, pin_memory=True) for k, n in zip(FIELDS, _dg_sizes(cfg))}
        s = dict(case=c, model=m, dt=b["dt"], out=out, view={k: v.numpy() for k, v in out.items()})
        if cfg.precision == "mixed":
            s["file"] = {k: torch.empty(v.numel(), dtype=torch.float32) for k, v in out.items()}
        return s
    if c["kind"] == "ens":
        bs = _members(c, seed)
        e = Ensemble([_host(b) for b in bs])
        for m, b in zip(e.members, bs):
            m.upload_state([_np(a) for a in b["q"]], _np(b["eta"]))
        dtype = torch.float32 if c["precision"] == "mixed" else F64
        tot = np.sum([_dg_sizes(b["cfg"]) for b in bs], axis=0)
        return dict(case=c, ens=e, dts=[b["dt"] for b in bs],
                    file={k: torch.empty(int(n), dtype=dtype) for k, n in zip(FIELDS, tot)})
    if c["kind"] == "amr":
        i = _amr_inputs(c, seed)
        m = DG3DIntegration(i["order"], i["mesh"])
        m.upload(i["U"])
        return dict(case=c, model=m, a=i["a"], dt=AMR_DT, U=i["U"])
    if c["kind"] == "bz":
        i = _bz_inputs(c, seed)
        s = BezierSmoother(i["n"], i["n"], i["L"], i["L"], i["d"], lam=i["lam"], ridge_epsilon=i["eps"])
        if c["precond"] == "mg":
            s.mg_setup()
        return dict(case=c, smoother=s)
    X, T, w = _cnn_inputs(c, seed)
    net = CNN()
    net.set_params(w)
    return dict(case=c, net=net, X=X, T=T)


def run(state):
    c = state["case"]
    if c["kind"] == "dg":
        m = state["model"]
        m.step(state["dt"], NSUB, c["steps"])
        m.output_stage(state["view"])
        m.output_wait()
        if "file" not in state:
            return state["out"]
        for k, v in state["file"].items():
            v.copy_(state["out"][k])
        return state["file"]
    if c["kind"] == "ens":
        state["ens"].step(state["dts"], NSUB, c["steps"])
        at = dict.fromkeys(FIELDS, 0)
        for m in state["ens"].members:
            d = m.download_state()
            for k in FIELDS:
                state["file"][k][at[k]:at[k] + d[k].size].copy_(torch.from_numpy(d[k]))
                at[k] += d[k].size
        return state["file"]
    if c["kind"] == "amr":
        m = state["model"]
        if c["steps"] == 0:
            return m.compute_rhs(state["U"], state["a"], flux=c["flux"], mode=c["mode"])
        m.step(state["a"], state["dt"], c["steps"], flux=c["flux"], mode=c["mode"])
        return m.download()
    if c["kind"] == "bz":
        return state["smoother"].solve(c["precond"], tol=1e-10, maxit=5000)[0]
    Y, grad, loss = state["net"].forward_backward(state["X"], state["T"])
    return dict(Y=Y, grad=grad, loss=loss)


# ------------------------------------------------------------------------------------------ work
def _dg_work(cfg, steps):
    s, np1 = (4 if cfg.precision == "mixed" else 8), cfg.order + 1
    bar = cfg.alpha != 0 or cfg.beta != 0
    # per stage: the 4 variables and their register read and written (no register read in the first stage), the 2D
    # fields once; per barotropic pass: state and forcing read, state written, in FP64
    bytes_ = steps * (cfg.n3 * s * (5 * 16 - 4) + cfg.n2 * 8 * (5 * 9 + 2 * NSUB * 8))
    # per stage and node: 4 variables' advection in 3 directions, second derivatives (2 + 2 horizontal, 4 vertical),
    # divergence and omega, 2 flops per term
    flops = steps * (5 * cfg.n3 * (2 * np1 * (12 + 8 + 3 + (5 if bar else 0)) + 60) + 2 * NSUB * cfg.n2 * (16 * np1 + 60))
    return bytes_, flops


def _mesh_size(c):
    lx, ly, lz = (np.asarray(a) for a in configs.c3_levels(c["nb"]))
    return int((2 ** (lx + ly + lz)).sum())  # of the configuration's own coastline


def work(case):
    c = case
    if c["kind"] == "dg":
        b, f = _dg_work(DGConfig(c["nx"], c["ny"], c["nz"], c["order"], 1.0, 1.0, precision=c["precision"],
                                 **({} if c["baroclinic"] else dict(alpha=0.0, beta=0.0))), c["steps"])
        out = 8 * (4 * c["nx"] * c["ny"] * c["nz"] * (c["order"] + 1) ** 3)
        return dict(bytes=b + out, flops=f)
    if c["kind"] == "ens":
        rng, b, f = np.random.default_rng(5), 0.0, 0.0
        for _ in range(c["members"]):
            nx, ny, nz = (int(v) for v in (rng.integers(c["nmin"], c["nmax"] + 1), rng.integers(c["nmin"], c["nmax"] + 1),
                                           rng.integers(c["zmin"], c["zmax"] + 1)))
            x, y = _dg_work(DGConfig(nx, ny, nz, c["order"], 1.0, 1.0, precision=c["precision"], alpha=0.0, beta=0.0),
                            c["steps"])
            b, f = b + x + 32 * nx * ny * nz * (c["order"] + 1) ** 3, f + y
        return dict(bytes=b, flops=f)
    if c["kind"] == "amr":
        p, ne = c["order"] + 1, _mesh_size(c)
        # per stage: state and register in and out; 7 one-dimensional products and the faces
        if c["steps"] == 0:
            return dict(bytes=16.0 * ne * p ** 3, flops=1.0 * ne * p ** 3 * (14 * p + 30))
        return dict(bytes=8.0 * ne * p ** 3 * (c["steps"] * 19 + 1), flops=5.0 * c["steps"] * ne * p ** 3 * (14 * p + 30))
    if c["kind"] == "bz":
        nd = 3 * c["n"] + 1
        it = {"none": 49, "jacobi": 30, "mg": 6}[c["precond"]]  # iterations at C4
        # an iteration's own vectors, each once: q = Q p, x, r and p updated; a V-cycle reads and writes about
        # 30 vectors' worth over its levels
        return dict(bytes=8.0 * nd * nd * it * (11 + (30 if c["precond"] == "mg" else 0)),
                    flops=1.0 * nd * nd * it * (70 + (700 if c["precond"] == "mg" else 0)))
    px = c["batch"] * c["crop"] ** 2
    macs = 9 * (16 * 32 + 32 * 32 + 32 * 32 + 32 * 16)
    return dict(bytes=8.0 * px * 16 * 3, flops=6.0 * px * macs)


# ------------------------------------------------------------------------------------------ exact: the DG model
def _sw(U, nx, ny, g):
    h, hu, hv = U
    u, v = hu / h, hv / h
    un = u * nx + v * ny
    return torch.stack([h * un, h * u * un + 0.5 * g * h * h * nx, h * v * un + 0.5 * g * h * h * ny])


def _flux2d(kind, L, R, nx, ny, g):
    """The shallow-water face flux F*(L, R, n): Lax-Friedrichs, HLLC (Einfeldt speeds) or Roe (Harten fix 0.1)."""
    FL, FR = _sw(L, nx, ny, g), _sw(R, nx, ny, g)
    hL, hR = L[0], R[0]
    uL, vL, uR, vR = L[1] / hL, L[2] / hL, R[1] / hR, R[2] / hR
    nL, nR = uL * nx + vL * ny, uR * nx + vR * ny
    cL, cR = torch.sqrt(g * hL), torch.sqrt(g * hR)
    if kind == "lf":
        return 0.5 * (FL + FR) - 0.5 * torch.maximum(nL.abs() + cL, nR.abs() + cR) * (R - L)
    if kind == "hllc":
        SL, SR = torch.minimum(nL - cL, nR - cR), torch.maximum(nL + cL, nR + cR)
        den = hL * (SL - nL) - hR * (SR - nR)
        ok = den.abs() > 1e-10
        Ss = torch.where(ok, (hL * nL * (SL - nL) - hR * nR * (SR - nR) + 0.5 * g * (hR * hR - hL * hL))
                         / torch.where(ok, den, torch.ones_like(den)), 0.5 * (nL + nR))

        def star(U, u, v, n, S, F):
            hs = U[0] * (S - n) / (S - Ss)
            return F + S * (torch.stack([hs, hs * (u + (Ss - n) * nx), hs * (v + (Ss - n) * ny)]) - U)
        F = torch.where(Ss >= 0, star(L, uL, vL, nL, SL, FL), star(R, uR, vR, nR, SR, FR))
        return torch.where(SL >= 0, FL, torch.where(SR <= 0, FR, F))
    sL, sR = torch.sqrt(hL), torch.sqrt(hR)
    hr, ur, vr = 0.5 * (hL + hR), (sL * uL + sR * uR) / (sL + sR), (sL * vL + sR * vR) / (sL + sR)
    un, cr = ur * nx + vr * ny, torch.sqrt(g * hr)
    d = 0.1 * cr
    fix = lambda l: torch.where(l.abs() < d, (l * l + d * d) / (2 * d), l.abs())  # noqa: E731
    dh, dn, dt = hR - hL, nR - nL, (vR * nx - uR * ny) - (vL * nx - uL * ny)
    a1, a2, a3 = fix(un - cr) * 0.5 * (dh - hr / cr * dn), un.abs() * hr * dt, fix(un + cr) * 0.5 * (dh + hr / cr * dn)
    return 0.5 * (FL + FR) - 0.5 * torch.stack([a1 + a3, a1 * (ur - cr * nx) - a2 * ny + a3 * (ur + cr * nx),
                                                a1 * (vr - cr * ny) + a2 * nx + a3 * (vr + cr * ny)])


class _Exact:
    """The coupled scheme in 64 bits: strong-form DGSEM on LGL nodes, tensors [ny, nx, (nz, k,) j, i]."""

    def __init__(self, b):
        cfg = self.cfg = b["cfg"]
        x, w, D = _lgl(cfg.order)
        self.N, self.nz = cfg.order, cfg.nz
        self.x, self.w, self.D = _t(x), _t(w), _t(D)
        dx, dy, self.ds = cfg.Lx / cfg.nx, cfg.Ly / cfg.ny, 1.0 / cfg.nz
        self.c = (2 / dx, 2 / dy, 2 / self.ds)
        self.L = tuple(v / float(w[0]) for v in self.c)
        E = D.copy()
        E[0, 0] += 1 / w[0]
        Ai = np.linalg.inv(E)
        self.Ai, self.a0 = _t(Ai), _t(Ai[:, 0] / w[0])
        g, gw = np.polynomial.legendre.leggauss(cfg.order + 2)  # S[k][m] = int_{-1}^{x_k} l_m
        self.S = _t(np.stack([0.5 * (v + 1) * gw @ _lagrange(x, -1 + 0.5 * (v + 1) * (g + 1)) for v in x]))
        self.h, self.f, self.tx, self.ty = b["h"], b["f"], b["taux"], b["tauy"]
        self.sg = (-1 + self.ds * (torch.arange(cfg.nz, dtype=F64, device=DEV)[:, None] + 0.5 * (self.x + 1)))[:, :, None, None]
        self.bar = cfg.alpha != 0 or cfg.beta != 0
        self.Q, self.eta, self.t = torch.stack(b["q"]), b["eta"].clone(), 0.0
        self.HU, self.HV = self.colint(self.Q[0]), self.colint(self.Q[1])
        self.eta_avg = self.eta

    def d(self, a, axis):  # derivative along 0 x, 1 y, 2 sigma
        if axis == 0:
            return torch.matmul(a, self.D.T)
        if axis == 1:
            return torch.matmul(self.D, a)
        return torch.matmul(self.D, a.flatten(-2)).reshape(a.shape)

    def colint(self, a):
        return 0.5 * self.ds * torch.einsum("yxzkji,k->yxji", a, self.w)

    def tide(self, t):
        return self.cfg.tide_amp * math.sin(2 * math.pi * t / self.cfg.tide_period)

    def outside(self, a, side, wall):
        """Values across a face: the neighbour column's opposite face line, `wall` at the basin's side.
        a: [..., ny, nx, <rest>, j, i] with ny at axis `y`."""
        lo, hi, y = a  # the fields' own low and high face lines, and the y axis
        n = lo.shape[y] if side >= 2 else lo.shape[y + 1]
        ax = y if side >= 2 else y + 1
        if side % 2 == 0:
            return torch.cat([wall.narrow(ax, 0, 1), hi.narrow(ax, 0, n - 1)], ax)
        return torch.cat([lo.narrow(ax, 1, n - 1), wall.narrow(ax, n - 1, 1)], ax)

    def line(self, a, side):  # the face line of side 0 W, 1 E, 2 S, 3 N
        i = self.N if side % 2 else 0
        return a[..., i] if side < 2 else a[..., i, :]

    def across(self, a, side, wall, y):
        s0 = side - side % 2
        return self.outside((self.line(a, s0), self.line(a, s0 + 1), y), side, wall)

    def add(self, r, side, v):
        self.line(r, side).sub_(v)

    def rhs3(self, Q, etab):
        cfg, c, L, D = self.cfg, self.c, self.L, self.d
        g, eta = cfg.g, self.eta
        up = lambda a: a[:, :, None, None]  # noqa: E731
        H2 = eta + self.h
        H, iH = up(H2), 1 / up(H2)
        et = self.tide(self.t)
        face = []
        for s in range(4):
            qm, em, hm = self.line(Q, s), self.line(eta, s), self.line(self.h, s)
            if cfg.bc[s] == "tide":
                ew, Hw = torch.full_like(em, et), et + hm
                qw = qm * (Hw / (em + hm))[:, :, None, None]
            else:
                ew, Hw, qw = em, em + hm, qm.clone()
                qw[s // 2] *= -1
            face.append((qm, self.across(Q, s, qw, 1), em, self.across(eta, s, ew, 0), em + hm,
                         self.across(H2, s, Hw, 0), Hw))
        de = c[0] * D(Q[0], 0) + c[1] * D(Q[1], 1)
        for s in range(4):
            qm, qp = face[s][:2]
            self.add(de, s, -L[s // 2] * (1 if s % 2 else -1) * 0.5 * (qp - qm)[s // 2])
        lay = 0.5 * self.ds * torch.einsum("yxzkji,k->yxzji", de, self.w)
        I = lay.sum(2)
        om, Mf, ys = torch.empty_like(de), [], torch.zeros_like(I)
        for z in range(self.nz):
            Mf.append(ys)
            gz = I[:, :, None] - de[:, :, z]
            om[:, :, z] = 0.5 * self.ds * torch.einsum("km,yxmji->yxkji", self.Ai, gz) \
                + self.a0[:, None, None] * ys[:, :, None]
            ys = ys + self.ds * I - lay[:, :, z]
        Mf = torch.stack(Mf + [torch.zeros_like(ys)], 2)
        om = om * iH
        vel = Q[:2] * iH
        r = -(c[0] * D(Q * vel[0], 0) + c[1] * D(Q * vel[1], 1) + c[2] * D(Q * om, 2))
        r[0] += up(self.f) * Q[1] - g * H * c[0] * up(D(eta, 0))
        r[1] += -up(self.f) * Q[0] - g * H * c[1] * up(D(eta, 1))
        if self.bar:
            Hb2 = etab + self.h
            Hb = up(Hb2)
            anom = cfg.beta * (Q[3] / Hb - cfg.S0) - cfg.alpha * (
                Q[2] / Hb - (cfg.Tref_s + cfg.Tref_dz * (up(etab) + self.sg * Hb)))
            J = 0.5 * self.ds * torch.einsum("km,yxzmji->yxzkji", self.S, anom)
            T = J[:, :, :, -1]
            below = torch.cumsum(T, 2) - T
            B = T.sum(2)[:, :, None, None] - below[:, :, :, None] - J
            P = Hb * Hb * B
            for a in (0, 1):
                slope = up(c[a] * D(etab, a)) + self.sg * up(c[a] * D(Hb2, a))
                r[a] -= g * (c[a] * D(P, a) - c[2] * D(Hb * B * slope, 2))
        r[:2] += cfg.nu_h * H * (c[0] ** 2 * D(D(vel, 0), 0) + c[1] ** 2 * D(D(vel, 1), 1))
        for v, k in enumerate((cfg.nu_v, cfg.nu_v, cfg.kappa_v_T, cfg.kappa_v_S)):
            r[v] += k * iH * c[2] ** 2 * D(D(Q[v] * iH, 2), 2)
        for s in range(4):
            qm, qp, em, ep, Hm, Hp, Hw = face[s]
            a, n, u2 = s // 2, (1 if s % 2 else -1), (lambda b: b[:, :, None, None])
            um, unp = qm[a] * n / u2(Hm), qp[a] * n / u2(Hp)
            lam = torch.maximum(um.abs(), unp.abs())
            self.add(r, s, L[a] * (0.5 * (qm * um + qp * unp) - 0.5 * lam * (qp - qm) - qm * um))
            pj = u2(g * Hm * 0.5 * (ep - em)).expand_as(um)
            if self.bar:
                Pm = self.line(P, s)
                Pw = u2(Hw * Hw) * self.line(B, s) if cfg.bc[s] == "tide" else Pm
                pj = pj + g * 0.5 * (self.across(P, s, Pw, 0) - Pm)
            self.add(r[a], s, L[a] * n * pj)
        N, iHz = self.N, iH[:, :, 0]
        for k, n in ((0, -1), (N, 1)):
            M = Mf[:, :, :-1] if k == 0 else Mf[:, :, 1:]
            qm, wm = Q[:, :, :, :, k], om[:, :, :, k] * n
            if k == 0:
                nb = torch.cat([qm[:, :, :, :1], Q[:, :, :, :-1, N]], 3)
                qu = torch.where(M > 0, nb, qm)
            else:
                nb = torch.cat([Q[:, :, :, 1:, 0], qm[:, :, :, -1:]], 3)
                qu = torch.where(M > 0, qm, nb)
            r[:, :, :, :, k] -= L[2] * (n * M * qu * iHz[None] - qm * wm)
        ub = vel[:, :, :, 0, 0]
        r[:2, :, :, 0, 0] -= L[2] * cfg.cd * torch.sqrt(ub[0] ** 2 + ub[1] ** 2) * ub
        r[0, :, :, -1, N] += L[2] * self.tx / cfg.rho0
        r[1, :, :, -1, N] += L[2] * self.ty / cfg.rho0
        return r, -I

    def rhs2(self, e, u, v, Fx, Fy, time):
        cfg, c, L, D, g = self.cfg, self.c, self.L, self.d, self.cfg.g
        H = e + self.h
        k = torch.stack([-(c[0] * D(u, 0) + c[1] * D(v, 1)),
                         -(c[0] * D(u * u / H, 0) + c[1] * D(u * v / H, 1)) - g * H * c[0] * D(e, 0) + self.f * v + Fx,
                         -(c[0] * D(u * v / H, 0) + c[1] * D(v * v / H, 1)) - g * H * c[1] * D(e, 1) - self.f * u + Fy])
        U, et = torch.stack([H, u, v]), self.tide(time)
        for s in range(4):
            Um = self.line(U, s)
            W = Um.clone()
            if cfg.bc[s] == "tide":
                W[0] = et + self.line(self.h, s)
                W[1:] *= W[0] / Um[0]
            else:
                W[1 + s // 2] *= -1
            nx, ny = ((-1, 0), (1, 0), (0, -1), (0, 1))[s]
            Up = self.across(U, s, W, 1)
            self.add(k, s, L[s // 2] * (_flux2d(cfg.flux2d, Um, Up, nx, ny, g) - _sw(Um, nx, ny, g)))
        return k

    def step(self, dt):
        res, rese, etas, dHU, dHV = 0.0, 0.0, self.eta, 0.0, 0.0
        Q = self.Q
        for a, b in zip(LSRK_A, LSRK_B):
            r, de = self.rhs3(Q, etas)
            res = a * res + dt * r
            Q = Q + b * res
            rese = a * rese + dt * de
            etas = etas + b * rese
            dHU, dHV = dHU + b * self.colint(res[0]), dHV + b * self.colint(res[1])
        e, u, v = self.eta, self.HU, self.HV
        k = self.rhs2(e, u, v, 0.0, 0.0, self.t)
        Fx, Fy = dHU / dt - k[1], dHV / dt - k[2]
        tb = dt / NSUB
        for m in range(NSUB):
            k1 = self.rhs2(e, u, v, Fx, Fy, self.t + m * tb)
            k2 = self.rhs2(e + tb * k1[0], u + tb * k1[1], v + tb * k1[2], Fx, Fy, self.t + m * tb + tb)
            s = 0.5 * tb * (k1 + k2)
            e, u, v = e + s[0], u + s[1], v + s[2]
        up = lambda a: a[:, :, None, None]  # noqa: E731
        Q[0] += up(u - (self.HU + dHU))
        Q[1] += up(v - (self.HV + dHV))
        Q[2:] *= up((e + self.h) / (etas + self.h))
        self.Q, self.eta, self.HU, self.HV, self.t = Q, e, u, v, self.t + dt

    def run(self, dt, steps):
        for _ in range(steps):
            self.step(dt)
        return dict(zip(FIELDS, [q.reshape(-1) for q in self.Q] + [a.reshape(-1) for a in (self.eta, self.HU, self.HV)]))


# ------------------------------------------------------------------------------------------ exact: AMR, Bezier, network
SUB = {1: ((-1, -1, 0, 1), (0, -1, 1, 1)), 2: ((-1, -1, 1, 0), (-1, 0, 1, 1)),
       5: ((-1, -1, 0, 0), (0, -1, 1, 0), (-1, 0, 0, 1), (0, 0, 1, 1))}  # sub-faces (t1 lo, t2 lo, t1 hi, t2 hi) by type


def _mortar_P(order, box):
    """Projection of a fine face's trace onto the mortar space (nodes of the coarse face): M^-1 B, B summed over the
    quadrature points inside the closed sub-face."""
    x = _lgl(order)[0]
    g, gw = np.polynomial.legendre.leggauss(2 * order + 1)
    g[order] = 0.0
    phi = _lagrange(x, g)
    P = []
    for lo, hi in ((box[0], box[2]), (box[1], box[3])):
        on = (g >= lo) & (g <= hi)
        B = (phi[on] * gw[on, None]).T @ _lagrange(x, 2 * (g[on] - lo) / (hi - lo) - 1)
        P.append(np.linalg.solve((phi * gw[:, None]).T @ phi, B))
    return _t(np.kron(P[1], P[0]))  # face node (it, jt) at it + np jt


def _exact_amr(c, seed):
    i = _amr_inputs(c, seed)
    mesh, order, a, dt = i["mesh"], i["order"], i["a"], AMR_DT
    p = order + 1
    x, w, D = _lgl(order)
    g, gw = np.polynomial.legendre.leggauss(order)
    B = _lagrange(x, g)
    K, M = _t((B @ D).T @ (gw[:, None] * B)), _t(B.T @ (gw[:, None] * B))
    w = _t(w)
    vi = np.arange(p ** 3).reshape(p, p, p)  # [k][j][i]
    side = [vi[:, :, 0], vi[:, :, -1], vi[:, 0], vi[:, -1], vi[0], vi[-1]]  # face nodes [jt][it]
    nodes = torch.as_tensor(np.stack([s.reshape(-1) for s in side]), device=DEV)
    wf = (w[:, None] * w[None]).reshape(-1)
    iM = 1 / (w[:, None, None] * w[None, :, None] * w[None, None]).reshape(-1)

    def flux(uL, uR, vn):
        if c["flux"] == "central":
            return 0.5 * vn * (uL + uR)
        if c["flux"] == "upwind":
            return torch.where(vn >= 0, vn * uL, vn * uR)
        return 0.5 * vn * (uL + uR) - 0.5 * vn.abs() * (uR - uL)
    vn_of = _t([s * a[f // 2] for f, s in enumerate((-1, 1) * 3)])
    faces = []
    if c["mode"] == "complete":
        cf, bd = torch.as_tensor(mesh["conf"], device=DEV), torch.as_tensor(mesh["bnd"], device=DEV)
        faces = [(cf[:, 0], cf[:, 1], cf[:, 2], cf[:, 3]), (cf[:, 2], cf[:, 3], cf[:, 0], cf[:, 1]),
                 (bd[:, 0], bd[:, 1], bd[:, 0], bd[:, 1])]
        faces = [(e[:, None] * p ** 3 + nodes[f], vn_of[f][:, None], e2[:, None] * p ** 3 + nodes[f2])
                 for e, f, e2, f2 in faces]
    ty, ce, cfc, fe, ff = (torch.as_tensor(v, device=DEV).long() for v in mesh["if_arrays"])
    mort = []
    for t, boxes in SUB.items():
        on = (ty == t).nonzero()[:, 0]
        if len(on):
            mort.append((ce[on][:, None] * p ** 3 + nodes[cfc[on]], vn_of[cfc[on]][:, None],
                         [(fe[on, k][:, None] * p ** 3 + nodes[ff[on, k]], _mortar_P(order, b)) for k, b in enumerate(boxes)]))
    def rhs(U):
        q = U.reshape(-1, p, p, p)
        ez = lambda A, v: torch.matmul(A, v.flatten(-2)).reshape(v.shape)  # noqa: E731
        Pz, Qz = ez(M, q), ez(K, q)
        r = -(a[0] * torch.matmul(torch.matmul(M, Pz), K.T)
              + torch.matmul(a[1] * torch.matmul(K, Pz) + a[2] * torch.matmul(M, Qz), M.T)).reshape(-1)
        Uf = U.reshape(-1)
        for at, vn, nb in faces:
            r.index_add_(0, at.reshape(-1), (wf * flux(Uf[at], Uf[nb], vn)).reshape(-1))
        for at, vn, fine in mort:  # lifts B^T M^-1 F with P = M^-1 B: F itself on the coarse side, P^T F on a fine one
            F = flux(Uf[at], sum(Uf[f] @ P.T for f, P in fine), vn)
            r.index_add_(0, at.reshape(-1), F.reshape(-1))
            for f, P in fine:
                r.index_add_(0, f.reshape(-1), -(F @ P).reshape(-1))
        return (r.reshape(-1, p ** 3) * iM).reshape(U.shape)
    U, res = _t(i["U"]), 0.0
    if c["steps"] == 0:
        return rhs(U)
    for _ in range(c["steps"]):
        for A, Bc in zip(LSRK_A, LSRK_B):
            res = A * res - dt * rhs(U)
            U = U + Bc * res
    return U


def _bernstein(t, d):
    s = 1 - t
    return np.array([[s ** 3, 3 * t * s * s, 3 * t * t * s, t ** 3],
                     [-3 * s * s, 3 * s * s - 6 * t * s, 6 * t * s - 3 * t * t, 3 * t * t],
                     [6 * s, 6 * t - 12 * s, 6 * s - 12 * t, 6 * t]][d])


def _exact_bz(c, seed):
    i = _bz_inputs(c, seed)
    n, dx, lam, eps = i["n"], i["L"] / i["n"], i["lam"], i["eps"]
    nd = 3 * n + 1
    g, gw = np.polynomial.legendre.leggauss(4)
    g, gw = 0.5 * (g + 1), 0.25 * gw  # the smoother's data weights sum to 1/4 an element
    b0, b1, b2 = (np.stack([_bernstein(t, d) for t in g]) for d in range(3))  # [q][i]
    k2 = lambda v, u: np.einsum("yj,xi->yxji", v, u).reshape(16, 16)  # noqa: E731  [q][dof], both x fastest
    W = np.diag(np.outer(gw, gw).reshape(-1))
    uu, vv, uv, ph = k2(b0, b2), k2(b2, b0), k2(b1, b1), k2(b0, b0)
    H = (uu.T @ W @ uu + vv.T @ W @ vv + uu.T @ W @ vv + vv.T @ W @ uu + 2 * uv.T @ W @ uv) / dx ** 2
    Bm = dx * dx * ph.T @ W @ ph

    def fro2(A):  # squared Frobenius norm of the assembled matrix, from its rows' 7 x 7 stencils
        A = A.reshape(4, 4, 4, 4)  # [aj][ai][bj][bi]
        tot = 0.0
        for rj, cj in ((0, 2), (1, n), (2, n), (3, n - 1)):  # boundary, two inner, shared rows along y
            for ri, ci in ((0, 2), (1, n), (2, n), (3, n - 1)):
                row = np.zeros((7, 7))
                for aj in ((0, 3) if rj == 3 else (rj,)):
                    for ai in ((0, 3) if ri == 3 else (ri,)):
                        row[3 - aj:7 - aj, 3 - ai:7 - ai] += A[aj, ai]
                tot += cj * ci * (row ** 2).sum()
        return tot
    alpha = math.sqrt(fro2(Bm) / fro2(H))
    Kt = _t(alpha * H + lam * Bm)
    cut = [(slice(j, j + 3 * n, 3), slice(k, k + 3 * n, 3)) for j in range(4) for k in range(4)]

    def scatter(e):  # [16, n, n] element values summed into the control points
        y = torch.zeros(nd, nd, dtype=F64, device=DEV)
        for k, at in enumerate(cut):
            y[at] += e[k]
        return y

    def Q(x):
        return scatter(torch.einsum("ab,byx->ayx", Kt, torch.stack([x[at] for at in cut]))) + lam * eps * x
    d = _t(i["d"]).reshape(n, n, 16).permute(2, 0, 1)
    b = scatter(torch.einsum("ab,byx->ayx", _t(lam * dx * dx * ph.T @ W), d))
    diag = scatter(torch.diagonal(Kt)[:, None, None].expand(16, n, n)) + lam * eps
    x = torch.zeros_like(b)
    r, z = b.clone(), b / diag
    q, rz = z.clone(), (b * b / diag).sum()
    for _ in range(400):
        Aq = Q(q)
        al = rz / (q * Aq).sum()
        x, r = x + al * q, r - al * Aq
        if float((r * r).sum()) <= 1e-30 * float((b * b).sum()):
            break
        z = r / diag
        new = (r * z).sum()
        q, rz = z + new / rz * q, new
    return x.reshape(-1)


def _exact_cnn(c, seed):
    X, T, flat = _cnn_inputs(c, seed)
    flat, ch, at, ps = _t(flat), CH, 0, []
    for l in range(4):
        n = ch[l + 1] * 9 * ch[l]
        ps += [flat[at:at + n].clone().requires_grad_(), flat[at + n:at + n + ch[l + 1]].clone().requires_grad_()]
        at += n + ch[l + 1]
    y = _t(X).permute(0, 3, 1, 2)
    for l in range(4):
        W = ps[2 * l].reshape(ch[l + 1], 3, 3, ch[l]).permute(0, 3, 1, 2)
        y = torch.nn.functional.conv2d(y, W, ps[2 * l + 1], padding=1)
        y = y.relu() if l < 3 else y
    Y = y.permute(0, 2, 3, 1)
    loss = ((Y - _t(T))[..., :9] ** 2).mean()
    loss.backward()
    return dict(Y=Y.detach(), grad=torch.cat([p.grad for p in ps]), loss=float(loss.detach()))


def exact(case, seed):
    c = case
    if c["kind"] == "dg":
        n3 = c["nx"] * c["ny"] * c["nz"] * (c["order"] + 1) ** 3
        if c["steps"] * (0.06 + n3 * 1e-8) > 18:  # seconds, about
            return None
        b = _dg_basin(c, seed)
        return _Exact(b).run(b["dt"], c["steps"])
    if c["kind"] == "ens":
        if c["steps"] * c["members"] * 0.06 > 18:
            return None
        bs = _members(c, seed)
        outs = [_Exact(b).run(b["dt"], c["steps"]) for b in bs]
        return {k: torch.cat([o[k] for o in outs]) for k in FIELDS}
    if c["kind"] == "amr":
        return None if c["steps"] * _mesh_size(c) * (c["order"] + 1) ** 3 > 6e8 else _exact_amr(c, seed)
    if c["kind"] == "bz":
        return _exact_bz(c, seed)
    return _exact_cnn(c, seed)
