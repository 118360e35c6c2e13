"""Workloads that stand for the use of this framework, each one pass through the public API.

A pass is what a solver run does with the device: the state goes up from pinned host memory, steps
are taken with the diagnostics in between, and the state comes back (`Solver`, `Ensemble`); or one
right-hand side, or one gradient of the time-integrated dissipation (`Solver.adjoint`), or one
right-hand side on the caller's own device arrays (`dsem_rhs_noalloc`).  Meshes are periodic boxes
of [0, 2 pi]^3 (Taylor-Green and isotropic flow), curved ones, ones with walls, and ones whose
elements have two orders; orders p = 1..8, every viscosity model.

`exact` evaluates the same discretisation (Chebyshev Gauss and Lobatto points, Roe fluxes, averaged
viscous fluxes, low-storage Runge-Kutta) with torch on whole-mesh arrays, for straight periodic
boxes of one order without a turbulence model; gradients by torch's reverse mode.
"""
import ctypes
import functools
import math
from types import SimpleNamespace

import numpy as np
import torch
from torch.utils.checkpoint import checkpoint

from dsem_b200 import mesh
from dsem_b200.solver import Ensemble, Solver, lib

GAMMA, PR, TWALL = 1.4, 0.72, 100.0
ARK = {3: (0.0, -5.0 / 9.0, -153.0 / 128.0), 4: (0.0, -0.4178904745, -1.192151694643, -1.697784692471, -1.514183444257)}
CRK = {3: (1.0 / 3.0, 15.0 / 16.0, 8.0 / 15.0),
       4: (0.1496590219993, 0.3792103129999, 0.8229550293869, 0.6994504559488, 0.1530572479681)}


def listed():
    def run(name, nx, ny, nz, p, blocks, steps, shape="box", model="none", iord=4, re=1600.0):
        return dict(name=name, kind="run", nx=nx, ny=ny, nz=nz, p=p, blocks=blocks, steps=steps, shape=shape,
                    model=model, iord=iord, re=re)

    return [
        # the smallest call: one step of the 4^3, p = 4 Taylor-Green case with its diagnostics, all latency
        run("step_4_p4", 4, 4, 4, 4, 1, 1),
        # the reference-scale Taylor-Green run, 22^3 elements at p = 8
        run("tgv_22_p8", 22, 22, 22, 8, 2, 20),
        # 12^3 at p = 6, the size of the gradient case's forward run
        run("tgv_12_p6", 12, 12, 12, 6, 4, 10),
        # many small elements
        run("tgv_20_p4", 20, 20, 20, 4, 2, 20),
        # an uneven box at an odd order with the Smagorinsky model and three-stage stepping
        run("les_11x7x9_p7", 11, 7, 9, 7, 2, 10, model="les", iord=3),
        # isotropic flow with entropy viscosity across a band of higher order (mortar projections)
        run("ev_band_10_p6_p8", 10, 10, 10, 6, 2, 5, shape="band", model="ev", re=115.0),
        # curved elements: the general-metric path
        run("curved_8_p8", 8, 8, 8, 8, 2, 10, shape="curved"),
        # walls in y, a channel
        run("walls_10x8x6_p5", 10, 8, 6, 5, 2, 10, shape="walls", re=500.0),
        # independent cases of several sizes and orders advanced together
        dict(name="ensemble_12", kind="ensemble", cases=12, pick=1, blocks=1, steps=20),
        # the gradient with every stage kept
        dict(name="adjoint_8_p6", kind="adjoint", nx=8, ny=8, nz=8, p=6, steps=30, window=10, snapshots=0,
             scheme="revolve", re=1600.0),
        # the gradient from a few stored states at the highest order
        dict(name="adjoint_5x4x6_p8_ckpt", kind="adjoint", nx=5, ny=4, nz=6, p=8, steps=20, window=5, snapshots=5,
             scheme="segments", re=400.0),
        # one right-hand side on device arrays of a caller that cannot allocate
        dict(name="rhs_noalloc_4_p8", kind="noalloc", nx=4, ny=4, nz=4, p=8, re=1600.0),
    ]


def _size(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["run"] * 6 + ["rhs", "ensemble", "adjoint", "noalloc"])
    p = rng.randint(1, 8)
    re = round(rng.uniform(100.0, 3200.0), 1)
    if kind == "ensemble":
        return dict(kind=kind, cases=rng.randint(2, 16), pick=rng.randrange(1 << 20), blocks=rng.randint(1, 2),
                    steps=rng.randint(2, 10))
    if kind == "adjoint":
        snaps = rng.choice([0, 0, 3, 5])
        p = rng.randint(3, 8)
        return dict(kind=kind, nx=_size(rng, 2, 7), ny=_size(rng, 2, 7), nz=_size(rng, 2, 7), p=p,
                    steps=rng.randint(6, 20), window=rng.randint(1, 6), snapshots=snaps,
                    scheme=rng.choice(["revolve", "segments"]), re=re)
    if kind == "noalloc":
        top = int((1 << 20) / (90 * (p + 1) ** 2 + 5 * (p + 1) ** 3))
        n = [rng.randint(2, max(2, int(top ** (1.0 / 3.0)))) for _ in range(3)]
        return dict(kind=kind, nx=n[0], ny=n[1], nz=n[2], p=p, re=re)
    shape = rng.choice(["box"] * 5 + ["curved", "walls", "band"])
    model = rng.choice(["none", "none", "none", "ev", "les"])
    if shape == "curved" and model == "les":  # the Smagorinsky model takes axis-aligned elements only
        model = "ev"
    big = 18 if shape == "box" else 8
    if shape == "band":
        p = rng.randint(2, 6)
    case = dict(kind=kind, nx=_size(rng, 3, big), ny=_size(rng, 3, big), nz=_size(rng, 3, big), p=p, shape=shape,
                re=re, model=model)
    if kind == "run":
        case.update(blocks=rng.randint(1, 3), steps=rng.randint(1, 10), iord=rng.choice([3, 4, 4]))
    else:
        case["model"] = "none"
    return case


# ------------------------------------------------------------------- meshes
@functools.lru_cache(maxsize=4)
def _straight(nx, ny, nz, p):
    """Descriptor of a straight periodic box of nx*ny*nz equal elements (y fastest, then x, then z),
    the arrays a Fortran caller packs: constant metrics, every face one conforming mortar."""
    G, ldx, ne = p + 1, p + 2, nx * ny * nz
    h = 2.0 * np.pi / np.array([nx, ny, nz], dtype=np.float64)
    J = h[0] * h[1] * h[2]
    gmetg, gmet = np.zeros((ne * ldx ** 3, 9)), np.zeros((ne * ldx ** 3, 9))
    for d in range(3):
        gmetg[:, 4 * d] = 1.0 / h[d]
        gmet[:, 4 * d] = J / h[d]
    el = np.arange(ne).reshape(nz, nx, ny)
    rows, nh, nrm = [], [], []
    # (axis of el, direction, high face, low face, the master of the periodic pair is the low face)
    for ax, d, hi, lo, low_master in ((2, 1, 2, 1, True), (1, 0, 4, 6, False), (0, 2, 5, 3, True)):
        a, b = el, np.roll(el, -1, axis=ax)  # face hi of a meets face lo of b
        wrap = np.zeros(el.shape, dtype=bool)
        np.moveaxis(wrap, ax, 0)[-1] = low_master
        r = np.zeros((ne, 17), dtype=np.int32)
        w = wrap.ravel()
        r[:, 0] = np.where(w, b.ravel(), a.ravel()) + 1
        r[:, 1] = np.where(w, a.ravel(), b.ravel()) + 1
        r[:, 2], r[:, 3] = np.where(w, lo, hi), np.where(w, hi, lo)
        r[:, 4:10] = G
        r[:, 11:] = 1
        rows.append(r)
        n = np.zeros((ne, ldx, ldx, 3))
        n[..., d] = 1.0
        nh.append(n)
        nrm.append(np.full((ne, ldx, ldx), J / h[d]))
    return dict(ngrid=ne, nmort=3 * ne, ldx=ldx, ncg=np.full(3 * ne, G, dtype=np.int32),
                jacob=np.full(ne * ldx ** 3, 1.0 / J), gmetg=gmetg.ravel(), gmet=gmet.ravel(),
                mortar=np.concatenate(rows).ravel(), n_hat=np.concatenate(nh).ravel(),
                norm=np.concatenate(nrm).ravel(), bcond=None)


@functools.lru_cache(maxsize=4)
def _shaped(nx, ny, nz, p, shape):
    """Box and descriptor of the other meshes: curved elements, walls in y, a band of order p + 2."""
    if shape == "curved":
        box = mesh.Box(nx, ny, nz, p, warp=0.02)
    elif shape == "walls":
        box = mesh.Box(nx, ny, nz, p, bc={"y": ("walladiab", "wallisoth")})
    else:
        orders = np.full((nz, nx, ny), p)
        orders[:, nx // 3:nx - nx // 3, :] = p + 2
        box = mesh.Box(nx, ny, nz, orders.ravel())
    return box, box.desc()


def _points(nx, ny, nz, p, device):
    """Coordinates x, y, z of the Gauss points, [e][l][m][n]."""
    g = torch.from_numpy(mesh.gauss_points(p + 1)).to(device)

    def axis(n):
        return (torch.arange(n, dtype=torch.float64, device=device)[:, None] + g) * (2.0 * math.pi / n)

    G = p + 1
    shape = (nz, nx, ny, G, G, G)
    x = axis(nx)[None, :, None, None, None, :].expand(shape)
    y = axis(ny)[None, None, :, None, :, None].expand(shape)
    z = axis(nz)[:, None, None, :, None, None].expand(shape)
    return [c.reshape(-1, G, G, G) for c in (x, y, z)]


def _flow(x, y, z, seed, amp=0.1, twall=TWALL):
    """Conserved variables of the Taylor-Green vortex plus a seeded divergence-free perturbation."""
    gen = np.random.default_rng(seed)
    u = torch.sin(x) * torch.cos(y) * torch.cos(z)
    v = -torch.cos(x) * torch.sin(y) * torch.cos(z)
    w = torch.zeros_like(x)
    rho = torch.ones_like(x)
    for _ in range(6):
        k = gen.integers(-3, 4, 3).astype(float)
        k[gen.integers(0, 3)] = 1.0 + gen.integers(0, 2)
        a = np.cross(k, gen.standard_normal(3))
        a *= amp / (np.linalg.norm(a) + 1e-12)
        c = torch.cos(k[0] * x + k[1] * y + k[2] * z + gen.uniform(0.0, 2.0 * np.pi))
        u, v, w = u + a[0] * c, v + a[1] * c, w + a[2] * c
        rho = rho + 0.005 * float(gen.standard_normal()) * c
    pr = twall / GAMMA + (torch.cos(2.0 * x) + torch.cos(2.0 * y)) * (torch.cos(2.0 * z) + 2.0) / 16.0
    return torch.stack([rho, rho * u, rho * v, rho * w, pr / (GAMMA - 1.0) + 0.5 * rho * (u * u + v * v + w * w)], 1)


def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _straight_state(case, seed):
    """Conserved variables [e][5][l][m][n] of a straight case, J, and the time step at CFL 0.5."""
    n, p = (case["nx"], case["ny"], case["nz"]), case["p"]
    twall = case.get("twall", TWALL)
    q = _flow(*_points(*n, p, _device()), seed, twall=twall)
    h = [2.0 * math.pi / k for k in n]
    cx = mesh.lobatto_points(p + 2)
    lam = (2.0 + math.sqrt(1.1 * twall)) * sum(1.0 / k for k in h) / float(np.diff(cx).min())
    return q, h[0] * h[1] * h[2], 0.5 / lam


def _pinned(shape):
    t = torch.zeros(shape, dtype=torch.float64, pin_memory=torch.cuda.is_available())
    return t, t.numpy()


def _padded(q, J):
    """J*Q on the host in the caller's padded layout (pinned)."""
    e, _, G = q.shape[:3]
    t, a = _pinned((e, 5, G + 1, G + 1, G + 1))
    t[..., :G, :G, :G].copy_(q * J)
    return a


def _phys(case):
    model = case.get("model", "none")
    return dict(re=case["re"], iord=case.get("iord", 4),
                **(dict(cmu=1.0, mumax=0.5, shock=1) if model == "ev" else {}))


def _ensemble_cases(case):
    """(n, p, Re, twall) of the members: sizes 4..10, p in {4, 6, 8}, Mach 0.05..0.3."""
    rng = np.random.default_rng(case["pick"])
    out = []
    for _ in range(case["cases"]):
        n, p = int(rng.choice((4, 6, 8, 10))), int(rng.choice((4, 6, 8)))
        re, ma = float(rng.uniform(400.0, 3200.0)), float(rng.uniform(0.05, 0.3))
        out.append(dict(nx=n, ny=n, nz=n, p=p, re=re, twall=1.0 / (ma * ma)))
    return out


# ------------------------------------------------------------------- passes
def prepare(case, seed):
    kind = case["kind"]
    if kind == "ensemble":
        members = _ensemble_cases(case)
        descs, qs, dts = [], [], []
        for k, m in enumerate(members):
            q, J, dt = _straight_state(m, seed * 100 + k)
            descs.append(_straight(m["nx"], m["ny"], m["nz"], m["p"]))
            qs.append(_padded(q, J))
            dts.append(dt)
        s = Ensemble(descs, [m["re"] for m in members])
        s.diag_batch(np.array(dts), first=True)  # the steps keep their gradients for the dissipation
        return SimpleNamespace(case=case, s=s, q=qs, dt=np.array(dts))
    if kind == "noalloc":
        return _prepare_noalloc(case, seed)
    shape = case.get("shape", "box")
    st = SimpleNamespace(case=case)
    if shape == "box":
        desc = _straight(case["nx"], case["ny"], case["nz"], case["p"])
        q, J, st.dt = _straight_state(case, seed)
        st.q = _padded(q, J)
    else:
        box, desc = _shaped(case["nx"], case["ny"], case["nz"], case["p"], shape)
        ldx = box.ldx
        x = [torch.from_numpy(np.ascontiguousarray(box.xg[..., k].reshape(-1, ldx, ldx, ldx))).to(_device())
             for k in range(3)]
        inv = np.where(box.jacob != 0.0, 1.0 / np.where(box.jacob != 0.0, box.jacob, 1.0), 0.0)
        q = _flow(*x, seed) * torch.from_numpy(inv.reshape(-1, 1, ldx, ldx, ldx)).to(_device())
        t, st.q = _pinned(box.qshape())
        t.copy_(q)
        st.dt = 0.3 * mesh.dtcalc(box, st.q)
    st.s = Solver(desc, **_phys(case))
    if shape == "walls":
        st.s.set_boundary(TWALL)
    if case.get("model") == "les":
        st.s.set_les(0.1, 1e3)
    st.out = _pinned(st.q.shape)[1]
    if kind == "run":
        st.s.diag(st.dt, first=True)  # the steps keep their gradients for the dissipation
    return st


def _prepare_noalloc(case, seed):
    n, p = (case["nx"], case["ny"], case["nz"]), case["p"]
    G, L, d = p + 1, p + 2, _straight(*n, p)
    q, J, _ = _straight_state(case, seed)
    ne, dev = d["ngrid"], _device()
    h = [2.0 * math.pi / k for k in n]
    nh = np.ascontiguousarray(d["n_hat"].reshape(-1, d["ldx"], d["ldx"], 3)[:, :G, :G])
    nrm = np.ascontiguousarray(d["norm"].reshape(-1, d["ldx"], d["ldx"])[:, :G, :G])

    def per_dir(vals, count):
        return torch.tensor(vals, dtype=torch.float64, device=dev)[None, :, None].repeat(ne, 1, count).contiguous()

    a = [torch.from_numpy(d["mortar"]).to(dev), torch.from_numpy(nh).to(dev), torch.from_numpy(nrm).to(dev),
         (q * J).contiguous(), torch.full((ne, G ** 3), 1.0 / J, dtype=torch.float64, device=dev),
         per_dir([1.0 / k for k in h], G ** 3), per_dir([J / k for k in h], L * G * G)]
    return SimpleNamespace(case=case, arrays=a, nel=ne, nmort=d["nmort"], qt=torch.zeros_like(q))


def run(state):
    case = state.case
    kind = case["kind"]
    if kind == "noalloc":
        vp = ctypes.c_void_p
        f = lib().dsem_rhs_noalloc
        f.argtypes = [ctypes.c_int] * 3 + [vp] * 7 + [ctypes.c_double] * 4 + [vp] * 2
        rc = f(state.nel, case["p"], state.nmort, *[vp(t.data_ptr()) for t in state.arrays], GAMMA, case["re"], PR,
               1.0, vp(state.qt.data_ptr()), vp(torch.cuda.current_stream().cuda_stream))
        if rc != 0:
            raise RuntimeError(lib().dsem_last_error(None).decode())
        return state.qt
    s = state.s
    if kind == "ensemble":
        for k, q in enumerate(state.q):
            s.upload_case(k, q)
        diags = []
        for b in range(case["blocks"]):
            s.step_batch(state.dt, case["steps"])
            diags.append(s.diag_batch(state.dt, first=b == 0))
        return [s.download_case(k) for k in range(case["cases"])], [np.concatenate(x) for x in zip(*diags)]
    s.upload(state.q)
    if kind == "rhs":
        return s.rhs()
    if kind == "adjoint":
        J, g, lr, _ = s.adjoint(state.dt, case["steps"], case["window"], case["snapshots"], scheme=case["scheme"])
        return J, g, lr
    diags = []
    for b in range(case["blocks"]):
        s.step(state.dt, case["steps"])
        diags.append(s.diag(state.dt, first=b == 0))
    return s.download(out=state.out), np.array(diags)


def _members(case):
    if case["kind"] == "ensemble":
        return [(m["nx"] * m["ny"] * m["nz"], m["p"]) for m in _ensemble_cases(case)]
    n = case["nx"] * case["ny"] * case["nz"]
    if case.get("shape") == "band":
        band = (case["nx"] - 2 * (case["nx"] // 3)) * case["ny"] * case["nz"]
        return [(n - band, case["p"]), (band, case["p"] + 2)]
    return [(n, case["p"])]


def work(case):
    """Stage evaluations times what one cannot do without.  Bytes: the state and the RK register read
    and written, the metrics read; the host arrays once each way.  Operations: the line contractions
    and the point fluxes (a multiply-add is two); a reversed stage counts as two evaluations."""
    kind = case["kind"]
    stages = len(CRK[case.get("iord", 4)])
    evals = 1.0 if kind in ("rhs", "noalloc") else float(stages * case["steps"] * case.get("blocks", 1))
    fwd = 3.0 if kind == "adjoint" else 1.0
    by = fl = 0.0
    for n, p in _members(case):
        G, L = p + 1, p + 2
        metrics = 9.0 * (G ** 3 + L * G * G) if case.get("shape") == "curved" else 3.0 * (G ** 3 + L * G * G)
        state = 5.0 * G ** 3
        by += 8.0 * n * (evals * fwd * (4.0 * state + G ** 3 + metrics) + (2.0 * state if kind != "noalloc" else 0.0))
        line = 3 * G * G * (5 * (L - 2) * 2 * G + 5 * G * 2 * L + 11 * L * 2 * G + 5 * G * 2 * (L - 2))
        point = 3 * L * G * G * 110 + 3 * G * G * 160 + 5 * G ** 3 * 17 + 30 * G * G * 2 * G
        fl += float(n) * evals * fwd * (line + point)
    return {"bytes": by, "flops": fl}


# -------------------------------------------------- the same in plain torch
def _operators(p, dev):
    """D [G][L]: derivative at the Gauss points from Lobatto values; B [L][G]: Gauss to Lobatto;
    w [G]: weights that integrate the Gauss interpolant over [0, 1]."""
    G, L = p + 1, p + 2
    cg, cl = mesh.gauss_points(G), mesh.lobatto_points(L)

    def basis(nodes, x):
        out = np.ones((len(x), len(nodes)))
        for j in range(len(nodes)):
            for m in range(len(nodes)):
                if m != j:
                    out[:, j] *= (x - nodes[m]) / (nodes[j] - nodes[m])
        return out

    D = np.zeros((G, L))
    for k in range(G):
        for j in range(L):
            for i in range(L):
                if i != j:
                    others = [m for m in range(L) if m not in (i, j)]
                    D[k, j] += np.prod([(cg[k] - cl[m]) / (cl[j] - cl[m]) for m in others]) / (cl[j] - cl[i])
    x, w = np.polynomial.legendre.leggauss(G + 2)
    wt = (0.5 * w[:, None] * basis(cg, 0.5 * (x + 1.0))).sum(0)
    return [torch.from_numpy(a).to(dev) for a in (D, basis(cg, cl), wt)]


def _along(M, a, d):
    """Contract the point axis of direction d (0: last) with the rows of M."""
    return torch.tensordot(a, M, dims=([-1 - d], [1])).movedim(-1, -1 - d)


def _roe(n, Ql, Qr):
    """Roe's flux with an entropy fix on the acoustic waves along axis n, from the upwind side."""
    out = []
    for Q in (Ql, Qr):
        r = Q[:, 0]
        vel = [Q[:, 1 + i] / r for i in range(3)]
        p = (GAMMA - 1.0) * (Q[:, 4] - 0.5 * r * (vel[0] ** 2 + vel[1] ** 2 + vel[2] ** 2))
        out.append((r, vel, p, 0.5 * (vel[0] ** 2 + vel[1] ** 2 + vel[2] ** 2) + GAMMA / (GAMMA - 1.0) * p / r))
    (rl, vl, pl, hl), (rr, vr, pr, hr) = out
    rt = torch.sqrt(rl * rr)
    b = rl / (rl + rt)
    vt = [b * vl[i] + (1.0 - b) * vr[i] for i in range(3)]
    ht = b * hl + (1.0 - b) * hr
    a2 = (GAMMA - 1.0) * (ht - 0.5 * (vt[0] ** 2 + vt[1] ** 2 + vt[2] ** 2))
    a, qt = torch.sqrt(a2), vt[n]
    dp, dq = (pr - pl) / a2, (vr[n] - vl[n]) * rt / a

    def side(r, vel, p, h, sgn):
        dw = 0.5 * (dp - sgn * dq)
        sp = qt - sgn * a
        e = -sp.abs() - sgn * (GAMMA + 1.0) / 4.0 * a / rt * dw
        # the wave's contribution, added on the left and taken off on the right
        ud = sgn * dw * (torch.clamp(sgn * sp, max=0.0) - 0.5 * torch.clamp(e, min=0.0))
        rq = r * vel[n]
        f = [rq + sgn * ud]
        for i in range(3):
            f.append(rq * vel[i] + (p if i == n else 0.0) + sgn * ud * (vt[i] - (sgn * a if i == n else 0.0)))
        f.append(rq * h + sgn * ud * (ht - sgn * qt * a))
        return torch.stack(f, 1)

    return torch.where((qt >= 0.0)[:, None], side(rl, vl, pl, hl, 1.0), side(rr, vr, pr, hr, -1.0))


def _viscous(d, Q, g, kap):
    """Viscous flux of direction d; g[j][v] is the gradient of variable v along j."""
    r = Q[:, 0]
    vel = [Q[:, 1 + i] / r for i in range(3)]
    dv = [[(g[j][1 + i] - vel[i] * g[j][0]) / r for j in range(3)] for i in range(3)]
    ke = vel[0] ** 2 + vel[1] ** 2 + vel[2] ** 2
    p = (GAMMA - 1.0) * (Q[:, 4] - 0.5 * r * ke)
    pd = (GAMMA - 1.0) * (g[d][4] - 0.5 * g[d][0] * ke - r * sum(vel[i] * dv[i][d] for i in range(3)))
    td = GAMMA * (pd - p * g[d][0] / r) / r
    div = dv[0][0] + dv[1][1] + dv[2][2]
    tau = [dv[i][d] + dv[d][i] - (2.0 / 3.0 * div if i == d else 0.0) for i in range(3)]
    return torch.stack([torch.zeros_like(r)] + tau + [sum(vel[i] * tau[i] for i in range(3)) + kap * td], 1)


class _Plain:
    """The right-hand side on a straight periodic box, arrays [e][...][l][m][n]."""

    AXIS = (1, 2, 0)  # of the element grid [z][x][y], per direction

    def __init__(self, case, dev):
        self.n = (case["nz"], case["nx"], case["ny"])
        self.h = [2.0 * math.pi / case[k] for k in ("nx", "ny", "nz")]
        self.J = self.h[0] * self.h[1] * self.h[2]
        self.re, self.G = case["re"], case["p"] + 1
        self.D, self.B, self.w = _operators(case["p"], dev)

    def neighbour(self, a, d, step):
        """a of the next (step = 1) or previous (-1) element along d."""
        return torch.roll(a.reshape(self.n + a.shape[1:]), -step, self.AXIS[d]).reshape(a.shape)

    def faces(self, a, d):
        """a's values (lo, hi) at the two ends of direction d of a Lobatto array."""
        return a.select(-1 - d, 0), a.select(-1 - d, a.shape[-1 - d] - 1)

    def gradients(self, Q):
        """Lobatto states per direction (face values averaged), Roe fluxes at the high faces, gradients."""
        lob, roe, grad = [], [], []
        for d in range(3):
            y = _along(self.B, Q, d)
            lo, hi = self.faces(y, d)
            nxt = self.neighbour(lo, d, 1)
            roe.append(_roe(d, hi, nxt))
            avg = 0.5 * (hi + nxt)
            mid = y.narrow(-1 - d, 1, y.shape[-1 - d] - 2)
            y = torch.cat([self.neighbour(avg, d, -1).unsqueeze(-1 - d), mid, avg.unsqueeze(-1 - d)], -1 - d)
            lob.append(y)
            grad.append(_along(self.D, y, d) / self.h[d])
        return lob, roe, grad

    def rhs(self, Q):
        """J times the time derivative of Q, and the gradients at the Gauss points."""
        lob, roe, grad = self.gradients(Q)
        total = 0.0
        kap = GAMMA / (PR * GAMMA * (GAMMA - 1.0))
        for d in range(3):
            area = self.J / self.h[d]
            g = [list(_along(self.B, grad[j], d).unbind(1)) for j in range(3)]
            vis = _viscous(d, lob[d], g, kap)
            q = lob[d]
            u = q[:, 1 + d] / q[:, 0]
            p = (GAMMA - 1.0) * (q[:, 4] - 0.5 * (q[:, 1] ** 2 + q[:, 2] ** 2 + q[:, 3] ** 2) / q[:, 0])
            f = q * u[:, None]
            add = [torch.zeros_like(p)] * 5
            add[1 + d], add[4] = p, u * p
            f = f + torch.stack(add, 1) - vis / self.re
            lo, hi = self.faces(vis, d)
            end = roe[d] - 0.5 * (hi + self.neighbour(lo, d, 1)) / self.re
            mid = f.narrow(-1 - d, 1, f.shape[-1 - d] - 2)
            f = torch.cat([self.neighbour(end, d, -1).unsqueeze(-1 - d), mid, end.unsqueeze(-1 - d)], -1 - d)
            total = total - area * _along(self.D, f, d)
        return total, grad

    def step(self, JQ, dt, iord, keep=False):
        """One step; the gradients of its last stage when keep."""
        g, grad = torch.zeros_like(JQ), None
        for k, (a, c) in enumerate(zip(ARK[iord], CRK[iord])):
            last = keep and k == len(CRK[iord]) - 1

            def stage(JQ, g, a=a, c=c, last=last):
                Qt, grad = self.rhs(JQ / self.J)
                g = a * g + Qt
                return (JQ + c * dt * g, g) + (tuple(grad) if last else ())

            r = checkpoint(stage, JQ, g, use_reentrant=False) if JQ.requires_grad else stage(JQ, g)
            JQ, g = r[0], r[1]
            grad = list(r[2:]) if last else None
        return JQ, grad

    def diag(self, JQ, grad, dt, previous):
        q = JQ / self.J
        vel = [q[:, 1 + i] / q[:, 0] for i in range(3)]
        w3 = self.w[:, None, None] * self.w[None, :, None] * self.w
        ke = 0.5 * (sum(v ** 2 for v in vel) * w3).sum() * self.J / (8.0 * math.pi ** 3)
        return ke, (previous - ke) / dt, self.eps(JQ, grad)

    def eps(self, JQ, grad):
        q = JQ / self.J
        dv = [[(grad[j][:, 1 + i] - q[:, 1 + i] / q[:, 0] * grad[j][:, 0]) / q[:, 0] for j in range(3)]
              for i in range(3)]
        w2 = (dv[2][1] - dv[1][2]) ** 2 + (dv[0][2] - dv[2][0]) ** 2 + (dv[1][0] - dv[0][1]) ** 2
        return 100.0 * w2.mean() / self.re


def _unpadded_to_padded(a):
    G = a.shape[-1]
    out = torch.zeros(a.shape[:2] + (G + 1,) * 3, dtype=a.dtype)
    out[..., :G, :G, :G] = a.detach().cpu()
    return out.numpy()


def _exact_run(case, q, J, dt):
    P = _Plain(case, q.device)
    JQ, prev, diags = q * J, 0.0, []
    for _ in range(case["blocks"]):
        for k in range(case["steps"]):
            JQ, grad = P.step(JQ, dt, case.get("iord", 4), keep=k == case["steps"] - 1)
        ke, dk, ep = P.diag(JQ, grad, dt, prev)
        prev = ke
        diags.append((float(ke), float(dk), float(ep)))
    return _unpadded_to_padded(JQ), np.array(diags)


def exact(case, seed):
    kind = case["kind"]
    if case.get("shape", "box") != "box" or case.get("model", "none") != "none":
        return None
    if kind == "ensemble":
        states, diags = [], []
        for k, m in enumerate(_ensemble_cases(case)):
            q, J, dt = _straight_state(m, seed * 100 + k)
            a, d = _exact_run(dict(m, blocks=case["blocks"], steps=case["steps"]), q, J, dt)
            states.append(a)
            diags.append(d)
        d = np.stack(diags, 1)  # [block][case][3]
        return states, [np.ascontiguousarray(d[..., i].ravel()) for i in range(3)]
    q, J, dt = _straight_state(case, seed)
    P = _Plain(case, q.device)
    if kind == "run":
        return _exact_run(case, q, J, dt)
    if kind in ("rhs", "noalloc"):
        Qt = P.rhs(q)[0]
        return Qt if kind == "noalloc" else _unpadded_to_padded(Qt)
    inv_re = torch.tensor(1.0 / case["re"], dtype=torch.float64, device=q.device, requires_grad=True)
    P.re = 1.0 / inv_re
    start = (q * J).requires_grad_(True)
    JQ, obj = start, 0.0
    for k in range(case["steps"]):
        inside = k >= case["steps"] - case["window"]
        JQ, grad = P.step(JQ, dt, 4, keep=inside)
        if inside:
            obj = obj + P.eps(JQ, grad) * dt
    g, lr = torch.autograd.grad(obj, (start, inv_re))
    return float(obj.detach()), _unpadded_to_padded(g), float(lr)
