"""The work a user of cmsl_gb300 has it do, as cases that can be timed.

Every case is one call sequence of a user's program through the public entry
points (``Film``, ``Batch``, ``Film.loop_gradient``, the C ABI's
``cmsl_film_depol_device``) on a synthetic film: a columnar periodic Voronoi
map, random grain orientations and the Landau coefficients of
``cmsl_gb300.workloads``.  ``kind`` says which:

  loop      a segment of a P-E loop: state in, ``steps`` time steps with one
            sweep row each, rows and state out
  batch     the same on several films of uneven size advancing together
  gradient  loss and Landau-coefficient gradient of a short loop (adjoint)
  depol     one depolarisation solve on the caller's device arrays, as the
            reference's Depol_field() callers do every step

``exact`` restates each of them in plain FP64 torch.
"""
from __future__ import annotations

import ctypes as C
import math
import random

import numpy as np
import torch

import cmsl_gb300 as cg
from cmsl_gb300 import workloads as wl

DEV = "cuda"
ONE = (30.0, 30.0, 30.0)       # permittivities of AFE, FE, DE: one for all materials
DECK = (50.0, 30.0, 15.0)      # the reference deck's


def _loop(name, nx, ny, nz, steps, *, precision="fp32", eps="one", zbc="dirichlet", grains=20, afe=0.4, de=0.0,
          init="pz", amp=4.0, period=4000):
    return dict(name=name, kind="loop", nx=nx, ny=ny, nz=nz, steps=steps, precision=precision, eps=eps, zbc=zbc,
                grains=grains, afe=afe, de=de, init=init, amp=amp, period=period)


def listed():
    return [
        # the plain small film (64 x 64 x 16, 20 FE grains, +-3 MV/cm), FP32-refined: a step is launch latency
        _loop("loop_64x64x16_fp32", 64, 64, 16, 200, afe=0.0, amp=3.0, period=2000),
        # the headline film: 256 x 256 x 32, 200 grains, 40 % AFE, +-4 MV/cm
        _loop("loop_256x256x32_fp32", 256, 256, 32, 120, grains=200),
        # the large film: 512 x 512 x 64, 2000 grains, 25 % AFE, from a random state
        _loop("loop_512x512x64_fp32", 512, 512, 64, 18, grains=2000, afe=0.25, init="random", amp=2.0),
        # a film of uneven sides of the ensemble's kind (2^a 3^b)
        _loop("loop_192x96x24_fp32", 192, 96, 24, 150, grains=60, afe=0.3),
        # the reference deck's permittivities with DE grains (50 / 30 / 15)
        _loop("loop_256x256x32_deck_fp32", 256, 256, 32, 40, grains=200, afe=0.3, de=0.1, eps="deck"),
        # odd, ragged sides: no fast transform applies, the persistent PCG solves
        _loop("loop_150x110x21_fp32", 150, 110, 21, 40, grains=50),
        # the Neumann z boundary the reference's deck can select
        _loop("loop_96x64x12_neumann_fp32", 96, 64, 12, 12, grains=30, zbc="neumann"),
        # the reference's precision and algorithm (FP64 PCG to 1e-8): small and headline film
        _loop("loop_64x64x16_fp64", 64, 64, 16, 20, precision="fp64", afe=0.0, amp=3.0, period=2000),
        _loop("loop_256x256x32_deck_fp64", 256, 256, 32, 4, precision="fp64", grains=200, afe=0.3, de=0.1, eps="deck"),
        # a campaign's films advancing together (sides 64 .. 256, 8 .. 32 planes)
        dict(name="batch_16_fp32", kind="batch", films=16, sizes=3, steps=60),
        # coefficient fitting: loss and gradient of a short loop on the 128 x 128 x 16 film
        dict(name="gradient_128x128x16", kind="gradient", nx=128, ny=128, nz=16, steps=16, every=8, grains=50, afe=0.3),
        # Depol_field() over the caller's device arrays, FP64
        dict(name="depol_96x80x20_fp64", kind="depol", nx=96, ny=80, nz=20, precision="fp64", eps="deck", grains=40,
             afe=0.3, de=0.1),
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng: random.Random):
    kind = rng.choice(["loop"] * 6 + ["batch", "gradient", "depol"])
    if kind == "batch":
        return dict(kind=kind, films=rng.randint(3, 16), sizes=rng.randint(4, 1 << 20), steps=rng.randint(20, 60))
    friendly = [32, 36, 48, 64, 72, 96, 108, 128, 144, 192, 216, 256, 288, 384, 512]
    if kind == "gradient":
        nx, ny = (rng.choice([24, 33, 48, 64, 90, 96, 128]) for _ in range(2))
        return dict(kind=kind, nx=nx, ny=ny, nz=rng.randint(5, 16), steps=rng.randint(6, 16), every=rng.randint(3, 16),
                    grains=rng.randint(4, 50), afe=round(rng.uniform(0.1, 0.6), 2))
    if kind == "depol":
        return dict(kind=kind, nx=_logint(rng, 17, 160), ny=_logint(rng, 17, 160), nz=rng.randint(5, 32),
                    precision=rng.choice(["fp64", "fp32"]), eps=rng.choice(["one", "deck"]), grains=rng.randint(4, 80),
                    afe=round(rng.uniform(0.1, 0.6), 2), de=0.1)
    what = rng.choice(["fast"] * 4 + ["odd", "neumann", "fp64", "fp64"])
    eps = rng.choice(["one", "one", "deck"])
    zbc, precision = "dirichlet", "fp32"
    if what == "fast":
        nz = _logint(rng, 5, 64)
        nx, ny = rng.choice(friendly), rng.choice(friendly)
        budget, cap = (3.0e8, 200) if eps == "one" else (6.0e7, 60)
    elif what == "odd":
        nx, ny, nz = _logint(rng, 25, 320), _logint(rng, 25, 320), rng.randint(5, 40)
        budget, cap, eps = 1.0e7, 60, "one"
    elif what == "neumann":
        nx, ny, nz = rng.choice(friendly[:7]), rng.choice(friendly[:7]), rng.randint(5, 14)
        budget, cap, zbc = 1.0e6, 20, "neumann"
    else:
        nx, ny, nz = _logint(rng, 25, 220), _logint(rng, 25, 220), rng.randint(5, 32)
        budget, cap, precision = 4.0e6, 20, "fp64"
    steps = max(3, min(cap, int(budget / (nx * ny * nz))))
    c = _loop("", nx, ny, nz, steps, precision=precision, eps=eps, zbc=zbc, grains=max(4, nx * ny // 350),
              afe=round(rng.uniform(0.0, 0.6), 2), de=0.1 if eps == "deck" else 0.0,
              init=rng.choice(["pz", "random"]), amp=round(rng.uniform(2.0, 5.0), 2), period=2000)
    del c["name"]
    return c


def _batch_films(case):
    """The films of a batch: sides and thickness as a campaign mixes them."""
    r = random.Random(case["sizes"])
    out = []
    for _ in range(case["films"]):
        side = r.choice([64, 96, 128, 192, 256])
        out.append(dict(kind="loop", nx=side, ny=side, nz=r.choice([8, 16, 32]), steps=case["steps"], precision="fp32",
                        eps="one", zbc="dirichlet", grains=r.randint(10, 400), afe=round(r.uniform(0.0, 0.6), 2), de=0.0,
                        init="pz", amp=round(r.uniform(2.0, 5.0), 2), period=2000))
    return out


# ------------------------------------------------------------------ inputs
def _nd(eps):
    """Non-dimensional materials [3, 8] and scales (workloads.hzo_film's coefficients)."""
    a1, a11, a111, J = -2.0e9, 1.0e10, 5.0e10, 3.0e9
    com = dict(a0=1.0e9, L=1.0, kappa=1.0e-10)
    fe = dict(alpha=4 * a1, beta=32 * a11, gamma1=192 * a111, g=0.0, eps_r=eps[1], **com)
    afe = dict(fe, alpha=4 * a1 - J, g=J, eps_r=eps[0])
    de = dict(alpha=abs(4 * a1), beta=0.0, gamma1=0.0, g=0.0, eps_r=eps[2], **com)
    ar, p0 = wl.make_phase_refs(fe)
    mats = np.stack([wl.make_nd(afe, ar, p0), wl.make_nd(fe, ar, p0), wl.make_nd(de, ar, p0)])
    return mats, 0.25 * ar * p0, 4.0 / (wl.EPS0 * abs(fe["alpha"])), p0


def _inputs(c, seed):
    """Grain map (in-plane, columnar), grain tables, materials and the initial P [6, nz, ny, nx] (GPU, FP64)."""
    nx, ny, nz, ng = c["nx"], c["ny"], c["nz"], c["grains"]
    rng = np.random.default_rng(seed)
    gen = torch.Generator(DEV).manual_seed(int(rng.integers(1 << 62)))
    sx, sy = (torch.from_numpy(rng.uniform(0.0, n, ng)).to(DEV) for n in (nx, ny))
    xs = torch.arange(nx, device=DEV, dtype=torch.float64) + 0.5
    g2 = torch.empty((ny, nx), dtype=torch.int64, device=DEV)
    rows = max(1, 40_000_000 // (nx * ng))
    dx = (xs[:, None] - sx).abs()
    dx = torch.minimum(dx, nx - dx) ** 2
    for j in range(0, ny, rows):
        ys = torch.arange(j, min(ny, j + rows), device=DEV, dtype=torch.float64) + 0.5
        dy = (ys[:, None] - sy).abs()
        dy = torch.minimum(dy, ny - dy) ** 2
        g2[j:j + rows] = (dx[None] + dy[:, None]).argmin(-1)
    TR = wl.tr_from_euler(*wl.orientations(ng, rng))
    gm = np.full(ng, 1, np.int32)
    order = rng.permutation(ng)
    n_afe, n_de = int(round(c["afe"] * ng)), int(round(c.get("de", 0.0) * ng))
    gm[order[:n_afe]] = 0
    gm[order[n_afe:n_afe + n_de]] = 2
    mats, E0, eps0, P0 = _nd(DECK if c.get("eps") == "deck" else ONE)
    mat2 = torch.from_numpy(gm.astype(np.int64)).to(DEV)[g2]
    P = torch.zeros((6, nz, ny, nx), dtype=torch.float64, device=DEV)
    if c.get("init", "random") == "pz":
        u = torch.rand((nz, ny, nx), dtype=torch.float64, device=DEV, generator=gen)
        P[2] = (0.02 * u - 0.01) / P0 * (mat2 == 1)
        P[3:] = (mat2 == 0).double()
    else:
        P.uniform_(-0.1, 0.1, generator=gen)
    Emax = c.get("amp", 4.0) * 1.0e8 / E0
    return dict(g2=g2, gm=gm, TR=TR, mats=mats, eps0=eps0, P=P, Emax=Emax, mat2=mat2)


def _schedule(c, Emax):
    """The first steps of the triangle wave (a field step per time step, evolve_schedule's), one row a step."""
    n = c["steps"]
    if c.get("init") == "random":
        Ez = np.full(n, Emax)
    else:
        Ez = np.arange(n) * (4.0 * Emax / c["period"])
    return Ez, np.arange(n, dtype=np.int32)


def _film_kw(c, inp):
    N = c["nx"] * c["ny"] * c["nz"]
    fp64 = c["precision"] == "fp64"
    return dict(nx=c["nx"], ny=c["ny"], nz=c["nz"],
                omega=inp["g2"].to(torch.int32).cpu().numpy()[None].repeat(c["nz"], 0).reshape(N), grain_mat=inp["gm"],
                TR=inp["TR"], mats=inp["mats"], del_h=0.5, del_t=1.0e-3, dep_flag=1, eps_0_nd=inp["eps0"],
                zbc=cg.NEUMANN if c.get("zbc") == "neumann" else cg.DIRICHLET,
                precision=cg.FP64 if fp64 else cg.FP32_REFINED, pcg_crit=cg.CRIT_RELRES, tol_rel=c.get("tol", 1e-8),
                max_iter=20000, refine_tol=1e-8, max_refine=6, inner_tol=1e-5, inner_max_iter=2000, warm_start=2)


class _Host:
    """Page-locked state arrays of one film, in and out, as a campaign keeps them."""

    def __init__(self, P):
        n = P[0].numel()
        self.P = cg.pinned_empty((6, n))
        self.P[:] = P.reshape(6, n).cpu().numpy()
        self.outP, self.outphi = cg.pinned_empty((6, n)), cg.pinned_empty((n,))
        self.Pin, self.out = [self.P[q] for q in range(6)], ([self.outP[q] for q in range(6)], self.outphi)


def _state32(h):
    """The film's state as FP32 tensors on the GPU: what an FP32_REFINED film holds of P and phi."""
    return {"P": torch.from_numpy(h.outP).to(DEV, non_blocking=True).float(),
            "phi": torch.from_numpy(h.outphi).to(DEV, non_blocking=True).float()}


def _rows(r, fp32):
    return {"rows": r[:, :10].astype(np.float32) if fp32 else r[:, :10].copy(), "n": r[:, 10].astype(np.int64)}


def prepare(case, seed):
    kind = case["kind"]
    if kind == "batch":
        films = _batch_films(case)
        inps = [_inputs(c, seed * 1000 + i) for i, c in enumerate(films)]
        b = cg.Batch([_film_kw(c, i) for c, i in zip(films, inps)])
        sch = [_schedule(c, i["Emax"]) for c, i in zip(films, inps)]
        return dict(kind=kind, batch=b, host=[_Host(i["P"]) for i in inps], Ez=np.stack([s[0] for s in sch]),
                    rows=np.stack([s[1] for s in sch]))
    c = dict(case)
    if kind == "gradient":
        c.update(precision="fp64", tol=1e-11, init="pz", amp=4.0, period=4000)
    if kind == "depol":
        c.update(init="random")
    inp = _inputs(c, seed)
    film = cg.Film(**_film_kw(c, inp))
    st = dict(kind=kind, film=film, fp32=c["precision"] == "fp32")
    if kind == "depol":
        st["P"] = [inp["P"][q].reshape(-1).contiguous() for q in range(3)]
        st["out"] = torch.zeros((4, inp["P"][0].numel()), dtype=torch.float64, device=DEV)
        return st
    st["host"] = _Host(inp["P"])
    st["Ez"], st["rows"] = _schedule(c, inp["Emax"])
    if kind == "gradient":
        st["every"] = c["every"]
        st["target"] = _target(c["steps"])
    return st


def _target(n):
    return 0.02 * np.sin(np.linspace(0.0, 2.0 * np.pi, n))


def run(state):
    kind = state["kind"]
    if kind == "batch":
        b = state["batch"]
        for i, h in enumerate(state["host"]):
            b.set_state(i, h.Pin)
        b.run(state["Ez"], state["rows"])
        out = []
        for i, h in enumerate(state["host"]):
            b.get_state(i, out=h.out)
            out.append({**_state32(h), **_rows(b.rows(i), True)})
        return out
    f = state["film"]
    if kind == "depol":
        # Depol_field(): Pm in; potential (from zero) and field out, all on the device
        from cmsl_gb300._lib import check, lib
        out = state["out"]
        out[0].zero_()
        it, st = np.zeros(2, np.int32), np.zeros(1, np.int32)
        p = [C.c_void_p(t.data_ptr()) for t in state["P"]] + [C.c_void_p(out[q].data_ptr()) for q in range(4)]
        ip = C.POINTER(C.c_int32)
        check(lib().cmsl_film_depol_device(f._h, *p, C.c_void_p(torch.cuda.current_stream().cuda_stream or None),
                                           it.ctypes.data_as(ip), st.ctypes.data_as(ip)))
        if st[0]:
            raise RuntimeError("depolarisation solve: status %d" % st[0])
        return {"phi_E": out.float() if state["fp32"] else out.clone()}
    h = state["host"]
    f.set_state(h.Pin)
    if kind == "gradient":
        loss, grad = f.loop_gradient(state["Ez"], state["rows"], state["target"], state["every"])
        return {"loss": np.array([loss]), "grad": grad}
    f.run(state["Ez"], state["rows"])
    f.get_state(out=h.out)
    r = _rows(f.rows(), state["fp32"])
    if state["fp32"]:
        return {**_state32(h), **r}
    return {"P": h.outP, "phi": h.outphi, **r}


def work(case):
    """Bytes: every step reads and writes P and the potential once and reads the grain map; the state goes in
    and out of the host once (doubles).  Flops: the TDGL update (about 200 a cell) and one transform solve."""
    if case["kind"] == "batch":
        w = [work(c) for c in _batch_films(case)]
        return {k: sum(x[k] for x in w) for k in ("bytes", "flops")}
    n = case["nx"] * case["ny"] * case["nz"]
    s = 8 if case.get("precision", "fp64") == "fp64" else 4
    solve = n * (10.0 * math.log2(case["nx"] * case["ny"]) + 30.0)
    if case["kind"] == "depol":
        return {"bytes": n * (3 * 8 + 4 + 4 * 8), "flops": solve + 30.0 * n}
    step_b, step_f = n * (12 * s + 16 + 4), 200.0 * n + solve
    if case["kind"] == "gradient":
        # forward, and a backward step of each (reads P, reads and writes lambda; one adjoint solve)
        return {"bytes": case["steps"] * (step_b + n * (6 * 8 + 12 * 8 + 16 + 4)) + 48 * n,
                "flops": case["steps"] * (step_f + 400.0 * n + solve)}
    return {"bytes": case["steps"] * step_b + n * (6 * 8 + 7 * 8), "flops": case["steps"] * step_f}


# ------------------------------------------------------------- exact (FP64)
class _Sim:
    """TDGL step and depolarisation solve of a columnar film in FP64 torch."""
    h, dt = 0.5, 1.0e-3

    def __init__(self, c, inp):
        self.nx, self.ny, self.nz = c["nx"], c["ny"], c["nz"]
        self.neu = c.get("zbc") == "neumann"
        self.t = torch.from_numpy(inp["TR"].reshape(-1, 9)).to(DEV)[inp["g2"]].permute(2, 0, 1).contiguous()[:, None]
        self.mat = inp["mat2"]
        self.m8 = torch.from_numpy(inp["mats"]).to(DEV)
        self.eps0 = inp["eps0"]
        eps = self.m8[:, 7]
        used = eps[torch.from_numpy(np.unique(inp["gm"]).astype(np.int64)).to(DEV)]
        self.one = bool((used == used[0]).all())
        self.eref = float(0.5 * (used.min() + used.max()))
        self.e2 = eps[self.mat]
        harm = lambda a, b: 2.0 * a * b / (a + b)  # noqa: E731
        self.ex, self.ey = harm(self.e2, self.e2.roll(-1, 1)), harm(self.e2, self.e2.roll(-1, 0))
        lx = 2.0 - 2.0 * torch.cos(2 * math.pi * torch.arange(self.nx // 2 + 1, device=DEV, dtype=torch.float64) / self.nx)
        ly = 2.0 - 2.0 * torch.cos(2 * math.pi * torch.arange(self.ny, device=DEV, dtype=torch.float64) / self.ny)
        n = self.nz if self.neu else self.nz - 2
        T = 2.0 * np.eye(n) - np.eye(n, k=1) - np.eye(n, k=-1)
        w = np.ones(n)
        if self.neu:
            T[0, 1] = T[-1, -2] = -2.0
            w[0] = w[-1] = 0.5
        sw = np.sqrt(w)
        lam, Q = np.linalg.eigh(sw[:, None] * T / sw[None])
        self.V, self.Vi = (torch.from_numpy(a).to(DEV) for a in (Q / sw[:, None], Q.T * sw[None]))
        if self.neu:
            lam[0] = 0.0
        den = torch.from_numpy(lam).to(DEV)[:, None, None] + ly[:, None] + lx
        self.inv = torch.where(den.abs() < 1e-11, torch.zeros_like(den), 1.0 / den)
        self.w = torch.from_numpy(w).to(DEV)[:, None, None]
        self.pin = (self.nz // 2, self.ny // 2, self.nx // 2)

    def params(self, m8):
        """Per-column TDGL coefficients of materials m8 [3, 8] (alpha, beta, gamma, g, a0, kappa, L, eps)."""
        g = lambda v: v[self.mat][None]  # noqa: E731
        A = m8[:, 5] * self.dt / (self.h * self.h)
        return dict(A=g(A), relax=g(1.0 - 6.0 * A), LdT=g(m8[:, 6] * self.dt), ag=g(2 * (m8[:, 0] + m8[:, 3])),
                    ags=g(2 * (m8[:, 0] - m8[:, 3])), b4=g(4 * m8[:, 1]), b12=g(12 * m8[:, 1]), g6=g(6 * m8[:, 2]),
                    a02=g(2 * m8[:, 4]))

    def field(self, phi):
        """-E = (phi_+ - phi_-) / 2h."""
        i2 = 1.0 / (2.0 * self.h)
        ex = (phi.roll(-1, 2) - phi.roll(1, 2)) * i2
        ey = (phi.roll(-1, 1) - phi.roll(1, 1)) * i2
        if self.neu:
            up = torch.cat([phi[1:], phi[-2:-1]])
            dn = torch.cat([phi[1:2], phi[:-1]])
        else:
            z = torch.zeros_like(phi[:1])
            up, dn = torch.cat([phi[1:], z]), torch.cat([z, phi[:-1]])
        return ex, ey, (up - dn) * i2

    def step(self, P, phi, Ez, K):
        t = self.t
        S = P.roll(-1, 3) + P.roll(1, 3) + P.roll(-1, 2) + P.roll(1, 2)
        S = S + torch.cat([P[:, 1:], P[:, -1:]], 1) + torch.cat([P[:, :1], P[:, :-1]], 1)
        loc = [t[3 * a] * P[3 * s] + t[3 * a + 1] * P[3 * s + 1] + t[3 * a + 2] * P[3 * s + 2] for s in (0, 1) for a in range(3)]
        m, q = loc[2], loc[5]
        dm = K["ag"] * m + K["b4"] * m ** 3 + K["b12"] * m * q * q + K["g6"] * (m ** 5 + 10 * m ** 3 * q * q + 5 * m * q ** 4)
        dq = K["ags"] * q + K["b4"] * q ** 3 + K["b12"] * q * m * m + K["g6"] * (q ** 5 + 10 * m * m * q ** 3 + 5 * q * m ** 4)
        E = self.field(phi)
        out = []
        for s, dz in ((0, dm), (1, dq)):
            dx, dy = K["a02"] * loc[3 * s], K["a02"] * loc[3 * s + 1]
            for a in range(3):
                b = t[a] * dx + t[3 + a] * dy + t[6 + a] * dz
                if s == 0:
                    b = b + E[a] - (Ez if a == 2 else 0.0)
                out.append(P[3 * s + a] * K["relax"] + K["A"] * S[3 * s + a] - K["LdT"] * b)
        return torch.stack(out), m, q

    def rows(self, P, m, q):
        o = torch.zeros(10, dtype=torch.float64, device=DEV)
        o[0], o[1], o[2], o[3] = P[2].mean(), P[5].mean(), m.mean(), q.mean()
        for i, k in ((4, 1), (6, 0), (8, 2)):
            sel = (self.mat == k).double()
            n = sel.sum() * self.nz
            if n > 0:
                o[i], o[i + 1] = (P[2] * sel).sum() / n, n / P[2].numel()
        return o

    def rhs(self, P):
        up = torch.cat([P[2][1:], P[2][-1:]])
        dn = torch.cat([P[2][:1], P[2][:-1]])
        b = -(self.eps0 / (2.0 * self.h)) * (P[0].roll(-1, 2) - P[0].roll(1, 2) + P[1].roll(-1, 1) - P[1].roll(1, 1) + up - dn)
        if self.neu:
            b = b.clone()
            b[self.pin] = 0.0
            return b
        z = torch.zeros_like(b[:1])
        return torch.cat([z, b[1:-1], z])

    def apply(self, x):
        """A x with the film's harmonic face permittivities (columnar: eps on the z faces)."""
        if self.neu:
            up, dn = torch.cat([x[1:], x[-2:-1]]), torch.cat([x[1:2], x[:-1]])
        else:
            z = torch.zeros_like(x[:1])
            up, dn = torch.cat([x[1:], z]), torch.cat([z, x[:-1]])
        fx, fy = self.ex * (x.roll(-1, 2) - x), self.ey * (x.roll(-1, 1) - x)
        a = fx - fx.roll(1, 2) + fy - fy.roll(1, 1) + self.e2 * (up + dn - 2.0 * x)
        a = -a / (self.h * self.h)
        if self.neu:
            a[self.pin] = x[self.pin]
            return a
        return torch.cat([x[:1], a[1:-1], x[-1:]])

    def fast(self, r):
        """The solve with eps = eref on every face (exact where it is the film's)."""
        if self.neu:
            r = r.clone()
            at = r[self.pin].clone()
            r[self.pin] = 0.0
            wp = self.w[self.pin[0], 0, 0]
            r[self.pin] = -(self.w * r).sum() / wp
        else:
            r = r[1:-1]
        s = self.h * self.h / self.eref
        X = torch.fft.rfft2(torch.einsum("ij,jyx->iyx", self.Vi, r)) * self.inv * s
        x = torch.einsum("ij,jyx->iyx", self.V, torch.fft.irfft2(X, s=(self.ny, self.nx)))
        if self.neu:
            return x - x[self.pin] + at
        z = torch.zeros_like(x[:1])
        return torch.cat([z, x, z])

    def solve(self, b, tol=1e-13):
        if self.one:
            return self.fast(b)
        # PCG in the inner product of the mirrored planes' weights, preconditioned by the one-eps solve
        W = self.w if self.neu else 1.0
        x = torch.zeros_like(b)
        r, bb = b, b.norm()
        z = self.fast(r)
        p, rz = z, (W * r * z).sum()
        for _ in range(100):
            if r.norm() <= tol * bb:
                break
            q = self.apply(p)
            if self.neu:
                q[self.pin] = p[self.pin]
            a = rz / (W * p * q).sum()
            x, r = x + a * p, r - a * q
            z = self.fast(r)
            rz, old = (W * r * z).sum(), rz
            p = z + (rz / old) * p
        return x


def _exact_loop(c, seed):
    inp = _inputs(c, seed)
    sim = _Sim(c, inp)
    Ez, _ = _schedule(c, inp["Emax"])
    K, P = sim.params(sim.m8), inp["P"]
    phi, rows = torch.zeros_like(P[0]), []
    for e in Ez:
        P, m, q = sim.step(P, phi, float(e), K)
        rows.append(sim.rows(P, m, q))
        phi = sim.solve(sim.rhs(P))
    return {"P": P.reshape(6, -1), "phi": phi.reshape(-1), "rows": torch.stack(rows), "n": None}


def exact(case, seed):
    kind = case["kind"]
    if kind == "loop":
        return _exact_loop(case, seed)
    if kind == "batch":
        return [_exact_loop(c, seed * 1000 + i) for i, c in enumerate(_batch_films(case))]
    c = dict(case)
    if kind == "depol":
        c.update(init="random")
        inp = _inputs(c, seed)
        sim = _Sim(c, inp)
        phi = sim.solve(sim.rhs(inp["P"]))
        return {"phi_E": torch.stack([phi.reshape(-1)] + [-e.reshape(-1) for e in sim.field(phi)])}
    c.update(init="pz", amp=4.0, period=4000)
    inp = _inputs(c, seed)
    sim = _Sim(c, inp)
    Ez, _ = _schedule(c, inp["Emax"])
    m8 = sim.m8.clone().requires_grad_(True)
    K, P = sim.params(m8), inp["P"]
    phi, means = torch.zeros_like(P[0]), []
    for e in Ez:
        P, _, _ = sim.step(P, phi, float(e), K)
        means.append(P[2].mean())
        phi = sim.solve(sim.rhs(P))
    loss = ((torch.stack(means) - torch.from_numpy(_target(c["steps"])).to(DEV)) ** 2).mean()
    loss.backward()
    g = m8.grad[:, [0, 1, 2, 3, 5]]
    return {"loss": loss.detach().reshape(1), "grad": g}
