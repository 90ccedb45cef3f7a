"""The direct solve of CMSL_FP32_REFINED films with the Neumann z boundary
(every plane an unknown, mirrored end rows, one pinned cell): chosen by
CMSL_INNER_AUTO on 2^a 3^b sides, refused when asked for by name as before.
Against the FP64 oracle solved to ||r|| <= 1e-12 ||b|| with the tolerances of
the other FP32_REFINED tests (P within 2e-5 of max |P|, phi 1e-4, rows 1e-5),
and against the PCG on the same film."""
import numpy as np
import pytest

import oracle
from tests.films import MATS_DEFAULT, random_film

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def gpu():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from cmsl_gb300 import build
    build.build()
    import cmsl_gb300
    return cmsl_gb300


KW = dict(refine_tol=1e-8, inner_tol=1e-5)


def _film(shape, seed, eps=None, zbc=oracle.NEUMANN):
    mats = MATS_DEFAULT.copy()
    if eps is not None:
        mats[:, 7] = eps
    f, P = random_film(*shape, seed=seed, zbc=zbc, eps_0_nd=3.0, del_t=5e-4, p_scale=0.2, layered=shape[2] >= 4,
                       mats=mats)
    f.crit, f.tol_rel, f.max_iter = oracle.CRIT_RELRES, 1e-12, 20000
    return f, P


def _check(Pg, phig, Pw, phiw):
    for a, b in zip(Pg, Pw):
        assert np.abs(a - b).max() <= 2e-5 * np.abs(b).max()
    assert np.abs(phig - phiw).max() <= 1e-4 * np.abs(phiw).max()


@pytest.mark.parametrize("layout", ["columns", "rows"])
@pytest.mark.parametrize("eps", [30.0, None])                  # one permittivity; 40 / 30 / 15
@pytest.mark.parametrize("shape", [(8, 9, 3), (32, 8, 4), (27, 16, 5), (64, 16, 8), (48, 36, 7)])
def test_neumann_direct_run_vs_oracle(gpu, shape, eps, layout, monkeypatch):
    monkeypatch.setenv("CMSL_SPEC_COLS", "1" if layout == "columns" else "0")
    f, P = _film(shape, sum(shape), eps)
    n = 10
    Ez, rows = np.linspace(0.0, 0.3, n), np.arange(n, dtype=np.int32)
    Pw, _, phiw, statw, _, rc = oracle.load().run(f, P, np.zeros(f.N), Ez, rows)
    assert rc == 0
    with gpu.Film.from_oracle_film(f, precision=gpu.FP32_REFINED, **KW) as g:
        assert g.inner_solver == gpu.INNER_DIRECT
        g.set_state(P)
        g.run(Ez, rows)
        Pg, phig = g.get_state()
        rg = g.rows()
        it, _ = g.iters()
    _check(Pg, phig, Pw, phiw)
    assert np.abs(rg[:, :10] - statw[:, :10]).max() <= 1e-5
    if eps is not None:
        assert (it <= 3).all()                                 # exact solves: two or three passes a step
    with gpu.Film.from_oracle_film(f, precision=gpu.FP32_REFINED, inner_solver=gpu.INNER_PCG, **KW) as g:
        assert g.inner_solver == gpu.INNER_PCG
        g.set_state(P)
        g.run(Ez, rows)
        _check(*g.get_state(), Pw, phiw)


def test_neumann_direct_depol_and_no_graph(gpu, monkeypatch):
    """One solve from zero, and a run of plain launches."""
    f, P = _film((32, 24, 6), 3, 30.0)
    b = -oracle.load().divergence(f, *P[:3])
    b[f.nx // 2 + f.nx * (f.ny // 2 + f.ny * (f.nz // 2))] = 0.0
    with gpu.Film.from_oracle_film(f, precision=gpu.FP32_REFINED, refine_tol=1e-8) as g:
        g.set_state(P)
        assert g.depol()["status"] == 0
        Pg, phi = g.get_state()
    r = b - oracle.load().apply_A(f, phi)
    assert np.linalg.norm(r) <= 1e-7 * np.linalg.norm(b)       # b of the FP64 P; the film's P is FP32
    monkeypatch.setenv("CMSL_NO_GRAPH", "1")
    Ez = np.linspace(0.0, 0.2, 5)
    Pw, _, phiw, _, _, rc = oracle.load().run(f, P, np.zeros(f.N), Ez)
    assert rc == 0
    with gpu.Film.from_oracle_film(f, precision=gpu.FP32_REFINED, **KW) as g:
        g.set_state(P)
        g.run(Ez)
        _check(*g.get_state(), Pw, phiw)


def test_neumann_direct_in_a_batch(gpu):
    """Neumann and Dirichlet films in one batch of direct solves, several
    blocks for the larger one's pinned sum."""
    films = [_film((64, 48, 8), 5, 30.0), _film((32, 24, 6), 6, None, oracle.DIRICHLET), _film((16, 27, 5), 7, None)]
    n = 8
    Ez = np.stack([a * np.linspace(0.0, 0.3, n) for a in (1.0, -1.0, 0.5)])
    with gpu.Batch.from_oracle_films([f for f, _ in films], precision=gpu.FP32_REFINED, **KW) as b:
        assert b.inner_solver == gpu.INNER_DIRECT
        for i, (_, P) in enumerate(films):
            b.set_state(i, P)
        assert (b.run(Ez) == 0).all()
        for i, (f, P) in enumerate(films):
            Pw, _, phiw, _, _, rc = oracle.load().run(f, P, np.zeros(f.N), Ez[i])
            assert rc == 0
            _check(*b.get_state(i), Pw, phiw)


def test_neumann_direct_selection(gpu):
    f, _ = _film((32, 24, 6), 4, 30.0)
    with pytest.raises(gpu.CmslError):                         # by name: refused as before
        gpu.Film.from_oracle_film(f, precision=gpu.FP32_REFINED, inner_solver=gpu.INNER_DIRECT)
    f, _ = _film((33, 24, 6), 4, 30.0)                         # 33 = 3 x 11
    with gpu.Film.from_oracle_film(f, precision=gpu.FP32_REFINED) as g:
        assert g.inner_solver == gpu.INNER_PCG


def _smooth_film(shape):
    """One grain, P a wave of one period along x: a potential of the longest mode."""
    nx, ny, nz = shape
    f, _ = _film(shape, 3, 30.0)
    f.omega = np.zeros(f.N, np.int32)
    f.grain_mat, f.TR = np.ones(1, np.int32), np.asarray(f.TR).reshape(-1, 9)[:1].reshape(-1)
    f.is_interface = np.zeros(f.N, np.int32)
    x = np.tile(np.arange(nx), ny * nz)
    return f, [0.2 * np.sin(2 * np.pi * x / nx + q) for q in range(6)]


@pytest.mark.parametrize("shape", [(512, 32, 5), (32, 256, 4)])
def test_neumann_direct_long_modes(gpu, shape):
    """The FP32 check of a step sees modes of a whole side as they are: one more
    solve removes what the first one rounded off, and no further one runs on
    rounding of the check itself (three passes a step at most)."""
    f, P = _smooth_film(shape)
    f.del_t = 2e-3
    with gpu.Film.from_oracle_film(f, precision=gpu.FP32_REFINED, **KW) as g:
        assert g.inner_solver == gpu.INNER_DIRECT
        g.set_state(P)
        g.run(np.linspace(0.0, 0.3, 16))
        it, rf = g.iters()
        g.sync()
    assert (it <= 2).all() and (rf <= 3).all()


@pytest.mark.parametrize("tol", [1e-10, 1e-11, 1e-12])
@pytest.mark.parametrize("shape", [(64, 96, 5), (27, 48, 12)])
def test_neumann_direct_tight_target(gpu, shape, tol):
    """A target below what an update from 1e-4 ||b|| rounds off is met by b - A phi."""
    f, P = _film(shape, 9, 30.0)
    with gpu.Film.from_oracle_film(f, precision=gpu.FP32_REFINED, refine_tol=tol, max_refine=20) as g:
        g.set_state(P)
        assert g.depol()["status"] == 0
        Pg, phi = g.get_state()
    b = -oracle.load().divergence(f, Pg[0], Pg[1], Pg[2])
    r = b - oracle.load().apply_A(f, phi)
    pin = f.nx // 2 + f.nx * (f.ny // 2 + f.ny * (f.nz // 2))
    b[pin], r[pin] = 0.0, 0.0
    # a full pass forms r to 2^-48 of terms up to (96 / 2 pi)^2 of it: 8e-13 at worst, a tenth of that in the mean square
    assert np.linalg.norm(r) <= 1.1 * tol * np.linalg.norm(b)


@pytest.mark.parametrize("tol", [1e-12, 3e-13, 1e-13])
def test_neumann_direct_target_below_the_potentials_bits(gpu, tol):
    """Where the stored potential's 48 bits do not resolve the target, the solve
    says so (status 3) unless b - A phi meets it."""
    f, _ = _smooth_film((512, 64, 6))
    P = list(np.random.default_rng(2).uniform(-0.2, 0.2, (6, f.N)))
    with gpu.Film.from_oracle_film(f, precision=gpu.FP32_REFINED, refine_tol=tol, max_refine=8) as g:
        g.set_state(P)
        status = g.depol()["status"]
        Pg, phi = g.get_state()
    b = -oracle.load().divergence(f, Pg[0], Pg[1], Pg[2])
    r = b - oracle.load().apply_A(f, phi)
    pin = f.nx // 2 + f.nx * (f.ny // 2 + f.ny * (f.nz // 2))
    b[pin], r[pin] = 0.0, 0.0
    assert status == 3 or np.linalg.norm(r) <= 1.1 * tol * np.linalg.norm(b)
