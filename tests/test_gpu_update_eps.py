"""FP32 update passes (r <- r - A dx) of films with several permittivities
under the direct solve: the potential they end on, against the FP64 operator.

A refinement ends on ||r|| <= 1e-8 ||b|| of the updated r.  An update rounds
A dx at 6e-8 of its six terms, which are (nz / pi) times the sum at most for
the smoothest mode: 6e-8 * 3 * 32 / pi < 2e-6 of ||r|| here, and the updates
start below 1e-4 ||b|| and shrink at least by 0.6 a pass (ratio 16), so the
true residual stays within 1e-8 + 2e-6 * 1e-4 / 0.4 = 1.05e-8."""
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


def _film(shape, ratio, seed, zbc=oracle.DIRICHLET):
    mats = MATS_DEFAULT.copy()
    mats[:, 7] = [15.0 * ratio, 15.0 * np.sqrt(ratio), 15.0]
    f, P = random_film(*shape, seed=seed, zbc=zbc, eps_0_nd=3.0, del_t=5e-4, p_scale=0.2, layered=shape[2] >= 4,
                       mats=mats)
    f.crit, f.tol_rel, f.max_iter = oracle.CRIT_RELRES, 1e-12, 20000
    return f, P


# tiles' remainders and sides below a tile, 2^a 3^b and chirp sides
@pytest.mark.parametrize("shape", [(8, 9, 3), (33, 32, 5), (64, 24, 12), (45, 41, 32)])
@pytest.mark.parametrize("ratio", [1.5, 3.3, 8.0, 15.9])
@pytest.mark.parametrize("zbc", [oracle.DIRICHLET, oracle.NEUMANN])
def test_update_residual(gpu, shape, ratio, zbc):
    f, P = _film(shape, ratio, sum(shape), zbc)
    orc = oracle.load()
    with gpu.Film.from_oracle_film(f, precision=gpu.FP32_REFINED, refine_tol=1e-8) as g:
        assert g.inner_solver == gpu.INNER_DIRECT
        g.set_state(P)
        res = g.depol()
        Pg, phi = g.get_state()
    assert res["status"] == 0
    b = -orc.divergence(f, Pg[0], Pg[1], Pg[2])
    k = np.repeat(np.arange(f.nz), f.nx * f.ny)
    if zbc == oracle.DIRICHLET:
        b[(k == 0) | (k == f.nz - 1)] = 0.0
        r = b - orc.apply_A(f, phi)
    else:
        r = b - orc.apply_A(f, phi)
        pin = f.nx // 2 + f.nx * (f.ny // 2 + (f.nz // 2) * f.ny)   # identity row, b = 0
        b[pin], r[pin] = 0.0, 0.0
    assert np.linalg.norm(r) <= 1.05e-8 * np.linalg.norm(b)


@pytest.mark.parametrize("ratio", [3.3, 15.9])
def test_update_run_vs_oracle(gpu, ratio):
    """Steps whose warm starts put the first updates right after the first pass."""
    f, P = _film((64, 48, 10), ratio, 7)
    Ez = np.linspace(0.0, 0.3, 12)
    Pw, _, phiw, _, _, rc = oracle.load().run(f, P, np.zeros(f.N), Ez)
    assert rc == 0
    with gpu.Film.from_oracle_film(f, precision=gpu.FP32_REFINED, refine_tol=1e-8, warm_start=2) as g:
        g.set_state(P)
        g.run(Ez)
        Pg, phig = g.get_state()
    for a, b in zip(Pg, Pw):
        assert np.abs(a - b).max() <= 2e-5 * np.abs(b).max()
    assert np.abs(phig - phiw).max() <= 1e-4 * np.abs(phiw).max()


# Targets below what updates from 1e-4 ||b|| on round off: convergence counts
# what the updates may have lost, and full double-float passes take over.  A
# full pass forms the residual to some 2^-48 of terms that exceed it by
# (nz / pi)^2 or (side / 2 pi)^2 <= 104, so to 4e-13 at worst and some 4e-14 in
# the mean square: within 5 % of the smallest target.
@pytest.mark.parametrize("tol", [1e-10, 1e-11, 1e-12])
@pytest.mark.parametrize("shape, ratio, zbc", [((64, 24, 12), 3.3, oracle.DIRICHLET), ((45, 41, 32), 15.9, oracle.DIRICHLET),
                                               ((48, 64, 10), 60.0, oracle.DIRICHLET), ((36, 32, 6), 3.3, oracle.NEUMANN),
                                               ((37, 41, 9), 15.9, oracle.NEUMANN)])
def test_update_tight_target(gpu, shape, ratio, zbc, tol):
    f, P = _film(shape, ratio, sum(shape), zbc)
    orc = oracle.load()
    inner = gpu.INNER_DIRECT if ratio > 16 else gpu.INNER_AUTO      # AUTO takes the PCG beyond 16
    with gpu.Film.from_oracle_film(f, precision=gpu.FP32_REFINED, refine_tol=tol, max_refine=60, inner_solver=inner) as g:
        assert g.inner_solver == gpu.INNER_DIRECT
        g.set_state(P)
        res = g.depol()
        Pg, phi = g.get_state()
    assert res["status"] == 0
    b = -orc.divergence(f, Pg[0], Pg[1], Pg[2])
    k = np.repeat(np.arange(f.nz), f.nx * f.ny)
    if zbc == oracle.DIRICHLET:
        b[(k == 0) | (k == f.nz - 1)] = 0.0
        r = b - orc.apply_A(f, phi)
    else:
        r = b - orc.apply_A(f, phi)
        pin = f.nx // 2 + f.nx * (f.ny // 2 + (f.nz // 2) * f.ny)
        b[pin], r[pin] = 0.0, 0.0
    assert np.linalg.norm(r) <= 1.05 * tol * np.linalg.norm(b)


@pytest.mark.parametrize("zbc", [oracle.DIRICHLET, oracle.NEUMANN])
def test_update_by_tensor_copies(gpu, zbc, monkeypatch):
    """Residual passes by tensor copies update r where the ring's do: the same
    arithmetic in the same order, so the same bits and pass counts."""
    f, P = _film((64, 24, 10), 3.3, 11, zbc)
    Ez = np.linspace(0.0, 0.3, 6)
    out = []
    for staging in ("00", "01"):
        monkeypatch.setenv("CMSL_STAGING", staging)
        with gpu.Film.from_oracle_film(f, precision=gpu.FP32_REFINED, refine_tol=1e-8) as g:
            assert g.tile_config()["residual_staging"] == ("cp.async ring", "tensor copies")[int(staging[1])]
            g.set_state(P)
            g.run(Ez)
            out.append((*g.get_state(), *g.iters()))
    for a, b in zip(out[0][0], out[1][0]):
        assert np.array_equal(a, b)
    for a, b in zip(out[0][1:], out[1][1:]):
        assert np.array_equal(a, b)
