"""The direct solve of CMSL_FP32_REFINED films with sides that are not 2^a 3^b
(chirp transforms): chosen by CMSL_INNER_AUTO from 1024 columns on and up to
sides of 2048, refused when asked for by name as before.  Against the FP64
oracle solved to ||r|| <= 1e-12 ||b|| with the tolerances of the other
FP32_REFINED tests (P within 2e-5 of max |P|, phi 1e-4, rows 1e-5), and
against the PCG on the same film."""
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


def _film(shape, seed, eps=None, zbc=oracle.DIRICHLET):
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


# both sides chirp, one side a power of two, one 2^a 3^b, sides below a radix,
# the longest chirp transforms (2047, 2048 - 1 through 4096 values)
@pytest.mark.parametrize("shape", [(41, 25, 3), (64, 35, 4), (50, 32, 5), (55, 48, 6), (36, 130, 4), (257, 5, 5),
                                   (5, 515, 4), (2047, 3, 3), (7, 1999, 3)])
@pytest.mark.parametrize("eps", [30.0, None])                  # one permittivity; 40 / 30 / 15
@pytest.mark.parametrize("zbc", [oracle.DIRICHLET, oracle.NEUMANN])
def test_chirp_run_vs_oracle(gpu, shape, eps, zbc):
    f, P = _film(shape, sum(shape), eps, zbc)
    n = 6
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


@pytest.mark.parametrize("lines", ["1", "3", "8"])             # lines per transform block: remainders too
def test_chirp_lines_per_block(gpu, lines, monkeypatch):
    monkeypatch.setenv("CMSL_SPEC_RB", lines)
    f, P = _film((45, 77, 9), 3, 30.0)
    Ez = np.linspace(0.0, 0.3, 4)
    Pw, _, phiw, _, _, rc = oracle.load().run(f, P, np.zeros(f.N), Ez)
    assert rc == 0
    with gpu.Film.from_oracle_film(f, precision=gpu.FP32_REFINED, **KW) as g:
        g.set_state(P)
        g.run(Ez)
        _check(*g.get_state(), Pw, phiw)


def test_chirp_batch(gpu):
    """Films of every kind of length together, each against its oracle run."""
    films = [_film(s, 20 + i, 30.0) for i, s in enumerate([(35, 44, 5), (32, 16, 7), (24, 27, 4), (96, 11, 6)])]
    Ez = np.stack([np.linspace(0.0, 0.1 * (i + 1), 5) for i in range(len(films))])
    with gpu.Batch.from_oracle_films([f for f, _ in films], precision=gpu.FP32_REFINED, **KW) as b:
        assert b.inner_solver == gpu.INNER_DIRECT
        for i, (_, P) in enumerate(films):
            b.set_state(i, P)
        assert (b.run(Ez) == 0).all()
        for i, (f, P) in enumerate(films):
            Pw, _, phiw, _, _, rc = oracle.load().run(f, P, np.zeros(f.N), Ez[i])
            assert rc == 0
            _check(*b.get_state(i), Pw, phiw)


def test_chirp_selection(gpu):
    kw = dict(precision=gpu.FP32_REFINED)
    f, _ = _film((35, 30, 6), 4, 30.0)
    with gpu.Film.from_oracle_film(f, **kw) as g:
        assert g.inner_solver == gpu.INNER_DIRECT
    with pytest.raises(gpu.CmslError):                         # by name: refused as before
        gpu.Film.from_oracle_film(f, inner_solver=gpu.INNER_DIRECT, **kw)
    with gpu.Film.from_oracle_film(f, inner_solver=gpu.INNER_PCG, **kw) as g:
        assert g.inner_solver == gpu.INNER_PCG
    for shape in [(31, 33, 4), (2049, 3, 3)]:                  # 1023 columns; a side above 2048
        f, _ = _film(shape, 4, 30.0)
        with gpu.Film.from_oracle_film(f, **kw) as g:
            assert g.inner_solver == gpu.INNER_PCG
    mats = MATS_DEFAULT.copy()
    mats[:, 7] = [300.0, 30.0, 15.0]                           # ratio 20: the PCG as for 2^a 3^b sides
    f, _ = random_film(35, 30, 6, seed=5, mats=mats)
    with gpu.Film.from_oracle_film(f, **kw) as g:
        assert g.inner_solver == gpu.INNER_PCG


def test_chirp_selection_thin_films_of_several_eps(gpu):
    """Thin films of many columns and several permittivities keep the PCG,
    which takes few iterations there; alone or beside another ragged film."""
    def solver(shape, eps, **kw):
        mats = MATS_DEFAULT.copy()
        mats[:, 7] = eps
        f, _ = random_film(*shape, seed=4, n_grains=6, fracs=(0.4, 0.4, 0.2), mats=mats, **kw)
        f.grain_mat[:3] = [0, 1, 2]
        return f
    PCG, DIRECT = gpu.INNER_PCG, gpu.INNER_DIRECT
    deck, near = [50.0, 30.0, 15.0], [50.0, 30.0, 30.0]                    # ratios 10/3 and 5/3
    for shape, eps, want in [((130, 131, 4), deck, PCG), ((130, 131, 8), deck, PCG), ((130, 131, 9), deck, DIRECT),
                             ((130, 131, 5), near, PCG), ((130, 131, 6), near, DIRECT), ((130, 131, 4), 30.0, DIRECT),
                             ((130, 126, 4), deck, DIRECT), ((128, 128, 4), deck, DIRECT)]:
        with gpu.Film.from_oracle_film(solver(shape, eps), precision=gpu.FP32_REFINED) as g:
            assert g.inner_solver == want, (shape, eps)
    with gpu.Film.from_oracle_film(solver((130, 131, 4), deck, zbc=oracle.NEUMANN), precision=gpu.FP32_REFINED) as g:
        assert g.inner_solver == DIRECT
    with gpu.Batch.from_oracle_films([solver((130, 131, 4), deck), solver((35, 44, 5), 30.0)],
                                     precision=gpu.FP32_REFINED) as b:
        assert b.inner_solver == PCG
