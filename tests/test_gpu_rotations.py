"""The FP32 TDGL step of films whose grain rotations are not orthonormal (the
general path: all nine values applied) and of orthonormal ones (the polar axis
only), against the FP64 oracle with the tolerances of the other FP32_REFINED
runs: P within 2e-5 of max |P|, rows within 1e-5."""
import dataclasses

import numpy as np
import pytest

import oracle
from tests.films import random_film

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


def _case(shape, general, seed):
    f, P = random_film(*shape, seed=seed, eps_0_nd=4.0, p_scale=0.2, layered=True)
    if general:
        r = np.random.default_rng(seed)
        f = dataclasses.replace(f, TR=np.asarray(f.TR) + 0.1 * r.normal(size=np.asarray(f.TR).shape))
    f.crit, f.tol_rel, f.max_iter = oracle.CRIT_RELRES, 1e-12, 20000
    return f, P


@pytest.mark.parametrize("general", [True, False])
@pytest.mark.parametrize("shape", [(64, 24, 6), (33, 17, 9), (27, 16, 5)])
def test_step_with_any_rotation(gpu, shape, general):
    f, P = _case(shape, general, sum(shape))
    n = 12
    Ez, rows = np.linspace(0.0, 0.3, n), np.arange(n, dtype=np.int32)
    Pw, _, _, statw, _, rc = oracle.load().run(f, P, np.zeros(f.N), Ez, rows)
    assert rc == 0
    with gpu.Film.from_oracle_film(f, precision=gpu.FP32_REFINED, refine_tol=1e-8, inner_tol=1e-5) as g:
        g.set_state(P)
        g.run(Ez, rows)
        Pg, _ = g.get_state()
        rg = g.rows()
        g.autotune()
        g.set_state(P)
        g.run(Ez, rows)
        Pt, _ = g.get_state()
    for a, t, b in zip(Pg, Pt, Pw):
        assert np.abs(a - b).max() <= 2e-5 * np.abs(b).max()
        assert np.abs(t - b).max() <= 2e-5 * np.abs(b).max()
    assert np.abs(rg[:, :10] - statw[:, :10]).max() <= 1e-5


def test_general_rotations_in_a_batch(gpu):
    films = [_case((32, 24, 6), True, 3), _case((64, 16, 5), False, 4)]
    n = 8
    Ez = np.stack([np.linspace(0.0, 0.3, n), np.linspace(0.0, -0.2, n)])
    with gpu.Batch.from_oracle_films([f for f, _ in films], precision=gpu.FP32_REFINED, refine_tol=1e-8,
                                     inner_tol=1e-5) as b:
        for i, (_, P) in enumerate(films):
            b.set_state(i, P)
        assert (b.run(Ez) == 0).all()
        for i, (f, P) in enumerate(films):
            Pw, _, _, _, _, rc = oracle.load().run(f, P, np.zeros(f.N), Ez[i])
            assert rc == 0
            for a, w in zip(b.get_state(i)[0], Pw):
                assert np.abs(a - w).max() <= 2e-5 * np.abs(w).max()


@pytest.mark.parametrize("setting", [("CMSL_TILE_Y", "4"), ("CMSL_TILE_Y", "16"), ("CMSL_STAGING", "11"), ("CMSL_DEFER", "0")])
@pytest.mark.parametrize("films", [1, 2])
def test_single_precision_rotations(gpu, setting, films, monkeypatch):
    """Rotations that passed through FP32 take the general path by every tile
    height, staging and form of the check that orthonormal ones have."""
    monkeypatch.setenv(*setting)
    if setting[0] == "CMSL_STAGING":
        monkeypatch.setenv("CMSL_DEFER", "0")                # the tensor-copy TDGL step
    fs = []
    for seed in range(films):
        f, P = _case((96, 24, 7), False, 5 + seed)        # a shape that no other test here tunes
        f = dataclasses.replace(f, TR=np.asarray(f.TR).astype(np.float32).astype(np.float64), mats=f.mats.copy())
        f.mats[:, 7] = 30.0
        f.crit, f.tol_rel, f.max_iter = oracle.CRIT_RELRES, 1e-12, 20000
        fs.append((f, P))
    Ez = np.linspace(0.0, 0.3, 10)
    kw = dict(precision=gpu.FP32_REFINED, refine_tol=1e-8, inner_tol=1e-5)
    if films == 1:
        with gpu.Film.from_oracle_film(fs[0][0], **kw) as g:
            cfg = g.tile_config()
            g.set_state(fs[0][1])
            g.run(Ez)
            got = [g.get_state()[0]]
    else:
        with gpu.Batch.from_oracle_films([f for f, _ in fs], **kw) as b:
            cfg = b.tile_config()
            for i, (_, P) in enumerate(fs):
                b.set_state(i, P)
            assert (b.run(np.stack([Ez] * films)) == 0).all()
            got = [b.get_state(i)[0] for i in range(films)]
    if setting[0] == "CMSL_TILE_Y":
        assert cfg["y"] == int(setting[1])
    if setting[0] == "CMSL_STAGING":
        assert cfg["tdgl_staging"] == cfg["residual_staging"] == "tensor copies"
    for (f, P), Pg in zip(fs, got):
        Pw, _, _, _, _, rc = oracle.load().run(f, P, np.zeros(f.N), Ez)
        assert rc == 0
        for a, w in zip(Pg, Pw):
            assert np.abs(a - w).max() <= 2e-5 * np.abs(w).max()
