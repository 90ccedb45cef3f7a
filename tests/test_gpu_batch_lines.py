"""Batches whose films together give the transform blocks many lines: eight rows
a block, in films whose own rows are no multiple of eight (27 rows of 2 packed
planes, 35 of 3, 5 of 2).  Each film against its solo run: the same transforms
and passes, so the fields agree to FP32 rounding over the steps (1e-6 of max |P|
and of max |phi|; an increment is below 1e-1 of P and rounds at 6e-8)."""
import numpy as np
import pytest

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


def test_batch_rows_per_block(gpu):
    mats = MATS_DEFAULT.copy()
    mats[:, 7] = 30.0
    shapes = [(64, 64, 16)] * 8 + [(24, 27, 5), (48, 35, 8), (256, 5, 6), (96, 64, 12)]
    films = [random_film(*s, seed=40 + i, eps_0_nd=3.0, del_t=5e-4, p_scale=0.2, mats=mats)
             for i, s in enumerate(shapes)]
    kw = dict(precision=gpu.FP32_REFINED, refine_tol=1e-8)
    Ez = np.stack([np.linspace(0.0, 0.02 * (i + 1), 4) for i in range(len(films))])
    with gpu.Batch.from_oracle_films([f for f, _ in films], **kw) as b:
        assert b.inner_solver == gpu.INNER_DIRECT
        for i, (_, P) in enumerate(films):
            b.set_state(i, P)
        assert (b.run(Ez) == 0).all()
        got = [b.get_state(i) for i in range(len(films))]
    for i, (f, P) in enumerate(films):
        with gpu.Film.from_oracle_film(f, **kw) as g:
            g.set_state(P)
            g.run(Ez[i])
            Pw, phiw = g.get_state()
        for a, w in zip(got[i][0], Pw):
            assert np.abs(a - w).max() <= 1e-6 * np.abs(w).max()
        assert np.abs(got[i][1] - phiw).max() <= 1e-6 * np.abs(phiw).max()
