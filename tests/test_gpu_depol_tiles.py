"""cmsl_film_depol on FP32_REFINED films of full 32 x 8 tiles, whose residual
passes may be staged by tensor copies: the solve reads the film's current P
(with one permittivity and with three), ||b - A phi|| <= 1.2e-8 ||b|| in
FP64."""
import numpy as np
import pytest

import oracle
from tests.films import MATS_DEFAULT, random_film

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("eps", [30.0, None])
@pytest.mark.parametrize("inner", ["direct", "pcg"])
def test_depol_reads_the_current_state(eps, inner):
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from cmsl_gb300 import build
    build.build()
    import cmsl_gb300 as cg
    mats = MATS_DEFAULT.copy()
    if eps is not None:
        mats[:, 7] = eps
    f, P = random_film(64, 24, 6, seed=9, eps_0_nd=4.0, mats=mats)
    orc = oracle.load()
    with cg.Film.from_oracle_film(f, precision=cg.FP32_REFINED, refine_tol=1e-8,
                                  inner_solver=cg.INNER_DIRECT if inner == "direct" else cg.INNER_PCG) as g:
        g.set_state(P)
        assert g.depol()["status"] == 0
        Pg, phi = g.get_state()
    b = -orc.divergence(f, *Pg[:3])
    k = np.repeat(np.arange(f.nz), f.nx * f.ny)
    b[(k == 0) | (k == f.nz - 1)] = 0.0
    assert np.linalg.norm(b - orc.apply_A(f, phi)) <= 1.2e-8 * np.linalg.norm(b)
