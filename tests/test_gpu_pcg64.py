"""The persistent FP64 PCG (pcg64.cuh) against the oracle's PCG of the same
algorithm and stop test: both forms (vectors resident in registers, and
streaming through memory, CMSL_P64_STREAM=1) at the edges of their units --
x tiles of 32 (whole, one over, one column), rows groups of 1, 2 and 4 with
remainders, z chunks with remainders, periodic sides shorter than a halo --
with both z boundaries and stop tests.  Same iteration count to one and the
potential to 1e-10 of its maximum, the tolerance of the FP64 PCG elsewhere
(only the order and the rounding of sums differ)."""
import os

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


@pytest.mark.parametrize("zbc", [oracle.DIRICHLET, oracle.NEUMANN])
@pytest.mark.parametrize("form", ["resident", "streaming"])
@pytest.mark.parametrize("shape", [(1, 1, 3), (3, 2, 4), (31, 5, 3), (32, 7, 5), (33, 4, 6), (64, 3, 17), (65, 33, 9),
                                   (96, 50, 21), (40, 130, 10)])
def test_pcg64_solve_vs_oracle(gpu, shape, form, zbc, monkeypatch):
    monkeypatch.setenv("CMSL_P64_STREAM", "1" if form == "streaming" else "0")
    f, P = random_film(*shape, seed=sum(shape), zbc=zbc, eps_0_nd=3.0, layered=shape[2] >= 4,
                       n_grains=max(2, shape[0] * shape[1] // 24))
    if zbc == oracle.NEUMANN and shape[0] * shape[1] * shape[2] > 20000:
        pytest.skip("the pinned operator's thousands of iterations amplify the rounding of sums beyond the tolerance")
    if sum(shape) % 2:
        f.tol_abs, f.tol_rel = 1e-10, 1e-8
    else:
        f.crit, f.tol_rel = oracle.CRIT_RELRES, 1e-9
    f.max_iter = 4000
    phi0 = np.random.default_rng(1).normal(size=f.N) * 1e-3     # warm start, also on the identity rows
    want, _, _, info = oracle.load().depol_field(f, P[:3], phi0)
    with gpu.Film.from_oracle_film(f) as g:
        g.set_state(P, phi0)
        res = g.depol()
        _, phi = g.get_state()
    if info["status"] or info["iters"] == f.max_iter:
        return                  # no solve: a start on the identity rows makes the 3-cell film's system non-symmetric
    assert res["status"] == 0
    assert abs(res["iters"] - info["iters"]) <= 1
    if res["iters"] == info["iters"]:
        assert np.abs(phi - want).max() <= 1e-10 * np.abs(want).max()
    else:                                                       # one iteration apart: the stop test's own accuracy
        assert np.abs(phi - want).max() <= 1e-6 * np.abs(want).max()


def test_pcg64_film_beyond_the_resident_form(gpu):
    """A film of more units than warps takes the streaming form by itself (z
    chunks and rows as its plan picks them)."""
    mats = MATS_DEFAULT.copy()
    mats[:, 7] = 30.0
    f, P = random_film(100, 96, 60, seed=9, eps_0_nd=3.0, mats=mats)
    f.crit, f.tol_rel, f.max_iter = oracle.CRIT_RELRES, 1e-9, 4000
    want, _, _, info = oracle.load().depol_field(f, P[:3], np.zeros(f.N))
    with gpu.Film.from_oracle_film(f) as g:
        g.set_state(P)
        res = g.depol()
        _, phi = g.get_state()
    assert res["status"] == 0 and abs(res["iters"] - info["iters"]) <= 1
    assert np.abs(phi - want).max() <= (1e-10 if res["iters"] == info["iters"] else 1e-6) * np.abs(want).max()


def test_pcg64_iteration_cap_and_two_kernel_form(gpu, monkeypatch):
    """A solve that ends on its iteration cap, and the two-kernel loop
    (CMSL_PCG_TWO_KERNEL=1), give the same iterate."""
    f, P = random_film(48, 20, 8, seed=5, eps_0_nd=3.0)
    f.crit, f.tol_rel, f.max_iter = oracle.CRIT_RELRES, 1e-12, 7
    out = []
    for two in ("0", "1"):
        monkeypatch.setenv("CMSL_PCG_TWO_KERNEL", two)
        with gpu.Film.from_oracle_film(f) as g:
            g.set_state(P)
            assert g.depol()["iters"] == 7
            out.append(g.get_state()[1])
    assert np.abs(out[0] - out[1]).max() <= 1e-12 * np.abs(out[1]).max()


def test_pcg64_wait_timeout_is_reported(gpu):
    """A block that never adds its sums (held back on the host at creation,
    with short waits): every wait runs out, the kernel returns, the run
    reports CMSL_ERR_CUDA and the context stays usable."""
    f, P = random_film(64, 32, 8, seed=71, eps_0_nd=3.0, p_scale=0.2)
    keys = {"CMSL_PCG_HOLD_BLOCK": "1", "CMSL_PCG_SPIN_LIMIT": "2000"}
    old = {k: os.environ.get(k) for k in keys}
    os.environ.update(keys)
    try:
        g = gpu.Film.from_oracle_film(f)
    finally:
        for k, v in old.items():
            os.environ.pop(k) if v is None else os.environ.__setitem__(k, v)
    try:
        g.set_state(P)
        with pytest.raises(gpu.CmslError) as e:
            g.run(np.full(2, 0.1))
        assert e.value.status == 2 and "barrier timed out" in str(e.value)
    finally:
        g.close()
    with gpu.Film.from_oracle_film(f) as h:
        h.set_state(P)
        h.run(np.full(2, 0.1))
        assert all(np.isfinite(p).all() for p in h.get_state()[0])


@pytest.mark.parametrize("form", ["resident", "streaming"])
def test_pcg64_wait_timeout_ends_single_calls(gpu, form, monkeypatch):
    """The calls that solve without a run -- depol, depol on device arrays, the
    loop gradient -- end on such a wait with CMSL_ERR_CUDA too, not with an
    unfinished potential; the wait is reported once."""
    import ctypes as C

    import torch
    from cmsl_gb300._lib import lib
    f, P = random_film(64, 32, 8, seed=71, eps_0_nd=3.0, p_scale=0.2)
    monkeypatch.setenv("CMSL_P64_STREAM", "1" if form == "streaming" else "0")
    monkeypatch.setenv("CMSL_PCG_HOLD_BLOCK", "1")
    monkeypatch.setenv("CMSL_PCG_SPIN_LIMIT", "2000")
    with gpu.Film.from_oracle_film(f) as g:
        g.set_state(P)
        with pytest.raises(gpu.CmslError) as e:
            g.depol()
        assert e.value.status == 2 and "barrier timed out" in str(e.value)
        assert lib().cmsl_film_sync(g._h) == 0

        t = [torch.from_numpy(p).cuda() for p in P[:3]] + [torch.zeros(f.N, dtype=torch.float64, device="cuda") for _ in range(4)]
        it, st = np.zeros(2, np.int32), np.zeros(1, np.int32)
        ip = C.POINTER(C.c_int32)
        assert lib().cmsl_film_depol_device(g._h, *[C.c_void_p(v.data_ptr()) for v in t], None, it.ctypes.data_as(ip),
                                            st.ctypes.data_as(ip)) == 2
        assert st[0] == 4

        g.set_state(P)
        with pytest.raises(gpu.CmslError) as e:
            g.loop_gradient(np.full(2, 0.1), np.arange(2, dtype=np.int32), np.zeros(2), 2)
        assert e.value.status == 2 and "barrier timed out" in str(e.value)


@pytest.mark.parametrize("form", ["resident", "streaming"])
@pytest.mark.parametrize("k", [-490, -470, -300, 400, 500])
def test_pcg64_over_the_exponent_range(gpu, form, k, monkeypatch):
    """P scaled by 2^k scales the solve exactly: the sums and their quotients
    hold down to subnormal r.z (2^k = 2^-490: 2^-977 at the start, 2^-1037 at
    the end, with 37 bits left) and up to 2^1003."""
    monkeypatch.setenv("CMSL_P64_STREAM", "1" if form == "streaming" else "0")
    f, P = random_film(64, 32, 8, seed=72, eps_0_nd=3.0)
    f.crit, f.tol_rel, f.max_iter = oracle.CRIT_RELRES, 1e-9, 4000
    out = []
    for s in (1.0, 2.0 ** k):
        with gpu.Film.from_oracle_film(f) as g:
            g.set_state([p * s for p in P])
            res = g.depol()
            assert res["status"] == 0
            out.append((res["iters"], g.get_state()[1] / s))
    assert out[0][0] == out[1][0]
    assert np.abs(out[0][1] - out[1][1]).max() <= 1e-10 * np.abs(out[0][1]).max()


@pytest.mark.parametrize("reps", [4, 40])
def test_pcg64_timing_leaves_steps_and_p(gpu, reps):
    """Kernel timing and tuning advance no step: P, the steps done (row column
    10) and the log of the last run stay, also for more repetitions than the
    run had steps."""
    f, P = random_film(48, 20, 8, seed=6, eps_0_nd=3.0)
    with gpu.Film.from_oracle_film(f) as g:
        g.set_state(P)
        g.run(np.full(3, 0.1), np.arange(3, dtype=np.int32))
        before, log = g.get_state()[0], g.iters()
        g.time_kernels(reps=reps)
        g.autotune()
        assert all(np.array_equal(a, b) for a, b in zip(before, g.get_state()[0]))
        assert all(np.array_equal(a, b) for a, b in zip(log, g.iters()))
        g.run(np.full(1, 0.1), np.zeros(1, np.int32))
        assert g.rows()[0, 10] == 4


def test_pcg64_film_without_room_for_its_vectors(gpu):
    """A film that fits the memory but for the persistent PCG's two vectors (12
    bytes a cell of 168) takes the two-kernel loop and solves as before."""
    import torch
    f, P = random_film(256, 256, 128, seed=8, n_grains=8, eps_0_nd=3.0)
    f.crit, f.tol_rel, f.max_iter = oracle.CRIT_RELRES, 1e-6, 40
    with gpu.Film.from_oracle_film(f) as g:
        need = g.device_bytes()
        g.set_state(P)
        want, phi = g.depol(), g.get_state()[1]
    torch.cuda.empty_cache()
    free = torch.cuda.mem_get_info()[0]
    hog = torch.empty(free - need + 6 * f.N, dtype=torch.uint8, device="cuda")
    try:
        with gpu.Film.from_oracle_film(f) as g:
            assert g.device_bytes() < need - 11 * f.N
            g.set_state(P)
            res, got = g.depol(), g.get_state()[1]
    finally:
        del hog
        torch.cuda.empty_cache()
    assert res == want and np.abs(got - phi).max() <= 1e-10 * np.abs(phi).max()


@pytest.mark.parametrize("form", ["resident", "streaming"])
@pytest.mark.parametrize("seed", [9, 27, 32, 35, 38])
def test_pcg64_sums_far_above_the_last_one(gpu, form, seed, monkeypatch):
    """Permittivities 1e8 apart: r.z grows by 2^20 and more within an iteration,
    beyond the units its fixed-point sum starts with."""
    monkeypatch.setenv("CMSL_P64_STREAM", "1" if form == "streaming" else "0")
    rng = np.random.default_rng(seed)
    mats = MATS_DEFAULT.copy()
    mats[:, 7] = [1e8, 30.0, 1.0]
    f, _ = random_film(1, 1, 20, seed=1, eps_0_nd=3.0, mats=mats)
    mat = rng.integers(0, 3, 20)
    f.omega, f.grain_mat = np.arange(20, dtype=np.int32), mat.astype(np.int32)
    f.TR = np.tile(np.eye(3).reshape(-1), 20)
    f.is_interface = np.zeros(20, np.int32)
    P = list(rng.uniform(-0.2, 0.2, (3, 20))) + [np.zeros(20)] * 3
    f.crit, f.tol_rel, f.max_iter = oracle.CRIT_RELRES, 1e-9, 4000
    want, _, _, info = oracle.load().depol_field(f, P[:3], np.zeros(20))
    assert info["status"] == 0 and info["iters"] < 200
    with gpu.Film.from_oracle_film(f) as g:
        g.set_state(P)
        res = g.depol()
        phi = g.get_state()[1]
    # the PCG of a system of condition 1e8 leaves its iterates to rounding: only the solution is compared
    assert res["status"] == 0 and res["iters"] < 400
    r = -oracle.load().divergence(f, *P[:3])
    r[[0, -1]] = 0.0
    b = np.linalg.norm(r)
    assert np.linalg.norm(r - oracle.load().apply_A(f, phi)) <= 1e-7 * b
