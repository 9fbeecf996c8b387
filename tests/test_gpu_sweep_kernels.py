"""The on-chip sweep kernels at the edges of their layouts, against the CPU oracle.

Tolerance: 1e-9 relative with a 1e-12 absolute floor, the FP64 mode's bound
(tests/test_gpu_parity.py); set before the first run.
"""
import numpy as np
import pytest

from negftrans_b200 import workloads as W
from negftrans_b200 import prepare as P
from negftrans_b200.negf import Engine, GreensFunction_tri_solver, transmission_batch

pytestmark = pytest.mark.gpu
RTOL, ATOL = 1e-9, 1e-12


def cut_problem(oracle, N, nz, nk=1, grid=32, seed=1000):
    """The first N plane waves of the smallest circular basis that has N of them."""
    V = W.MSTAR * W.qpc_potential(grid, grid, nz, 100.0, nz * 1.0, 0.050, 15.0, max(nz / 6.0, 1.0), disorder=0.002,
                                  seed=seed)
    pr = P.prepare(W._deck(nz * 10.0, (N + 12) * 4.9e-5, 30.0, 16, nk=nk), V)
    assert pr.N >= N
    args = (np.ascontiguousarray(pr.nx[:N]), np.ascontiguousarray(pr.ny[:N])) + pr.engine_args()[2:]
    return args, oracle.Problem(*args), pr


# the register kernels hold 24, 48 and 72 plane waves; rows come in 32s
@pytest.mark.parametrize("N", [1, 2, 23, 24, 25, 33, 47, 48, 49, 64, 65, 71, 72, 73])
def test_small_bases(oracle, N):
    args, op, pr = cut_problem(oracle, N, nz=3, nk=2)
    kin = 0.5 * ((2 * np.pi * pr.nx[:N] / pr.atomic.LX) ** 2 + (2 * np.pi * pr.ny[:N] / pr.atomic.LY) ** 2)
    # no open channel, a few, about half, and every one of them
    E = np.array([-1e-6, 1e-5, 0.5 * kin.max() + 1e-5, 4.0 * kin.max() + 1e-4])
    ref, _ = oracle.transmission_jobs(op, E, nthreads=4)
    with Engine(*args) as eng:
        tau, info = eng.transmission(E)
        again, _ = eng.transmission(E)
    assert info == 0
    np.testing.assert_allclose(tau, ref, rtol=RTOL, atol=ATOL)
    assert (tau == again).all()


def test_batch_over_every_small_kernel(oracle):
    """One batch over problems of all three register kernels and the larger variants."""
    probs = [cut_problem(oracle, N, nz, nk=1) for N, nz in ((20, 4), (48, 2), (70, 5), (90, 3), (24, 6))]
    E = P.transmission_energies(probs[0][2].atomic, 16)[1::5]
    engines = [Engine(*p[0]) for p in probs]
    try:
        tau, info, stats = transmission_batch(engines, E)
    finally:
        for e in engines:
            e.close()
    assert info == 0 and stats.n_jobs == len(E) * len(probs)
    for p, t in zip(probs, tau):
        ref, _ = oracle.transmission_jobs(p[1], E, nthreads=4)
        np.testing.assert_allclose(t, ref, rtol=RTOL, atol=ATOL)


# the register slab kernels: tiles of 8, warps' columns of 12, rows of 32
@pytest.mark.parametrize("N,Nz", [(1, 3), (2, 2), (8, 4), (23, 2), (24, 5), (25, 3), (47, 2), (48, 4), (49, 3), (65, 3),
                                  (71, 2), (72, 5), (73, 3)])
def test_small_tri_solves(oracle, N, Nz):
    rng = np.random.default_rng(100 * N + Nz)
    D = rng.standard_normal((N, N, Nz)) + 1j * rng.standard_normal((N, N, Nz))
    D[np.arange(N), np.arange(N)] += 4.0 * np.sqrt(N)
    D[0, 0, 0] = 0.0  # the first column's natural pivot is no pivot
    D = np.asfortranarray(D)
    ref, rinfo = oracle.tri_solver(D, "DFL")
    got, info = GreensFunction_tri_solver(D, "DFL")
    assert info == rinfo
    if N == 1:  # the left sweep's first block is singular: reported, not trusted
        assert info == 1
        return
    assert info == 0
    for key in "DFL":
        scale = np.max(np.abs(ref[key]))
        assert np.max(np.abs(got[key] - ref[key])) <= RTOL * scale
        only, _ = GreensFunction_tri_solver(D, key)  # alone, the other planes' passes left out
        assert np.max(np.abs(only[key] - ref[key])) <= RTOL * scale


@pytest.mark.parametrize("N,nk", [(20, 2), (48, 1), (69, 1), (72, 1)])
@pytest.mark.parametrize("bias", [1e-5, -1e-5])
def test_small_biased_density(oracle, N, nk, bias):
    args, op, pr = cut_problem(oracle, N, nz=4, nk=nk)
    a = pr.atomic
    ref, _ = oracle.density_neq(op, 3, 4, pr.min_V, a.MU + bias, a.MU, a.GAP, a.TEMPERATURE)
    with Engine(*args) as eng:
        dm, info = eng.density_neq(3, 4, pr.min_V, a.MU + bias, a.MU, a.GAP, a.TEMPERATURE)
    assert info == 0
    assert np.max(np.abs(dm - ref)) <= RTOL * np.max(np.abs(ref))


def test_nan_and_singular_blocks_are_reported(oracle):
    """A NaN energy and a singular block end as an info, with the other jobs intact."""
    args, op, pr = cut_problem(oracle, 45, nz=3)
    E = P.transmission_energies(pr.atomic, 16)[2:5].copy()
    ref, _ = oracle.transmission_jobs(op, E, nthreads=4)
    bad = E.copy()
    bad[1] = np.nan
    with Engine(*args) as eng:
        tau, info = eng.transmission(bad)
        assert info > 0 and eng.last_stats.n_singular == 1 and eng.last_stats.first_bad_job == 1
    np.testing.assert_allclose(tau[[0, 2]], ref[[0, 2]], rtol=RTOL, atol=ATOL)
    for N in (5, 30, 60):
        D = np.asfortranarray(np.zeros((N, N, 3), np.complex128))
        D[np.arange(N), np.arange(N)] = 3.0
        D[:, N // 2, 2] = 0.0  # a zero column in the block the right sweep starts from
        _, info = GreensFunction_tri_solver(D, "DF")
        assert info == N // 2 + 1


# the panel kernel: panels of 32, row slots of 32 (basis and open channels), at most 320 rows; few jobs, so teams of
# eight CTAs (up to about 15 jobs), four (33) and two (74)
@pytest.mark.parametrize("N,nE", [(73, 4), (96, 20), (97, 4), (128, 40), (129, 4), (161, 4), (200, 20), (255, 4),
                                  (256, 40), (257, 4), (272, 4), (273, 4)])
def test_panel_teams(oracle, N, nE):
    args, op, pr = cut_problem(oracle, N, nz=3, grid=64)
    kin = 0.5 * ((2 * np.pi * pr.nx[:N] / pr.atomic.LX) ** 2 + (2 * np.pi * pr.ny[:N] / pr.atomic.LY) ** 2)
    # from no open channel to every one (which takes several passes where 2 N > 320)
    E = np.concatenate([[-1e-6, 1.1 * kin.max() + 1e-5], np.linspace(0.03, 0.6, nE - 2) * kin.max() + 1e-6])
    ref, _ = oracle.transmission_jobs(op, E, nthreads=8)
    with Engine(*args) as eng:
        tau, info = eng.transmission(E)
        again, _ = eng.transmission(E)
    assert info == 0
    np.testing.assert_allclose(tau, ref, rtol=RTOL, atol=ATOL)
    assert (tau == again).all()


def test_panel_batch_of_one_cta_per_job(oracle):
    """Bases on both sides of 256 in one batch of more jobs than clusters, and a NaN energy among them."""
    probs = [cut_problem(oracle, N, nz, grid=64) for N, nz in ((180, 3), (260, 2), (75, 5), (263, 3))]
    E = P.transmission_energies(probs[0][2].atomic, 30)[1:]
    bad = np.concatenate([E, [np.nan]])
    engines = [Engine(*p[0]) for p in probs]
    try:
        tau, info, stats = transmission_batch(engines, E)
        tau_bad, info_bad, stats_bad = transmission_batch(engines, bad)
    finally:
        for e in engines:
            e.close()
    assert info == 0 and stats.n_jobs == len(E) * len(probs)
    assert info_bad > 0 and stats_bad.n_singular == len(probs)
    for p, t, b in zip(probs, tau, tau_bad):
        ref, _ = oracle.transmission_jobs(p[1], E, nthreads=8)
        np.testing.assert_allclose(t, ref, rtol=RTOL, atol=ATOL)
        assert (b[:-1] == t).all()
