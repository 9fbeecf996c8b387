"""The on-chip sweep kernels at the edges of their layouts, against the CPU oracle.

Tolerance: 1e-9 relative with a 1e-12 absolute floor, the FP64 mode's bound
(tests/test_gpu_parity.py); set before the first run.
"""
import numpy as np
import pytest

from negftrans_b200 import workloads as W
from negftrans_b200 import prepare as P
from negftrans_b200.negf import Engine, transmission_batch

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
