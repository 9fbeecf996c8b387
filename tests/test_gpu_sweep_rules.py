"""Which kernel a call gets, what it may allocate, and the order its inputs arrive in.

Tolerance against the CPU oracle: 1e-9 relative with a 1e-12 absolute floor, the FP64
mode's bound (tests/test_gpu_parity.py).
"""
import numpy as np
import pytest

from negftrans_b200.negf import GreensFunction_tri_solver

pytestmark = pytest.mark.gpu
RTOL, ATOL = 1e-9, 1e-12


def random_blocks(N, Nz, seed):
    rng = np.random.default_rng(seed)
    D = rng.standard_normal((N, N, Nz)) + 1j * rng.standard_normal((N, N, Nz))
    D[np.arange(N), np.arange(N)] += 4.0 * np.sqrt(N)
    return np.asfortranarray(D)


@pytest.mark.parametrize("key", ["DFL", "F", "L"])
def test_tri_solve_waits_for_its_blocks(oracle, key):
    """27 MB of pageable blocks, other ones at each call; the right sweep starts at the copy's last bytes."""
    for seed in range(3):
        D = random_blocks(24, 3000, seed)
        ref, _ = oracle.tri_solver(D, key)
        got, info = GreensFunction_tri_solver(D, key)
        assert info == 0
        for k in key:
            assert np.max(np.abs(got[k] - ref[k])) <= RTOL * np.max(np.abs(ref[k]))
