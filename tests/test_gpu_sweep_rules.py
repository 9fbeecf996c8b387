"""Which kernel a call gets, what it may allocate, and the order its inputs arrive in.

Tolerance against the CPU oracle: 1e-9 relative with a 1e-12 absolute floor, the FP64
mode's bound (tests/test_gpu_parity.py).
"""
import numpy as np
import pytest

from negftrans_b200 import prepare as P
from negftrans_b200 import workloads as W
from negftrans_b200._lib import NEGF_ERR_UNSUPPORTED, NegfError
from negftrans_b200.negf import Engine, GreensFunction_tri_solver, transmission_batch

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


def diagonal_blocks_80_bits(D):
    """G_kk of math_kernel.f90:81-109 in 80-bit arithmetic (Gauss-Jordan, largest pivot of the column)."""
    def inverse(A):
        A, N = A.copy(), len(A)
        free, prow = np.ones(N, bool), np.zeros(N, int)
        for k in range(N):
            p = prow[k] = int(np.argmax(np.where(free, abs(A[:, k]), -1)))
            free[p] = False
            m = A[:, k].copy()
            row = A[p] / m[p]
            row[k] = 1 / m[p]
            A[:, k] = 0
            A -= m[:, None] * row
            A[p] = row
        out = np.empty_like(A)
        out[:, prow] = A[prow]
        return out

    N, _, Nz = D.shape
    D = D.astype(np.clongdouble)
    g = [None] * Nz
    for b in range(Nz - 1, -1, -1):
        g[b] = inverse(D[:, :, b] - (g[b + 1] if b < Nz - 1 else 0))
    out = [g[0]]
    for k in range(1, Nz):
        out.append(g[k] @ (np.eye(N) + out[-1] @ g[k]))
    return np.stack(out, 2)


# The limits lie between the means that an emulation of the kernel's arithmetic on the CPU gives over these eight
# problems, in units of 2^-53: 3.26, 4.40, 5.25 with the pivot row's 1 kept apart; 4.04, 5.50, 6.57 with it stored
# (which the listed bound of scaled rows, 3.93, 5.59, 6.79, is about as far off as).
@pytest.mark.parametrize("N,most", [(24, 3.6), (48, 4.95), (69, 5.9)])
def test_register_inverse_keeps_its_last_bits(N, most):
    err = []
    for seed in range(8):
        rng = np.random.default_rng(seed)
        D = 0.02 * (rng.standard_normal((N, N, 12)) + 1j * rng.standard_normal((N, N, 12)))
        D[np.arange(N), np.arange(N)] += 3.0 + rng.uniform(0, 1, (N, 12)) + 1j * rng.uniform(0, 1, (N, 12))
        got, info = GreensFunction_tri_solver(np.asfortranarray(D), "D")
        assert info == 0
        ref = diagonal_blocks_80_bits(D)
        err.append(float(np.sqrt(np.sum(abs(got["D"] - ref) ** 2) / np.sum(abs(ref) ** 2))) * 2.0 ** 53)
    assert np.mean(err) <= most


# N = 800, two blocks: 61 MB of blocks, plane and slab, 61 MB of workspace, and as a choice 20 and 61 MB more for the
# second pass beside the first
@pytest.mark.parametrize("free_mb", [260, 175, 135])
def test_tri_solve_in_little_memory(free_mb):
    import torch
    D = random_blocks(800, 2, 7)
    ref, info = GreensFunction_tri_solver(D, "DL")
    assert info == 0
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    fill = torch.empty(torch.cuda.mem_get_info()[0] - free_mb * 1000000, dtype=torch.uint8, device="cuda")
    try:
        got, info = GreensFunction_tri_solver(D, "DL")
    finally:
        del fill
        torch.cuda.empty_cache()
    assert info == 0
    for key in "DL":
        assert (got[key] == ref[key]).all()


def cut_problem(oracle, N, nz, nk=1, grid=64, seed=1000):
    """The first N plane waves of a larger circular basis; the largest kinetic energy of theirs."""
    V = W.MSTAR * W.qpc_potential(grid, grid, nz, 100.0, nz * 1.0, 0.050, 15.0, max(nz / 6.0, 1.0), disorder=0.002,
                                  seed=seed)
    pr = P.prepare(W._deck(nz * 10.0, (N + 12) * 4.9e-5, 30.0, 16, nk=nk), V)
    assert pr.N >= N
    args = (np.ascontiguousarray(pr.nx[:N]), np.ascontiguousarray(pr.ny[:N])) + pr.engine_args()[2:]
    kin = 0.5 * ((2 * np.pi * pr.nx[:N] / pr.atomic.LX) ** 2 + (2 * np.pi * pr.ny[:N] / pr.atomic.LY) ** 2)
    return args, oracle.Problem(*args), kin.max()


# a block of the panel kernel has 320 - N rows for channels: at and past that, few jobs and many, every entry
@pytest.mark.parametrize("N,nE,variant", [(240, 40, 0), (256, 74, 0), (257, 40, 1), (272, 150, 1)])
def test_many_open_channels_take_one_sweep(oracle, N, nE, variant):
    import torch
    args, op, kmax = cut_problem(oracle, N, nz=3)
    E = np.linspace(1.1, 1.2, nE) * kmax
    E[1] = np.nan
    check = [0, 2, nE - 1]
    ref, _ = oracle.transmission_jobs(op, E[check], nthreads=8)
    with Engine(*args) as eng:
        best = {}
        for v in (-1, variant):
            eng.set_variant(v)
            ms = []
            for _ in range(4):
                tau, info = eng.transmission(E)
                ms.append(eng.last_stats.device_ms)
                assert info > 0 and eng.last_stats.n_singular == 1 and eng.last_stats.first_bad_job == 1
                np.testing.assert_allclose(tau[check], ref, rtol=RTOL, atol=ATOL)
            best[v] = min(ms)
            if v < 0:
                dE = torch.tensor(E, device="cuda")
                dt = torch.zeros(nE, dtype=torch.float64, device="cuda")
                torch.cuda.synchronize()
                eng.transmission_device(dE.data_ptr(), nE, dt.data_ptr())
                torch.cuda.synchronize()
                assert (dt.cpu().numpy()[check] == tau[check]).all()
        eng.set_variant(-1)
        both, info, _ = transmission_batch([eng], E)
        np.testing.assert_allclose(both[0][check], ref, rtol=RTOL, atol=ATOL)
    # several sweeps per job take two to four times as long
    assert best[-1] <= 1.4 * best[variant]


# about as many channels as a block has room for, on both sides of it; one and two passes in the largest teams
@pytest.mark.parametrize("N,nE", [(200, 4), (221, 30), (260, 4), (272, 20)])
def test_open_channels_at_the_edge_of_the_block(oracle, N, nE):
    args, op, kmax = cut_problem(oracle, N, nz=2)
    kin = np.sort(0.5 * ((2 * np.pi * args[0] / args[3]) ** 2 + (2 * np.pi * args[1] / args[4]) ** 2))
    for passes in (1, 2):
        room = min(N, passes * (320 - N))
        for top in (0.5 * (kin[room - 2] + kin[room - 1]), kin[min(room, N - 1)] * (1 + 1e-9) + 1e-9):
            E = np.linspace(0.3, 1.0, nE) * top
            ref, _ = oracle.transmission_jobs(op, E, nthreads=8)
            with Engine(*args) as eng:
                tau, info = eng.transmission(E)
                both, _, _ = transmission_batch([eng], E)
            assert info == 0
            np.testing.assert_allclose(tau, ref, rtol=RTOL, atol=ATOL)
            np.testing.assert_allclose(both[0], ref, rtol=RTOL, atol=ATOL)


# bins of few and of many plane waves, on both sides of a batch of eight; an elongated basis; vectors held twice or more
@pytest.mark.parametrize("N,mx,my,twice", [(1, 0, 0, 0), (7, 1, 1, 0), (69, 5, 4, 0), (97, 40, 1, 0), (300, 9, 10, 0),
                                           (40, 4, 3, 5), (9, 0, 0, 0)])
def test_real_space_density(N, mx, my, twice):
    from negftrans_b200.grid import Greensfunction_PlanewaveToReal
    rng = np.random.default_rng(N)
    pos = [(x, y) for y in range(-my, my + 1) for x in range(-mx, mx + 1)]
    pick = np.sort(rng.choice(len(pos), min(N, len(pos)), replace=False))
    pick = np.concatenate([pick, rng.choice(pick, N - len(pick)), ])
    pick[:twice] = pick[-1]
    nx, ny = np.array([pos[i] for i in pick], np.int32).T
    Nx, Ny, nz = 2 * mx + 3, 2 * my + 2, 3
    G = np.asfortranarray(rng.standard_normal((N, N, nz)) + 1j * rng.standard_normal((N, N, nz)))
    ref = np.stack([Greensfunction_PlanewaveToReal(G[:, :, k], nx, ny, Nx, Ny) for k in range(nz)], 2)
    with Engine(nx, ny, np.zeros((4 * mx + 1, 4 * my + 1, nz), complex), 1.0, 1.0, 1.0, 0.0, 0.0, 1e-6,
                [[0, 0, 1]]) as eng:
        got = eng.dm_real(G, Nx, Ny, 1.0, 1.0, float(nz))
    # at most N^2 terms a point: sums of random signs, far inside N^2 eps
    assert np.max(np.abs(got - ref.imag)) <= 1e-12 * N


def test_real_space_density_of_the_longest_basis():
    """1000 plane waves over 4241 along x: tables of 199 KB and the index lists on top."""
    from negftrans_b200.grid import Greensfunction_PlanewaveToReal
    rng = np.random.default_rng(3)
    N, mx = 1000, 2120
    nx = np.sort(rng.choice(2 * mx + 1, N, replace=False)).astype(np.int32) - mx
    nx[0], nx[-1] = -mx, mx
    ny = np.zeros(N, np.int32)
    G = np.asfortranarray(rng.standard_normal((N, N, 2)) + 1j * rng.standard_normal((N, N, 2)))
    ref = Greensfunction_PlanewaveToReal(G, nx, ny, 2 * mx + 3, 1)
    with Engine(nx, ny, np.zeros((4 * mx + 1, 1, 2), complex), 1.0, 1.0, 1.0, 0.0, 0.0, 1e-6, [[0, 0, 1]]) as eng:
        got = eng.dm_real(G, 2 * mx + 3, 1, 1.0, 1.0, 2.0)
    assert np.max(np.abs(got - ref.imag)) <= 1e-12 * N


# the kernels of a batch run side by side: bases of every kernel, jobs above and below the number of slots
@pytest.mark.parametrize("nE", [3, 60])
def test_batch_of_every_kernel(oracle, nE):
    probs = [cut_problem(oracle, N, nz) for N, nz in ((20, 4), (40, 3), (72, 3), (150, 2), (256, 2), (260, 2), (290, 2))]
    E = np.linspace(0.05, 0.2, nE) * probs[3][2]
    check = slice(None) if nE < 10 else slice(0, nE, 19)
    bad = E.copy()
    bad[1] = np.nan
    engines = [Engine(*p[0]) for p in probs]
    try:
        tau, info, stats = transmission_batch(engines, E)
        tau_bad, info_bad, stats_bad = transmission_batch(engines, bad)
        turned, _, _ = transmission_batch(engines[::-1], E)
    finally:
        for e in engines:
            e.close()
    assert info == 0 and stats.n_jobs == nE * len(probs) and stats.n_singular == 0
    assert info_bad > 0 and stats_bad.n_singular == len(probs)
    assert (turned[::-1] == tau).all()
    keep = np.arange(nE) != 1
    for p, t, b in zip(probs, tau, tau_bad):
        ref, _ = oracle.transmission_jobs(p[1], E[check], nthreads=8)
        np.testing.assert_allclose(t[check], ref, rtol=RTOL, atol=ATOL)
        assert (b[keep] == t[keep]).all()


def test_one_wide_basis_does_not_slow_a_batch(oracle):
    """1800 sweeps of N = 221 fill the chip two to an SM; a base above 256 beside them leaves them there."""
    a = cut_problem(oracle, 221, 8)[0]
    w = cut_problem(oracle, 260, 2)[0]
    E = np.linspace(0.01, 0.2, 150) * 1e-4
    engines = [Engine(*a) for _ in range(12)] + [Engine(*w)]
    try:
        def ms(which):
            return min(transmission_batch(which, E)[2].device_ms for _ in range(3))
        # the 300 slices of N = 260 are 1.04 times the work; in panels those of N = 221 took 1.19 times as long
        assert ms(engines) <= 1.12 * ms(engines[:-1])
    finally:
        for e in engines:
            e.close()


# workspaces of 58 MB (N = 300) and 15 MB (N = 221): side by side, and one after the other where 66 MB are free
def test_batch_in_little_memory(oracle):
    import torch
    probs = [cut_problem(oracle, N, 2) for N in (300, 221)]
    E = np.linspace(0.05, 0.2, 10) * probs[0][2]
    engines = [Engine(*p[0]) for p in probs]
    other = [Engine(*p[0]) for p in probs]
    try:
        ref, _, _ = transmission_batch(engines, E)
        torch.cuda.synchronize()
        torch.cuda.empty_cache()
        fill = torch.empty(torch.cuda.mem_get_info()[0] - 66000000, dtype=torch.uint8, device="cuda")
        try:
            tau, info, _ = transmission_batch(other, E)
        finally:
            del fill
            torch.cuda.empty_cache()
    finally:
        for e in engines + other:
            e.close()
    assert info == 0 and (tau == ref).all()


@pytest.mark.parametrize("N", [257, 272])
def test_the_autotuner_times_the_default_kernel(oracle, N):
    args, op, kmax = cut_problem(oracle, N, nz=3)
    E = np.linspace(0.02, 0.12, 20) * kmax
    ref, _ = oracle.transmission_jobs(op, E[::7], nthreads=8)
    with Engine(*args) as eng:
        default, _ = eng.transmission(E)
        ms = min((eng.transmission(E), eng.last_stats.device_ms)[1] for _ in range(3))
        eng.set_variant(3)
        forced, _ = eng.transmission(E)
        assert (forced == default).all()
        np.testing.assert_allclose(forced[::7], ref, rtol=RTOL, atol=ATOL)
        v, rates = eng.autotune(E)
        assert rates[0] == 0 and (rates[1:] > 0).all() and rates[v] == rates.max()
        eng.transmission(E)
        # a tuned call is no slower than an untuned one: 16 x 2 x 1 takes 2.4 times as long here
        assert eng.last_stats.device_ms <= 1.2 * ms
    with Engine(*cut_problem(oracle, 273, nz=2)[0]) as eng, pytest.raises(NegfError) as exc:
        eng.set_variant(3)
    assert exc.value.code == NEGF_ERR_UNSUPPORTED


def sms():
    import torch
    return torch.cuda.get_device_properties(0).multi_processor_count


# above one job per two SMs: one CTA per SM (8 x 1 x 1), two (8 x 1 x 2), and more jobs than places; panels above 256
@pytest.mark.parametrize("N", [73, 96, 97, 129, 192, 193, 221, 255, 256, 257, 272])
def test_many_jobs_of_middle_bases(oracle, N):
    args, op, kmax = cut_problem(oracle, N, nz=2)
    with Engine(*args) as eng:
        for nE in (sms() // 2 + 1, sms() + 1, 2 * sms() + 3):
            E = np.concatenate([[-1e-6], np.linspace(0.01, 0.15, nE - 1) * kmax])
            check = [0, 1, nE // 2, nE - 2, nE - 1]
            ref, _ = oracle.transmission_jobs(op, E[check], nthreads=8)
            tau, info = eng.transmission(E)
            both, _, stats = transmission_batch([eng], E)
            assert info == 0 and stats.n_jobs == nE
            np.testing.assert_allclose(tau[check], ref, rtol=RTOL, atol=ATOL)
            assert (both[0] == tau).all()


# remainders of the 32-column panels and of the 32- and 64-row tiles
@pytest.mark.parametrize("N", [65, 97, 100, 191, 225, 256])
@pytest.mark.parametrize("variant", [0, 1, 2, 3])
def test_every_variant_beyond_one_panel(oracle, N, variant):
    args, op, kmax = cut_problem(oracle, N, nz=3)
    E = np.linspace(0.05, 1.2, 4) * kmax
    ref, _ = oracle.transmission_jobs(op, E, nthreads=8)
    with Engine(*args) as eng:
        eng.set_variant(variant)
        tau, info = eng.transmission(E)
    assert info == 0
    np.testing.assert_allclose(tau, ref, rtol=RTOL, atol=ATOL)


def test_batch_of_many_middle_bases(oracle):
    """More sweeps than places, all of 73 to 256 plane waves: two on an SM, taken from one counter."""
    probs = [cut_problem(oracle, N, nz) for N, nz in ((73, 3), (256, 2), (129, 2), (221, 2))]
    E = np.linspace(0.02, 0.3, sms()) * probs[0][2]
    engines = [Engine(*p[0]) for p in probs]
    try:
        tau, info, stats = transmission_batch(engines, E)
    finally:
        for e in engines:
            e.close()
    assert info == 0 and stats.n_jobs == 4 * len(E)
    for p, t in zip(probs, tau):
        ref, _ = oracle.transmission_jobs(p[1], E[::49], nthreads=8)
        np.testing.assert_allclose(t[::49], ref, rtol=RTOL, atol=ATOL)


def test_context_has_its_inputs_when_it_is_made(oracle):
    """7 MB of V table, another one at each context, used at once; the sweep starts at its last slice."""
    for seed in (1, 2, 3):
        args, op, kmax = cut_problem(oracle, 20, nz=1500, grid=32, seed=seed)
        E = np.array([4.0, 5.0]) * kmax
        ref, _ = oracle.transmission_jobs(op, E, nthreads=4)
        with Engine(*args) as eng:
            tau, info = eng.transmission(E)
        assert info == 0
        np.testing.assert_allclose(tau, ref, rtol=RTOL, atol=ATOL)


def test_contexts_in_two_threads(oracle):
    """Calls of different bases in the same kernels, 200 in each of three threads."""
    import threading
    probs = [cut_problem(oracle, N, 2) for N in (80, 160, 256)]
    E = [np.linspace(0.05, 0.15, 3) * p[2] for p in probs]
    ref = [oracle.transmission_jobs(p[1], e, nthreads=8)[0] for p, e in zip(probs, E)]
    seen = [None] * len(probs)

    def work(i):
        try:
            with Engine(*probs[i][0]) as eng:
                for _ in range(200):
                    tau, info = eng.transmission(E[i])
                    assert info == 0
                    np.testing.assert_allclose(tau, ref[i], rtol=RTOL, atol=ATOL)
                seen[i] = "done"
        except Exception as e:
            seen[i] = repr(e)

    threads = [threading.Thread(target=work, args=(i,)) for i in range(len(probs))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert seen == ["done"] * len(probs)


@pytest.mark.parametrize("N,nE", [(69, 3), (221, 3), (221, 80), (272, 20)])
def test_transmission_in_a_graph(oracle, N, nE):
    """The device entry under stream capture, one kernel or two, replayed on other energies."""
    import torch
    args, op, kmax = cut_problem(oracle, N, nz=2)
    with Engine(*args) as eng:
        dE = torch.linspace(0.05, 0.15, nE, dtype=torch.float64, device="cuda") * kmax
        dt = torch.zeros(nE, dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        eng.transmission_device(dE.data_ptr(), nE, dt.data_ptr())  # grows the workspace
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            eng.transmission_device(dE.data_ptr(), nE, dt.data_ptr(), stream=torch.cuda.current_stream().cuda_stream)
        for top in (0.12, 1.2):
            E = np.linspace(0.05, top, nE) * kmax
            dE.copy_(torch.tensor(E))
            graph.replay()
            torch.cuda.synchronize()
            ref, _ = oracle.transmission_jobs(op, E[::7], nthreads=8)
            np.testing.assert_allclose(dt.cpu().numpy()[::7], ref, rtol=RTOL, atol=ATOL)
        del graph
