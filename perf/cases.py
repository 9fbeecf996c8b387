"""The work that a user of this framework has it do, as cases that can be timed and checked.

Every case is one call of a public entry point (``Engine.transmission`` in FP64 or mixed precision,
``transmission_batch``, ``Engine.density_real``, ``Engine.density_neq``, ``Engine.ldos``,
``GreensFunction_tri_solver``) on a seeded split-gate device of ``negftrans_b200.workloads``: bases from a few
dozen plane waves to the 797 of the large-block workload, slices of 0.5 to 1 nm, one energy (a resonance being
refined) to a few hundred (a grid).  Host arrays go in and host arrays come out, as in the driver.

A case: ``call`` (the entry point), ``n`` (plane waves asked for; the circular cutoff gives the nearest shell),
``nz`` slices, ``n_e`` energies (for a density: the contour's points), ``grid`` real-space points in x and y,
``nk`` k-points per axis, ``lead`` the lead model.
"""
import math

import numpy as np
import torch

from negftrans_b200 import prepare as P
from negftrans_b200 import workloads as W
from negftrans_b200.negf import NEGF_MIXED, Engine, GreensFunction_tri_solver, transmission_batch

HARTREE, A_0 = 27.211386245988, 0.529177210903
K_B = 8.617333262e-5 / HARTREE
MSTAR = W.MSTAR
L_A = 1000.0                 # the 100 nm cell (Angstrom)
ENCUTS = {69: 0.0033091, 221: 0.0105288, 797: 0.0385807}  # the named workloads' cutoffs (eV)
T_K = MSTAR * 1.1605         # kT = 0.1 meV
MU = MSTAR * 20e-3 / HARTREE
LDOS_GRID = (0, -1, 0)       # the x-z map, integrated over y


def _case(name, call, n, nz, n_e, grid=64, nk=1, lead=0):
    return {"name": name, "call": call, "n": n, "nz": nz, "n_e": n_e, "grid": grid, "nk": nk, "lead": lead}


def listed():
    return [
        # one RGF solve of a small device: a bisection on a resonance, the sampler's single points
        _case("point_n69", "transmission", 69, 200, 1),
        # the whole energy grid of the 69-plane-wave QPC workload
        _case("grid_n69", "transmission", 69, 200, 512),
        # a handful of energies added around a threshold of the 221-plane-wave device
        _case("refine_n221", "transmission", 221, 160, 9),
        # an energy grid of the 221-plane-wave device: a full chip of sweeps
        _case("grid_n221", "transmission", 221, 160, 288),
        # the large-block workload in FP64
        _case("grid_n797", "transmission", 797, 16, 148, grid=128),
        # the large-block workload in mixed precision
        _case("mixed_n797", "mixed", 797, 60, 70, grid=128),
        # the medium workload in mixed precision
        _case("mixed_n221", "mixed", 221, 160, 148),
        # many k-points with bases of their own (180-263 plane waves) and devices of three lengths in one call
        _case("uneven_batch", "batch", 220, 15, 12, nk=4),
        # the equilibrium density of the 221-plane-wave device, matrix and real space
        _case("density_n221", "density", 221, 80, 152),
        # the density under a 1 mV bias of a small device
        _case("bias_n69", "bias", 69, 100, 120),
        # an LDOS map of the 69-plane-wave workload
        _case("ldos_n69", "ldos", 69, 200, 300),
        # the kernel-level solver that replaces math_kernel.f90's, called with the caller's own blocks
        _case("tri_solve_n69", "tri_solve", 69, 40, 1),
    ]


def draw(rng):
    call = rng.choice(["transmission"] * 6 + ["mixed"] * 2 + ["batch", "density", "density", "bias", "ldos", "ldos", "tri_solve"])
    while True:
        n = round(math.exp(rng.uniform(math.log(24), math.log(420 if call in ("transmission", "mixed") else 260))))
        nz = round(math.exp(rng.uniform(math.log(12), math.log(240))))
        n_e = round(math.exp(rng.uniform(math.log(1 if call == "transmission" else 8), math.log(400))))
        nk, lead = 1, 0
        if call == "tri_solve":
            n_e, nz = 1, min(nz, 60)
        elif call == "batch":
            n, nz, nk, n_e = rng.randint(190, 230), rng.randint(8, 24), rng.choice([2, 3, 4]), rng.randint(4, 24)
        elif call == "transmission":
            nk, lead = rng.choice([1, 1, 1, 2]), rng.choice([0, 0, 0, 1])
        elif call in ("ldos", "density") and n < 120:
            nk = rng.choice([1, 2])
        sweeps = n_e * nk * nk * (3 if call in ("density", "bias", "ldos") else 1)
        # a drawn case costs no more than the largest listed one, on the chip and (few jobs) along one sweep
        if float(n) ** 3 * nz * sweeps < 4e11 and n * nz < 3e4:
            return {"call": call, "n": n, "nz": nz, "n_e": n_e, "grid": 64, "nk": nk, "lead": lead}


# ---------------------------------------------------------------- inputs
def _encut(case):
    return ENCUTS.get(case["n"], case["n"] * 4.767e-5)


def _dz_nm(case):
    return 0.5 if case["n"] == 221 else 1.0


def _problem(case, seed):
    """A seeded QPC with disorder, prepared as main.f90 does; the k-mesh comes with it."""
    rng = np.random.Generator(np.random.PCG64(seed))
    nz, g, dz = case["nz"], case["grid"], _dz_nm(case)
    v = MSTAR * W.qpc_potential(g, g, nz, 100.0, nz * dz, rng.uniform(0.03, 0.07), rng.uniform(10.0, 22.0),
                                min(20.0, nz * dz / 8), disorder=0.002, seed=int(rng.integers(1, 1 << 31)))
    deck = W._deck(nz * dz * 10.0, _encut(case), 40.0, 16, nk=case["nk"])
    return P.prepare(deck, v), rng


def _energies(case, rng):
    """Ascending energies of [0.5, 40) meV (scaled): a grid with a seeded offset, or single points."""
    n = case["n_e"]
    return MSTAR * 1e-3 / HARTREE * (0.5 + 39.0 * (np.arange(n) + rng.uniform(0.05, 0.95)) / n)


def _batch_problems(case, seed):
    nz = case["nz"]
    return W.batched_uneven(nkx=case["nk"], nzs=(nz, 2 * nz, 4 * nz), seed=seed, n_range=(case["n"] - 40, case["n"] + 40))


def _contour(case):
    circle = max(4, case["n_e"] // 6)
    return circle, case["n_e"] - circle


def _lz_a(case):
    return case["nz"] * _dz_nm(case) * 10.0


def prepare(case, seed):
    if case["call"] == "batch":
        rng = np.random.Generator(np.random.PCG64(seed + 77))
        return {"case": case, "engines": [Engine(*p["args"]) for p in _batch_problems(case, seed)],
                "E": _energies(case, rng) * (30.0 / 40.0)}
    pr, rng = _problem(case, seed)
    st = {"case": case, "E": _energies(case, rng), "min_V": pr.min_V}
    if case["call"] == "tri_solve":
        D, _, _ = _blocks(pr.engine_args(), 0, st["E"][:1] + 1j * pr.atomic.ETA, "cpu")
        st["D"] = np.asfortranarray(np.stack([D(k)[0].numpy() for k in range(case["nz"])], axis=2))
    else:
        st["eng"] = Engine(*pr.engine_args(), lead_model=case["lead"])
    return st


def run(st):
    case = st["case"]
    call, g = case["call"], case["grid"]
    if call in ("transmission", "mixed"):
        return st["eng"].transmission(st["E"], NEGF_MIXED) if call == "mixed" else st["eng"].transmission(st["E"])
    if call == "batch":
        tau, info, _ = transmission_batch(st["engines"], st["E"])
        return tau, info
    if call == "density":
        circle, line = _contour(case)
        return st["eng"].density_real(circle, line, st["min_V"], MU, 6 * K_B * T_K, T_K, g, g, L_A, L_A, _lz_a(case))
    if call == "bias":
        circle, window = _contour(case)
        half = 0.5 * MSTAR * 1e-3 / HARTREE
        return st["eng"].density_neq(circle, window, st["min_V"], MU + half, MU - half, 6 * K_B * T_K, T_K)
    if call == "ldos":
        return st["eng"].ldos(st["E"][0], st["E"][0] + MSTAR * 30e-3 / HARTREE, case["n_e"], LDOS_GRID, g, g, L_A, L_A,
                              _lz_a(case))
    return GreensFunction_tri_solver(st["D"], "DFL")


# ---------------------------------------------------------------- the least work
def _count(encut_ev, kx=0.0, ky=0.0):
    b = 2 * math.pi / (L_A / A_0)
    r = int(math.sqrt(2 * encut_ev / HARTREE) / b) + 2
    i = np.arange(-r, r + 1) * b
    return int(np.sum((i[:, None] + kx) ** 2 + (i[None, :] + ky) ** 2 <= 2 * encut_ev / HARTREE))


def work(case):
    call, nz, n_e, g = case["call"], case["nz"], case["n_e"], case["grid"]
    sweeps = n_e * case["nk"] ** 2
    if call == "batch":  # sizes spread evenly over n-40 .. n+40, lengths nz, 2nz, 4nz
        sizes = np.linspace(case["n"] - 40, case["n"] + 40, case["nk"] ** 2)
        return {"flops": float(8 * np.sum(sizes ** 3) * 7 * nz * n_e), "bytes": float(16 * np.sum(sizes * 4) * 7 * nz)}
    n = _count(_encut(case))
    table = 16.0 * 4 * n * nz  # the V table has a few entries per plane wave and slice
    inverse, product = 8.0 * n ** 3 * nz, 8.0 * n ** 3 * (nz - 1)
    if call in ("transmission", "mixed"):
        return {"flops": inverse * sweeps, "bytes": table + 16.0 * n_e}
    if call == "tri_solve":  # D: inverses and two products a slice; F and L: one product each, and L's own inverses
        return {"flops": 2 * inverse + 4 * product, "bytes": 4 * 16.0 * n * n * nz}
    out = {"density": 16.0 * n * n * nz + 8.0 * g * g * nz, "bias": 16.0 * n * n * nz, "ldos": 8.0 * g * nz * n_e}[call]
    return {"flops": (inverse + 2 * product) * sweeps, "bytes": table + out}


# ---------------------------------------------------------------- the same in plain torch, 64 bits
def _blocks(args, ik, E, dev, lead=0):
    """D(k) -> (n_E, N, N) blocks of 2 dz^2 (E - H) - 2 with the lead terms, for complex energies E, and the
    transmission weights gamma (n_E, N) of both leads at Re E."""
    nx, ny, vhat, lx, ly, lz, v_l, v_r, _, kpt = args
    nz = vhat.shape[2]
    dz = lz / nz
    kx, ky, _ = np.asarray(kpt).reshape(-1, 3)[ik]
    ax, ay = 2 * np.pi * nx / lx + kx, 2 * np.pi * ny / ly + ky
    k2 = ax ** 2 + ay ** 2
    ix = nx[:, None] - nx[None, :] + (vhat.shape[0] - 1) // 2
    iy = ny[:, None] - ny[None, :] + (vhat.shape[1] - 1) // 2
    V = torch.as_tensor(np.ascontiguousarray(np.moveaxis(vhat, 2, 0))).to(dev)
    ix, iy = torch.as_tensor(ix).to(dev), torch.as_tensor(iy).to(dev)
    E = np.asarray(E, np.complex128)

    def lead_term(v):
        if lead == 0:
            q = np.sqrt(2 * (E[:, None] - v) - k2 + 0j)
            qr = np.sqrt(np.maximum(2 * (E.real[:, None] - v) - k2, 0.0))
            return np.exp(1j * q * dz), np.sin(qr * dz) / dz ** 2
        d = 2 * dz ** 2 * (E[:, None] - v - k2 / 2) - 2
        s = np.sqrt(d * d - 4 + 0j)
        g1, g2 = (d + s) / 2, (d - s) / 2
        dr = 2 * dz ** 2 * (E.real[:, None] - v - k2 / 2) - 2
        return (-np.where(abs(g1) <= abs(g2), g1, g2),
                np.where(abs(dr) < 2, np.sqrt(np.maximum(1 - dr * dr / 4, 0.0)), 0.0) / dz ** 2)

    (sl, gl), (sr, gr) = lead_term(v_l), lead_term(v_r)
    diag = torch.as_tensor(2 * dz ** 2 * (E[:, None] - k2 / 2) - 2).to(dev)
    sl, sr = torch.as_tensor(sl).to(dev), torch.as_tensor(sr).to(dev)

    def D(k):
        off = -2 * dz ** 2 * V[k][ix, iy]
        d = diag + (sl if k == 0 else 0) + (sr if k == nz - 1 else 0)
        return off + torch.diag_embed(d)

    return D, torch.as_tensor(gl).to(dev), torch.as_tensor(gr).to(dev)


def _right(D, nz):
    """The right-connected inverses X_b = inv(D_b - X_{b+1}), b = nz-1 .. 0."""
    x = None
    for b in range(nz - 1, -1, -1):
        x = torch.linalg.inv(D(b) if x is None else D(b) - x)
        yield b, x


def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _exact_tau(args, E, eta, lead):
    nz = args[2].shape[2]
    dz = args[5] / nz
    kpt = np.asarray(args[9]).reshape(-1, 3)
    tau = np.zeros(len(E))
    for ik in range(len(kpt)):
        D, gl, gr = _blocks(args, ik, E + 1j * eta, _device(), lead)
        rows = torch.nonzero((gl != 0).any(0)).flatten()
        p = None
        for _, x in _right(D, nz):
            p = x[:, rows, :] if p is None else p @ x
        t = torch.einsum("er,erc,ec->e", gl[:, rows], (2 * dz ** 2 * p).abs() ** 2, gr)
        tau += kpt[ik, 2] * t.cpu().numpy()
    return tau


def _diagonal(args, ik, E, per_slice, lead=0, spectral=None):
    """Calls per_slice(k, G_kk of all energies E, Y_k) with Y_k = G_k0[:, open] sqrt(gamma_L) where asked for."""
    nz = args[2].shape[2]
    D, gl, _ = _blocks(args, ik, E, _device(), lead)
    xs = [None] * nz
    for b, x in _right(D, nz):
        xs[b] = x
    g = xs[0]
    y = g * gl.sqrt()[:, None, :] if spectral else None
    eye = torch.eye(g.shape[1], dtype=g.dtype, device=g.device)
    for k in range(nz):
        if k:
            y = -(xs[k] @ y) if spectral else None
            g = xs[k] @ (eye + g @ xs[k])
            xs[k] = None
        per_slice(k, g, y)


def _phases(nx, ny, g):
    u = np.arange(g)
    f = np.exp(2j * np.pi * nx[:, None] * u / g)[:, :, None] * np.exp(2j * np.pi * ny[:, None] * u / g)[:, None, :]
    return torch.as_tensor(f.reshape(len(nx), g * g)).to(_device())


def _simpson(n, a, b):
    """The reference's composite rule: 1/3 throughout for odd n, the last four nodes by 3/8 for even n."""
    c = np.array([1 / 3 if i == 1 else 4 / 3 if i % 2 == 0 else 2 / 3 for i in range(1, n + 1)])
    if n % 2:
        c[-1] = 1 / 3
    else:
        c[n - 4] = 1 / 3 + 3 / 8 if n > 4 else 1 / 3
        c[n - 3:] = 9 / 8, 9 / 8, 3 / 8
    return np.linspace(a, b, n), c * (b - a) / (n - 1)


def _chunks(args, n_e):
    step = max(1, int(20e9 / (16.0 * len(args[0]) ** 2 * args[2].shape[2])))
    return [slice(i, min(n_e, i + step)) for i in range(0, n_e, step)]


def exact(case, seed):
    call, nz, g = case["call"], case["nz"], case["grid"]
    if call == "batch":
        rng = np.random.Generator(np.random.PCG64(seed + 77))
        E = _energies(case, rng) * (30.0 / 40.0)
        probs = _batch_problems(case, seed)
        return np.stack([_exact_tau(p["args"], E, p["args"][8], 0) for p in probs]), None
    pr, rng = _problem(case, seed)
    args, a = pr.engine_args(), pr.atomic
    E, dz = _energies(case, rng), pr.atomic.LZ / nz
    kpt = np.asarray(pr.kpoint).reshape(-1, 3)
    if call in ("transmission", "mixed"):
        if float(pr.N) ** 3 * nz * case["n_e"] > 3e12:
            return None
        return _exact_tau(args, E, a.ETA, case["lead"]), None
    if call == "tri_solve":
        D, _, _ = _blocks(args, 0, E[:1] + 1j * a.ETA, "cpu")
        blocks = [D(k)[0].numpy() for k in range(nz)]
        eye = np.eye(pr.N)
        right, left = [None] * nz, [None] * nz
        for k in range(nz):
            left[k] = np.linalg.inv(blocks[k] - (left[k - 1] if k else 0))
            b = nz - 1 - k
            right[b] = np.linalg.inv(blocks[b] - (right[b + 1] if k else 0))
        diag, first, last = [right[0]], [right[0]], [None] * nz
        for k in range(1, nz):
            diag.append(right[k] @ (eye + diag[-1] @ right[k]))
            first.append(-right[k] @ first[-1])
        last[nz - 1] = left[nz - 1]
        for k in range(nz - 2, -1, -1):
            last[k] = -left[k] @ last[k + 1]
        return {"D": np.stack(diag, 2), "F": np.stack(first, 2), "L": np.stack(last, 2)}, None
    if call == "ldos":
        E = E[0] + MSTAR * 30e-3 / HARTREE * np.arange(case["n_e"]) / case["n_e"]
        out = torch.zeros((g, 1, nz, case["n_e"]), dtype=torch.float64, device=_device())
        scale = nz / (L_A * L_A * _lz_a(case)) / HARTREE * (L_A / g)  # times dy: the y axis is integrated
        ph = _phases(args[0], args[1], g)
        for ik in range(len(kpt)):
            for c in _chunks(args, len(E)):
                def per_slice(k, G, _):
                    d = ((G.transpose(1, 2) @ ph) * ph.conj()).sum(1).imag.reshape(-1, g, g)
                    out[:, 0, k, c] += (-kpt[ik, 2] / np.pi * 2 * dz ** 2 * scale) * d.sum(2).T
                _diagonal(args, ik, E[c] + 1j * a.ETA, per_slice)
        return out.cpu().numpy(), None
    gap, kT = 6 * K_B * T_K, K_B * T_K
    bias = 0.5 * MSTAR * 1e-3 / HARTREE if call == "bias" else 0.0
    circle, line = _contour(case)
    lo, hi = MU - bias, MU + bias
    left_end = pr.min_V - 1 / HARTREE
    e_c, e_r = (lo - gap + left_end) / 2, (lo - gap - left_end) / 2
    if call == "bias":
        x, wt = np.polynomial.legendre.leggauss(circle)
        th, wt = np.pi / 2 * (x + 1), np.pi / 2 * wt
        x, wx = np.polynomial.legendre.leggauss(line)
        x, wx = (lo + hi) / 2 + (hi - lo + 2 * gap) / 2 * x, (hi - lo + 2 * gap) / 2 * wx
    else:
        th, wt = _simpson(circle, 0.0, np.pi)
        x, wx = _simpson(line, lo - gap, lo + gap)
    f_lo, f_hi = 1 / (np.exp((x - lo) / kT) + 1), 1 / (np.exp((x - hi) / kT) + 1)
    E = np.concatenate([e_c + e_r * np.exp(1j * th), x])
    cd = np.concatenate([2 / np.pi * wt * 1j * e_r * np.exp(1j * th), -2 / np.pi * wx * f_lo])
    ca = np.concatenate([0 * wt, 1j / np.pi * wx * (f_hi - f_lo) * (2 * dz ** 2)])
    dm = torch.zeros((nz, pr.N, pr.N), dtype=torch.complex128, device=_device())
    for ik in range(len(kpt)):
        for c in _chunks(args, len(E)):
            wd = torch.as_tensor(kpt[ik, 2] * cd[c]).to(dm.device)
            wa = torch.as_tensor(kpt[ik, 2] * ca[c]).to(dm.device)

            def per_slice(k, G, Y):
                dm[k] += 2 * dz ** 2 * torch.einsum("e,eij->ij", wd, G)
                if Y is not None:
                    dm[k] += 2 * dz ** 2 * torch.einsum("e,eic,ejc->ij", wa, Y, Y.conj())
            _diagonal(args, ik, E[c] + 1j * a.ETA, per_slice, spectral=call == "bias")
    matrix = dm.permute(1, 2, 0).cpu().numpy()
    if call == "bias":
        return matrix, None
    ph = _phases(args[0], args[1], g)
    real = torch.stack([((dm[k].T @ ph) * ph.conj()).sum(0).imag.reshape(g, g) for k in range(nz)], 2)
    return (real * (nz / (L_A * L_A * _lz_a(case)))).cpu().numpy(), matrix, None
