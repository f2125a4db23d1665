"""Timed cases of the coupled-channel path, through the entry points that a program calls.

Every case is one collision system of ``pyticc_b200.workloads`` (the rigid and the vibrating A+BC
rotor, the AB+CD rotor pair, the ultracold capture system) at some channel basis, radial range and
number of energies.  The seed draws the energies and the anisotropy of the potential, so that another
seed is another collision; coupling matrices and radial grids are those of the physical system.

kinds (``case["kind"]``):
  logd       ``propagate_logD``: all energies through a window of sectors, W matrices in hand
  window     ``propagation.propagate``: the same from the PES grid, plain or mixed precision
  blocks     ``propagation.propagate_blocks``: the K blocks of a coupled-states or NNCC system
  sweep      ``PartialWaveSweep.propagate``: uneven (J, parity) blocks replayed as one CUDA graph
  contract   ``contract_device``: PES values on the quadrature -> V(R)
  transform  ``transform_logD_BF_to_SF``
  match      ``get_Smat``
  solve      ``solve``: PES grid to S matrices
"""

from __future__ import annotations

import math

import numpy as np
import torch

import pyticc_b200 as tb
from pyticc_b200 import workloads
from pyticc_b200.matrix.interaction import contract_device, device_basis
from pyticc_b200.propagation import propagate, propagate_blocks
from pyticc_b200.scattering import build_hamiltonian, build_k_blocks

F64 = torch.float64

# energy range above the ground state (cm^-1; K for the capture system), half-step (bohr),
# innermost radius of a window, outer end of the grid
# (on the repulsive wall; ``window`` starts at WINDOW_R0, where part of the channels are open)
WINDOW_R0 = 5.0
FAMILIES = {
    "rigid": dict(energy=(10.0, 500.0), h=0.05, R0=4.4, R1=30.0),
    "morse": dict(energy=(100.0, 3000.0), h=0.02, R0=4.4, R1=40.0),
    "pair": dict(energy=(5.0, 800.0), h=0.05, R0=5.0, R1=30.0),
    "capture": dict(energy=(1.0e-6, 1.0e-3), h=0.05, R0=12.0, R1=1500.0),
}


def listed():
    return [
        # the smallest call: one energy of the J = 0 block of a rigid rotor; launches and latency
        dict(name="logd_j0", kind="logd", family="rigid", jmax=20, J=0, parity=1, sectors=16, energies=1),
        # the rigid-rotor block that one process solves most often (N = 231, 16 energies)
        dict(name="logd_rigid", kind="logd", family="rigid", jmax=20, J=20, parity=1, sectors=8, energies=16),
        # a middle partial wave of the vibrating system, few energies (N = 660)
        dict(name="logd_mid", kind="logd", family="morse", jmax=30, J=6, parity=-1, sectors=4, energies=5),
        # the vibrating benchmark block, plain FP64 (N = 1984)
        dict(name="logd_vib", kind="logd", family="morse", jmax=30, J=30, parity=1, sectors=1, energies=16),
        # incoming-wave capture: complex log-derivatives (N = 396)
        dict(name="logd_capture", kind="logd", family="capture", jmax=40, J=10, parity=1, sectors=3, energies=8),
        # the vibrating block of the other parity in mixed precision, a production batch of energies (N = 1860)
        dict(name="window_mixed", kind="window", family="morse", jmax=30, J=30, parity=-1, sectors=2, energies=32, precision="mixed"),
        # coupled states: 21 K blocks of 1 to 21 channels propagated together
        dict(name="blocks_cs", kind="blocks", family="rigid", jmax=20, J=20, parity=1, sectors=12, energies=16, approx="cs"),
        # partial-wave sum over uneven blocks (N = 36 to 340), replayed
        dict(name="sweep_uneven", kind="sweep", family="morse", jmax=12, J=8, J_step=4, sectors=10, energies=8),
        # V(R) of the AB+CD pair: complex bispherical rows (N = 899, 2700 grid points)
        dict(name="contract_pair", kind="contract", family="pair", jmax=6, J=4, parity=1, points=33),
        # asymptotic frame change of the vibrating block
        dict(name="transform_vib", kind="transform", family="morse", jmax=30, J=30, parity=1, energies=8),
        # matching of the rigid-rotor block
        dict(name="match_rigid", kind="match", family="rigid", jmax=20, J=20, parity=1, energies=16),
        # the whole call: PES grid to S matrices
        dict(name="solve_rigid", kind="solve", family="rigid", jmax=20, J=20, parity=1, sectors=24, energies=16),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 0.49)))))))


def draw(rng):
    kind = rng.choice(["logd", "logd", "logd", "window", "window", "blocks", "sweep", "contract", "transform", "match", "solve"])
    case = dict(kind=kind)
    if kind in ("contract",):
        case.update(family=rng.choice(["pair", "morse", "rigid"]))
    elif kind in ("blocks", "solve"):
        case.update(family="rigid")
    elif kind == "sweep":
        case.update(family=rng.choice(["rigid", "morse"]))
    elif kind == "window":
        case.update(family="morse", precision=rng.choice(["fp64", "mixed"]))
    elif kind == "logd":
        case.update(family=rng.choice(["rigid", "morse", "morse", "capture"]))
    else:
        case.update(family=rng.choice(["rigid", "morse"]))
    family = case["family"]
    top = {"rigid": 20, "morse": 30, "pair": 6, "capture": 40}[family]
    if kind == "sweep":
        case.update(jmax=rng.randint(6, 12), J=rng.randint(4, 10), J_step=rng.randint(2, 4), sectors=rng.randint(5, 20), energies=_log_int(rng, 1, 12))
        return case
    low = 3 if family == "pair" else 6
    case.update(jmax=rng.randint(low, top))
    case.update(J=rng.randint(1, {"pair": 4, "capture": 12}.get(family, case["jmax"])), parity=rng.choice([1, -1]))
    if kind == "contract":
        case.update(points=_log_int(rng, 1, 33))
        return case
    case.update(energies=_log_int(rng, 1, 32))
    if kind in ("logd", "window", "blocks", "solve"):
        # no more work than the largest listed case: 2 inversions of N^3 flops a sector and energy
        n = sum(max(0, case["jmax"] + 1 - K) for K in range(case["J"] + 1)) * {"morse": 4}.get(family, 1)
        cost = 2.0 * n**3 * (4 if family == "capture" else 1)
        case["energies"] = int(max(1, min(case["energies"], 4.0e11 // cost)))
        case["sectors"] = int(max(1, min(rng.randint(8, 24) if kind == "solve" else rng.randint(1, 4) if kind == "window" else _log_int(rng, 1, 16), 4.0e11 // (cost * case["energies"]))))
    elif kind == "transform":
        case["energies"] = min(case["energies"], 16)
    if kind == "blocks":
        case["approx"] = rng.choice(["cs", "nncc"])
    return case


# ---- inputs ---------------------------------------------------------------------------------------


def _energies(case, E_int, seed):
    """The family's energies, each moved by the seed inside its own gap between two thresholds, so
    that the channels open at it are the same for every seed."""
    family, count = case["family"], case.get("energies", 1)
    rng = np.random.default_rng([seed, 17])
    lo, hi = FAMILIES[family]["energy"]
    at = (np.arange(count) + 0.5) / count
    base = lo * (hi / lo) ** at * tb.K2AU if family == "capture" else (lo + (hi - lo) * at) * tb.CM2AU
    levels = np.unique(np.concatenate([[0.0], np.asarray(E_int)]))
    above = np.searchsorted(levels, base, side="right")
    gap = np.minimum(base - levels[above - 1], np.concatenate([levels, [2.0 * base[-1]]])[above] - base)
    return base + 0.4 * gap * rng.uniform(-1.0, 1.0, count)


def _workload(case, seed, *, J=None, parity=None, sectors=None):
    """The physical system with a radial grid of the case's window and one wide sector out to R1
    (the channel order looks at the outermost point); ``solve`` and ``sweep`` use the window only."""
    family = case["family"]
    f = FAMILIES[family]
    rng = np.random.default_rng([seed, 5])
    count = sectors if sectors is not None else case.get("sectors", 1)
    R0 = WINDOW_R0 if case["kind"] == "window" else f["R0"]
    end = R0 + 2.0 * f["h"] * count
    boundaries, steps = (R0, end, f["R1"]), (f["h"], 0.5 * (f["R1"] - end))
    if case["kind"] in ("solve", "sweep"):
        boundaries, steps = (R0, end), (f["h"],)
    common = dict(J=case["J"] if J is None else J, parity=case.get("parity", 1) if parity is None else parity, jmax=case["jmax"], boundaries=boundaries, half_steps=steps)
    if family == "rigid":
        if "approx" in case:
            common["approx"] = tb.Approx.CS if case["approx"] == "cs" else tb.Approx.NNCC
        return workloads.rigid_atom_diatom(a1=0.3 + 0.1 * rng.uniform(-1, 1), a2=0.2 + 0.1 * rng.uniform(-1, 1), n_energy=1, **common)
    if family == "morse":
        return workloads.morse_atom_diatom(seed=int(seed), n_energy=1, **common)
    if family == "pair":
        return workloads.rotor_pair(seed=int(seed), n_energy=1, **common)
    return workloads.ultracold_capture(seed=int(seed), n_energy=1, **common)


def _device():
    return torch.device("cuda", torch.cuda.current_device())


def _interaction(hamiltonian, points, device, indices=None):
    """V(R) in plain torch for the channels ``indices``."""
    basis = hamiltonian.V_basis
    n = basis.n_channel if indices is None else len(indices)
    place = {c: k for k, c in enumerate(range(basis.n_channel) if indices is None else indices)}
    values = torch.as_tensor(np.ascontiguousarray(hamiltonian.potential_grid.take(points).reshape(len(points), -1)), device=device)
    V = torch.zeros((len(points), n, n), dtype=F64, device=device)
    for K, members in basis.channel_indices.items():
        rows = [r for r, c in enumerate(members) if c in place]
        if not rows:
            continue
        out = torch.as_tensor([place[members[r]] for r in rows], device=device)
        for part in (basis.B_real[K],) if basis.B_imag is None else (basis.B_real[K], basis.B_imag[K]):
            B = torch.as_tensor(np.ascontiguousarray(part[rows]), device=device)
            for r in range(len(points)):
                V[r][out[:, None], out[None, :]] += basis.normalization * ((B * values[r]) @ B.T)
    return 0.5 * (V + V.transpose(-1, -2))


def _W(hamiltonian, points, device, indices=None):
    """W_base(R) = U/R^2 + 2 mu [V(R) + diag(E_int)] in plain torch."""
    mu = hamiltonian.reduced_mass
    idx = np.arange(hamiltonian.basis.n_channel) if indices is None else np.asarray(indices)
    U = torch.as_tensor(np.ascontiguousarray(hamiltonian.centrifugal(None if indices is None else tuple(indices))), device=device)
    E = torch.as_tensor(np.ascontiguousarray(hamiltonian.E_int[idx]), device=device)
    R = torch.as_tensor(np.ascontiguousarray(points), device=device)[:, None, None]
    return U[None] / (R * R) + 2.0 * mu * (_interaction(hamiltonian, points, device, indices) + torch.diag(E)[None])


def _initial(W0, energies, mu, is_complex):
    d = torch.diagonal(W0)[None, :] - 2.0 * mu * energies[:, None]
    if not is_complex:
        return torch.diag_embed(torch.sqrt(torch.abs(d)))
    zero = torch.zeros_like(d)
    return torch.diag_embed(torch.complex(torch.sqrt(torch.clamp(d, min=0.0)), torch.where(d < 0.0, -torch.sqrt(torch.clamp(-d, min=0.0)), zero)))


def _window_points(grid, count):
    sectors = grid.sectors[:count]
    points = [sectors[0].radial_start]
    for s in sectors:
        points += [s.radial_mid, s.radial_end]
    return sectors, np.asarray(points)


def _sweep_systems(case, seed):
    out = []
    for J in range(0, case["J"] + 1, case["J_step"]):
        for parity in (1, -1):
            out.append(_workload(case, seed, J=J, parity=parity))
    return out


def prepare(case, seed):
    dev, kind, family = _device(), case["kind"], case["family"]
    if kind == "sweep":
        parts = _sweep_systems(case, seed)
        bound = 2.0 * FAMILIES[family]["energy"][1] * tb.CM2AU
        energies = _energies(case, parts[0].system.basis.E_int, seed)
        plan = tb.PartialWaveSweep([w.system for w in parts], parts[0].grid, tb.Propagation(), n_energy=case["energies"], energy_bound=bound)
        plan.propagate(energies)
        return dict(kind=kind, plan=plan, energies=energies)
    wl = _workload(case, seed)
    if kind == "solve":
        return dict(kind=kind, system=wl.system, grid=wl.grid, energies=_energies(case, wl.system.basis.E_int, seed))
    hamiltonian = build_hamiltonian(wl.system, wl.grid)
    if kind == "contract":
        rng = np.random.default_rng([seed, 23])
        strength = 0.1 + rng.uniform(size=(case["points"], 1))
        values = wl.grid.values[:1].reshape(1, -1) * strength + 1.0e-4 * rng.normal(size=(case["points"], wl.grid.values[0].size))
        return dict(kind=kind, basis=hamiltonian.V_basis, cache=device_basis(hamiltonian.V_basis), values=torch.as_tensor(values, device=dev))
    energies = _energies(case, hamiltonian.E_int, seed)
    if kind == "window":
        return dict(kind=kind, hamiltonian=hamiltonian, energies=energies, sectors=wl.grid.sectors[: case["sectors"]], config=tb.Propagation(precision=case["precision"]))
    if kind == "blocks":
        blocks = tuple(b.channel_indices for b in build_k_blocks(hamiltonian))
        return dict(kind=kind, hamiltonian=hamiltonian, blocks=blocks, energies=energies, sectors=wl.grid.sectors[: case["sectors"]], config=tb.Propagation())
    mu = hamiltonian.reduced_mass
    if kind == "logd":
        sectors, points = _window_points(wl.grid, case["sectors"])
        # most strongly closed channels first, as callers of propagate_logD order them
        outer = torch.diagonal(_W(hamiltonian, wl.grid.radial_points[-1:], dev)[0])
        order = torch.argsort(outer, descending=True, stable=True)
        W = _W(hamiltonian, points, dev)[:, order][:, :, order].contiguous()
        E = torch.as_tensor(energies, device=dev)
        halves = torch.as_tensor(np.asarray([s.radial_half_step for s in sectors]), device=dev)
        Y = _initial(W[0], E, mu, family == "capture")
        return dict(kind=kind, Y=Y, E=E, mu=mu, h=halves, Ws=W[0:-1:2].contiguous(), Wm=W[1::2].contiguous(), We=W[2::2].contiguous())
    # a log-derivative batch at the matching radius: the wavenumbers on the diagonal, couplings off it
    n = hamiltonian.basis.n_channel
    B, L = tb.get_Bmat_BF_to_SF(hamiltonian.basis)
    gen = torch.Generator(device=dev).manual_seed(int(seed))
    E = torch.as_tensor(energies, device=dev)
    k2 = 2.0 * mu * (E[:, None] - torch.as_tensor(np.ascontiguousarray(hamiltonian.E_int), device=dev)[None, :])
    k = torch.sqrt(torch.abs(k2))
    C = torch.randn((energies.size, n, n), generator=gen, dtype=F64, device=dev)
    C = 0.5 * (C + C.transpose(-1, -2)) * (0.3 / math.sqrt(n)) * torch.sqrt(k[:, :, None] * k[:, None, :])
    tilt = torch.where(k2 > 0.0, 2.0 * torch.rand((energies.size, n), generator=gen, dtype=F64, device=dev) + 0.5, torch.ones_like(k2))
    Y = (C + torch.diag_embed(k * tilt)).contiguous()
    return dict(kind=kind, Y=Y, B=B, L=np.round(L), E_int=np.ascontiguousarray(hamiltonian.E_int), energies=energies, mu=mu, Rmatch=FAMILIES[family]["R1"])


def run(state):
    kind = state["kind"]
    if kind == "logd":
        return tb.propagate_logD(state["Y"], state["E"], state["mu"], state["h"], state["Ws"], state["Wm"], state["We"])
    if kind == "window":
        return propagate(state["hamiltonian"], state["energies"], state["sectors"], state["config"])
    if kind == "blocks":
        return list(propagate_blocks(state["hamiltonian"], state["blocks"], state["energies"], state["sectors"], state["config"]))
    if kind == "sweep":
        return [Y for Y in state["plan"].propagate(state["energies"]) if Y is not None]
    if kind == "contract":
        return contract_device(state["basis"], state["cache"], state["values"])
    if kind == "transform":
        return tb.transform_logD_BF_to_SF(state["Y"], state["B"])
    if kind == "match":
        return list(tb.get_Smat(state["Y"], state["Rmatch"], state["energies"], state["mu"], state["E_int"], state["L"]))
    result = tb.solve(state["system"], state["energies"], state["grid"], tb.Propagation())
    return dict(S=list(result.Smat), Y=result.Y_propagated)


# ---- work -----------------------------------------------------------------------------------------


def _propagation_work(n, energies, sectors, is_complex):
    """Two symmetric inversions (n^3 flops each; 4 times that when complex) a sector and energy and
    one energy-shared real inversion a sector; W read once, Y read and written once."""
    flops = sectors * (2 * energies * (4 if is_complex else 1) + 1) * float(n) ** 3
    return dict(bytes=8.0 * n * n * (2 * energies * (2 if is_complex else 1) + 2 * sectors + 1), flops=flops)


def _contraction_work(basis, points):
    grid = math.prod(basis.grid_shape)
    parts = 1 if basis.B_imag is None else 2
    pairs = sum(len(m) * (len(m) + 1) // 2 for m in basis.channel_indices.values())
    return dict(bytes=8.0 * (parts * basis.n_channel * grid + points * grid + points * basis.n_channel**2), flops=2.0 * grid * parts * pairs * points)


def _plus(*works):
    return dict(bytes=sum(w["bytes"] for w in works), flops=sum(w["flops"] for w in works))


def work(case):
    kind, family = case["kind"], case["family"]
    if kind == "sweep":
        sizes = [(w.system.basis.n_channel, build_hamiltonian(w.system, w.grid)) for w in _sweep_systems(case, 1) if w.system.basis.n_channel]
        return _plus(*[_plus(_propagation_work(n, case["energies"], case["sectors"], False), _contraction_work(h.V_basis, 2 * case["sectors"] + 1)) for n, h in sizes])
    wl = _workload(case, 1)
    n, ne = wl.system.basis.n_channel, case.get("energies", 1)
    if kind == "logd":
        return _propagation_work(n, ne, case["sectors"], family == "capture")
    if kind == "transform":
        return dict(bytes=8.0 * n * n * (2 * ne + 1), flops=4.0 * ne * float(n) ** 3)
    if kind == "match":
        # closed channels eliminated (one symmetric inversion), one complex solve of the open block
        e = _energies(case, wl.system.basis.E_int, 1)
        opened = [int(np.sum(wl.system.basis.E_int < v)) for v in e]
        return dict(bytes=8.0 * n * n * ne + 16.0 * sum(o * o for o in opened), flops=ne * float(n) ** 3 + sum(8.0 / 3.0 * 4.0 * float(o) ** 3 for o in opened))
    hamiltonian = build_hamiltonian(wl.system, wl.grid)
    if kind == "contract":
        return _contraction_work(hamiltonian.V_basis, case["points"])
    if kind == "blocks":
        sizes = [len(b.channel_indices) for b in build_k_blocks(hamiltonian)]
        total = [_propagation_work(m, ne, case["sectors"], False) for m in sizes]
        return _plus(*total, _contraction_work(hamiltonian.V_basis, 2 * case["sectors"] + 1))
    whole = _plus(_propagation_work(n, ne, case["sectors"], False), _contraction_work(hamiltonian.V_basis, 2 * case["sectors"] + 1))
    if kind == "solve":
        whole = _plus(whole, dict(bytes=0.0, flops=5.0 * ne * float(n) ** 3))
    return whole


# ---- the same in 64 bits, in plain torch and numpy -------------------------------------------------


def _reference_pair(p2, h):
    mag = torch.sqrt(torch.abs(p2))
    arg = mag * h
    small = torch.abs(arg) < 1.0e-5
    safe = torch.where(small, torch.ones_like(arg), arg)
    y1 = torch.where(p2 >= 0.0, mag / torch.tanh(safe), mag / torch.tan(safe))
    y2 = torch.where(p2 >= 0.0, mag / torch.sinh(safe), mag / torch.sin(safe))
    s1 = 1.0 / h + p2 * h / 3.0 - p2 * p2 * h**3 / 45.0
    s2 = 1.0 / h - p2 * h / 6.0 + 7.0 * p2 * p2 * h**3 / 360.0
    return torch.where(small, s1, y1), torch.where(small, s2, y2)


def _propagate64(Y, E, mu, halves, Ws, Wm, We):
    n = Y.shape[-1]
    eye = torch.eye(n, dtype=F64, device=Y.device)
    Y = Y.clone()
    for s, h in enumerate(float(v) for v in halves):
        ref = torch.diagonal(Wm[s])
        Qs, Qe = h / 3.0 * (Ws[s] - torch.diag(ref)), h / 3.0 * (We[s] - torch.diag(ref))
        Qm = 4.0 / h * (torch.linalg.inv(eye - h * h / 6.0 * (Wm[s] - torch.diag(ref))) - eye)
        for e in range(Y.shape[0]):
            y1, y2 = _reference_pair(ref - 2.0 * mu * E[e], h)
            d = torch.diag(y1)
            mid = Qm + d - y2[:, None] * torch.linalg.inv(Y[e] + Qs + d) * y2[None, :]
            Y[e] = Qe + d - y2[:, None] * torch.linalg.inv(mid + Qm + d) * y2[None, :]
    return Y


def _propagate_system64(hamiltonian, sectors, energies, device, indices=None):
    _, points = _window_points(hamiltonian.potential_grid, len(sectors))
    W = _W(hamiltonian, points, device, indices)
    E = torch.as_tensor(energies, device=device)
    mu = hamiltonian.reduced_mass
    return _propagate64(_initial(W[0], E, mu, False), E, mu, [s.radial_half_step for s in sectors], W[0:-1:2], W[1::2], W[2::2])


def _riccati(ell, x):
    """x j_l, x y_l and derivatives for one integer l: y upward, j downward from far above."""
    n0, n1 = math.sin(x), -math.cos(x)  # l = -1, 0
    for k in range(ell):
        n0, n1 = n1, (2 * k + 1) / x * n1 - n0
    top = int(max(ell, x)) + 60 + int(4.0 * math.sqrt(max(ell, x)))
    a, b, at, below = 0.0, 1.0e-290, 0.0, 0.0  # l = top + 1, top
    for k in range(top, -1, -1):  # b at l = k
        if k == ell:
            at = b
        if k == ell - 1:
            below = b
        a, b = b, (2 * k + 1) / x * b - a
        if abs(b) > 1.0e200:
            a, b, at, below = a * 1.0e-200, b * 1.0e-200, at * 1.0e-200, below * 1.0e-200
    if ell == 0:
        below = b  # l = -1
    # b ~ cos x (l = -1), a ~ sin x (l = 0)
    scale = math.sin(x) / a if abs(math.sin(x)) > abs(math.cos(x)) else math.cos(x) / b
    j, jm = at * scale, below * scale
    return j, n1, jm - ell / x * j, n0 - ell / x * n1


def _smat64(Y, Rmatch, energies, mu, E_int, L):
    out = []
    L = np.round(L).astype(int)
    for e, E in enumerate(energies):
        opened = np.flatnonzero(E_int < E)
        k = np.sqrt(2.0 * mu * np.abs(E - E_int))
        gamma = np.zeros(E_int.size)
        for i in np.flatnonzero(E_int > E):
            r, x = 1.0, k[i] * Rmatch
            for m in range(L[i]):
                r = 1.0 / (r + (2 * m + 1) / x)
            gamma[i] = 0.5 / Rmatch + k[i] * (-r - (L[i] + 0.5) / x)
        G = np.linalg.inv(Y[e] - np.diag(gamma))[np.ix_(opened, opened)]
        f = np.array([_riccati(L[i], k[i] * Rmatch) for i in opened]).reshape(-1, 4)
        root = np.sqrt(k[opened])
        J, N, Jp, Np = f[:, 0] / root, f[:, 1] / root, f[:, 2] * root, f[:, 3] * root
        A = np.diag(N - 1j * J) - G * (Np - 1j * Jp)[None, :]
        B = np.diag(N + 1j * J) - G * (Np + 1j * Jp)[None, :]
        out.append(np.linalg.solve(A, B))
    return out


def exact(case, seed):
    dev, kind = _device(), case["kind"]
    if kind == "sweep":
        parts = [w for w in _sweep_systems(case, seed) if w.system.basis.n_channel]
        energies = _energies(case, parts[0].system.basis.E_int, seed)
        return [_propagate_system64(build_hamiltonian(w.system, parts[0].grid), parts[0].grid.sectors, energies, dev) for w in parts]
    if kind in ("window", "blocks", "solve"):
        wl = _workload(case, seed)
        hamiltonian = build_hamiltonian(wl.system, wl.grid)
        energies = _energies(case, hamiltonian.E_int, seed)
        sectors = wl.grid.sectors[: case["sectors"]]
        if kind == "window":
            return _propagate_system64(hamiltonian, sectors, energies, dev)
        if kind == "blocks":
            return [_propagate_system64(hamiltonian, sectors, energies, dev, b.channel_indices) for b in build_k_blocks(hamiltonian)]
        Y = _propagate_system64(hamiltonian, sectors, energies, dev).cpu().numpy()
        B, L = tb.get_Bmat_BF_to_SF(hamiltonian.basis)
        return dict(S=_smat64(B.T @ Y @ B, sectors[-1].radial_end, energies, hamiltonian.reduced_mass, np.asarray(hamiltonian.E_int), L), Y=Y)
    state = prepare(case, seed)
    if kind == "logd":
        return _propagate64(state["Y"], state["E"], state["mu"], state["h"], state["Ws"], state["Wm"], state["We"])
    if kind == "contract":
        basis, values = state["basis"], state["values"]
        V = torch.zeros((values.shape[0], basis.n_channel, basis.n_channel), dtype=F64, device=dev)
        for K, members in basis.channel_indices.items():
            at = torch.as_tensor(members, device=dev)
            for part in (basis.B_real[K],) if basis.B_imag is None else (basis.B_real[K], basis.B_imag[K]):
                rows = torch.as_tensor(part, device=dev)
                for r in range(values.shape[0]):
                    V[r][at[:, None], at[None, :]] += basis.normalization * ((rows * values[r]) @ rows.T)
        return V
    if kind == "transform":
        B = torch.as_tensor(state["B"], device=dev)
        return B.T @ state["Y"] @ B
    return _smat64(state["Y"].cpu().numpy(), state["Rmatch"], state["energies"], state["mu"], state["E_int"], state["L"])
