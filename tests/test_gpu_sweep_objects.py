"""Two partial-wave sweeps alive at once: the graph of the first keeps its own workspace, whatever a later, larger sweep or a
cleared workspace cache does to the shared ones."""

from __future__ import annotations

import pytest
import torch

import pyticc_b200 as tb
from pyticc_b200 import _native as nat
from pyticc_b200 import workloads

pytestmark = pytest.mark.gpu


def _plan(J, n_energy):
    parts = [workloads.rigid_atom_diatom(jmax=6, J=J, parity=p, n_energy=n_energy, boundaries=(2.5, 5.0)) for p in (1, -1)]
    plan = tb.PartialWaveSweep([w.system for w in parts], parts[0].grid, tb.Propagation(), n_energy=n_energy, energy_bound=float(parts[0].energies.max()), autotune=False)
    return plan, parts[0].energies


def _resident(plan) -> bool:
    """The workspace the graph replays into is a live tensor of the plan's own, large enough for every launch."""
    held = {id(b) for b in nat.Workspace._buffers.values()}
    return isinstance(plan.workspace, torch.Tensor) and id(plan.workspace) not in held and plan.workspace.numel() >= max(l.workspace_bytes for l in plan.launches)


def test_a_larger_sweep_leaves_the_first_ones_graph_alone():
    first, energies = _plan(1, 2)
    first.propagate(energies)  # direct, then captured
    want = [Y.clone() for Y in first.propagate(energies)]
    assert _resident(first)
    second, more = _plan(6, 8)
    assert second.workspace.numel() > first.workspace.numel() and second.workspace.data_ptr() != first.workspace.data_ptr()
    second.propagate(more)
    expected = [Y.clone() for Y in second.propagate(more)]
    nat.Workspace.release()
    torch.cuda.empty_cache()
    for _ in range(2):
        for Y, W in zip(first.propagate(energies), want, strict=True):
            assert torch.equal(Y, W)
        for Y, W in zip(second.propagate(more), expected, strict=True):
            assert torch.equal(Y, W)
