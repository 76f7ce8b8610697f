"""Which per-edge buffers a force field allocates for the memory that is free, on the CPU: the device's memory is a number
that the allocations are taken from."""
import types
import weakref

import numpy as np
import pytest
import torch

from fastmace_b200 import _lib, forcefield
from fastmace_b200.model import SPECS, init_weights
from fastmace_b200.packing import PackedModel

CAPACITY, ATOMS = 4096, 64
PACKED = {}


def _allocated(monkeypatch, model, free, total, **options):
    """A force field with its work buffers allocated on a device with ``free`` of ``total`` bytes, and what is left."""
    spec = SPECS[model]
    if model not in PACKED:
        PACKED[model] = PackedModel(spec, init_weights(spec, 1), [11, 17], "cpu")
    used = [0]
    real = torch.zeros

    def zeros(*shape, **kw):
        t = real(*shape, **kw)
        if used[0] + t.nbytes > free:
            raise torch.OutOfMemoryError
        used[0] += t.nbytes
        weakref.finalize(t, lambda n=t.nbytes: used.__setitem__(0, used[0] - n))
        return t

    monkeypatch.setattr(forcefield, "DEFAULT_CHUNK_EDGES", 256)
    for name, value in dict(mem_get_info=lambda *_: (free - used[0], total), memory_reserved=lambda *_: 0,
                            memory_allocated=lambda *_: 0, empty_cache=lambda: None).items():
        monkeypatch.setattr(torch.cuda, name, value)
    ff = object.__new__(forcefield.B200ForceField)
    ff.spec, ff.packed, ff._device, ff._compute_stress = spec, PACKED[model], torch.device("cpu"), False
    ff.atom_capacity = ff.natoms = ATOMS
    ff.neighbours = types.SimpleNamespace(capacity=CAPACITY)
    ff.numbers = np.full(ATOMS, 11)
    ff.n_owned, ff.n_inner, ff.halo_exchange = options.get("n_owned", -1), options.get("n_inner", -1), False
    ff.chunk_edges, ff.edge_adjoint = None, options.get("edge_adjoint")
    ff.species, ff.symcon_groups, ff.n_symcon_groups = torch.zeros(1), torch.zeros(1), 0
    ff._outputs()
    with monkeypatch.context() as patch:
        patch.setattr(torch, "zeros", zeros)
        ff._allocate_work()
    return ff, free - used[0]


def _sweep(model, low=0.3, high=4.0):
    """Amounts of free memory around what the whole list takes as one chunk."""
    spec = SPECS[model]
    paths, hidden = max(len(spec.paths(t)) for t in range(2)), (spec.hidden_lmax + 1) ** 2
    whole = CAPACITY * (1132 + hidden * 512 + 0.5625 * 2 * paths * 512) + ATOMS * 4 * 20000
    return [int(whole * f) for f in np.geomspace(low, high, 40)]


@pytest.mark.parametrize("model", ["small", "medium", "large"])
@pytest.mark.parametrize("share", [1.0, 0.5, 0.17])                  # of the device that is free
def test_pair_rows_come_with_their_map(monkeypatch, model, share):
    """Radial weights sized for one row per pair of opposite edges need the pair map, which needs the hand-over buffers."""
    seen = set()
    for free in _sweep(model):
        try:
            ff, _ = _allocated(monkeypatch, model, free, int(free / share))
        except torch.OutOfMemoryError:
            continue
        w = ff.work
        assert not w.pair_capacity or (w.edge_slot and w.canon_list and w.canon_count and w.chunk_edges == CAPACITY)
        assert ff.buf["tp_w"].shape[0] == 2 * (w.pair_capacity or w.chunk_edges)
        seen.add(bool(w.pair_capacity))
    assert seen == {False, True}


@pytest.mark.parametrize("model", ["small", "medium", "large"])
@pytest.mark.parametrize("n_owned,n_inner,same", [(10, 20, False), (10, -1, False), (10, 10, True), (ATOMS, -1, True)])
def test_pair_rows_need_both_interactions_on_the_same_atoms(monkeypatch, model, n_owned, n_inner, same):
    """With an inner halo the adjoint covers more atoms than the forward pass and cannot use its radial weights."""
    free = _sweep(model)[-1]
    ff, _ = _allocated(monkeypatch, model, free, free, n_owned=n_owned, n_inner=n_inner)
    assert bool(ff.work.pair_capacity) == same


@pytest.mark.parametrize("model", ["small", "medium", "large"])
@pytest.mark.parametrize("share", [1.0, 0.5])
@pytest.mark.parametrize("edge_adjoint", [None, False])
def test_hand_over_buffers_leave_a_tenth_of_the_device(monkeypatch, model, share, edge_adjoint):
    """Those of the whole list and those of one chunk; both occur in the sweep, and so does going without."""
    seen = set()
    for free in _sweep(model, 0.2):
        try:
            ff, left = _allocated(monkeypatch, model, free, int(free / share), edge_adjoint=edge_adjoint)
        except torch.OutOfMemoryError:
            continue
        handed = [name in ff.buf for name in ("mirror", "edge_q", "edge_dx")]
        assert all(handed) or not any(handed)
        assert not any(handed) or left >= int(free / share) // 10
        seen.add(len(ff.buf["edge_dx"]) if all(handed) else 0)
    assert seen >= {0, CAPACITY} and (edge_adjoint is False or 256 in seen or share == 0.5)
