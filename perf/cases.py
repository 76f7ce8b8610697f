"""The work of this package as a program that uses it has it done: force calls, Langevin steps, neighbour builds and
steps of a spatially decomposed run, from a few dozen atoms to the sizes where the per-edge work fills the device.

``listed()`` names the cases, ``draw(rng)`` gives more of the same ranges, ``prepare`` makes what a program holds before
the call, ``run`` is one pass, ``work`` and ``tolerance`` state what a pass cannot do without and how far two correct
fp32 implementations may differ, ``exact`` is the same computation in plain float64 torch.

The models are the three sizes of the benchmark (hidden irreps up to l = 0, 1, 2; 128 channels, r_cut 6 Å) with their
fixed random weights; positions, species and velocities come from the seed.
"""

from __future__ import annotations

import dataclasses
import functools
import math

import numpy as np
import torch
from torch.utils.checkpoint import checkpoint

from fastmace_b200.engine import B200Engine
from fastmace_b200.forcefield import B200ForceField
from fastmace_b200.halo import DomainSimulation
from fastmace_b200.langevin import IntegratorConfig, Langevin
from fastmace_b200.model import SPECS, init_weights
from fastmace_b200.neighbours import CellListNeighbours
from fastmace_b200.state import SimulationState
from fastmace_b200.structures import FS, KB, fcc_alloy, nacl, silica

WEIGHT_SEED = {"small": 0, "medium": 1, "large": 2}
NEIGHBOURS = {"nacl": 32.0, "alloy": 32.0, "silica": 60.0}       # avg_num_neighbors the model was set up with
SKIN = 0.3


# ------------------------------------------------------------------------------------------------ the cases


def listed():
    return [
        # one-off evaluation of a small crystal from host arrays (the call of a calculator): latency, launches, copies
        dict(name="evaluate_small_nacl_216", call="evaluate", model="small", system="nacl", nx=3, ny=3, nz=3, stress=True),
        # the smallest MD step: a cell about as wide as the interaction range, every kernel a fraction of a wave
        dict(name="step_small_nacl_64", call="step", model="small", system="nacl", nx=2, ny=2, nz=2, stress=False),
        # small MD cell with the middle model, ragged atom count
        dict(name="step_medium_silica_249", call="step", model="medium", system="silica", nx=83, ny=1, nz=1, stress=True),
        # the headline: NVT steps of 1,944 atoms with forces and stress
        dict(name="step_medium_nacl_1944", call="step", model="medium", system="nacl", nx=9, ny=9, nz=3, stress=True),
        # force calls (list compacted, energy + forces) inside another program's loop, scalar model
        dict(name="forces_small_nacl_2744", call="forces", model="small", system="nacl", nx=7, ny=7, nz=7, stress=False),
        # five species and the largest model, ordinary size, triclinic cell
        dict(name="forces_large_alloy_1728", call="forces", model="large", system="alloy", nx=12, ny=12, nz=12, stress=True),
        # amorphous, long rows of neighbours, no order in memory
        dict(name="forces_medium_silica_10368", call="forces", model="medium", system="silica", nx=3456, ny=1, nz=1, stress=True),
        # the largest model at 13,824 atoms of a random alloy
        dict(name="forces_large_alloy_13824", call="forces", model="large", system="alloy", nx=24, ny=24, nz=24, stress=False),
        # a large cell whose whole edge list fits as one chunk
        dict(name="forces_medium_silica_36993", call="forces", model="medium", system="silica", nx=12331, ny=1, nz=1, stress=True),
        # the path of lists whose per-edge buffers do not fit the device (chunks, weights recomputed), played on a cell
        # that can be compared
        dict(name="forces_medium_nacl_17576_chunked", call="chunked", model="medium", system="nacl", nx=13, ny=13, nz=13, stress=True),
        # neighbour rebuild and compaction of a large cell
        dict(name="neighbours_nacl_110592", call="neighbours", model="medium", system="nacl", nx=24, ny=24, nz=24, stress=False),
        # a step of a run decomposed into bricks with per-layer halo exchange (all bricks on this device)
        dict(name="bricks_medium_nacl_6912", call="bricks", model="medium", system="nacl", nx=12, ny=12, nz=6, stress=True),
    ]


def _log_int(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    call = rng.choice(["evaluate", "step", "step", "forces", "forces", "forces", "chunked", "neighbours", "bricks"])
    model = rng.choice(["small", "medium", "medium", "large"])
    system = rng.choice(["nacl", "alloy", "silica"])
    if call == "chunked":                    # an option of large lists with the middle model
        model = "medium"
    if call == "neighbours":
        model = "medium"
    if call == "bricks":
        model, system = "medium", "nacl"
    # atoms: up to what the listed cases of the same call reach
    top = {"evaluate": 1500, "step": 4000, "forces": 37000 if model != "large" else 13500, "chunked": 17000,
           "neighbours": 110000, "bricks": 6800}[call]
    low = {"evaluate": 60, "step": 60, "forces": 100, "chunked": 9000, "neighbours": 500, "bricks": 2500}[call]
    atoms = _log_int(rng, low, top)
    stress = rng.random() < 0.5
    if call == "bricks":
        side = (atoms / 8 / 4) ** (1 / 3)    # about twice as wide along x and y
        nx, ny = (max(4, min(12, int(round(2 * side + rng.uniform(-1, 1))))) for _ in range(2))
        nz = max(3, min(6, int(atoms / 8 / (nx * ny))))
        return dict(call=call, model=model, system=system, nx=nx, ny=ny, nz=nz, stress=True)
    if system == "silica":
        return dict(call=call, model=model, system=system, nx=max(20, atoms // 3), ny=1, nz=1, stress=stress)
    per = 8 if system == "nacl" else 1
    side = (atoms / per) ** (1 / 3)
    least = 2 if system == "nacl" else 4
    nx = max(least, int(round(side * math.exp(rng.uniform(-0.3, 0.3)))))
    ny = max(least, int(round(side * math.exp(rng.uniform(-0.3, 0.3)))))
    nz = max(least, int(atoms / per / (nx * ny)))
    while nx * ny * nz * per > 1.05 * top and max(nx, ny, nz) > least:
        if nx >= max(ny, nz):
            nx -= 1
        elif ny >= nz:
            ny -= 1
        else:
            nz -= 1
    return dict(call=call, model=model, system=system, nx=nx, ny=ny, nz=nz, stress=stress)


# ------------------------------------------------------------------------------------------------ inputs


@functools.lru_cache(maxsize=None)
def _weights(model: str):
    return init_weights(SPECS[model], WEIGHT_SEED[model])


def _spec(case):
    return dataclasses.replace(SPECS[case["model"]], avg_num_neighbors=NEIGHBOURS[case["system"]])


def _structure(case, seed):
    shape = (case["nx"], case["ny"], case["nz"])
    if case["system"] == "nacl":
        s = nacl(shape, 0.05, seed)
    elif case["system"] == "alloy":
        s = fcc_alloy(shape, 0.1, seed)
    else:
        s = silica(case["nx"], seed=seed)
    return s.with_velocities(1000.0 if case["system"] == "alloy" else 300.0, seed + 1)


def _temperature(case):
    return 1000.0 if case["system"] == "alloy" else 300.0


BRICKS = 2


def prepare(case, seed):
    structure = _structure(case, seed)
    spec, weights, call = _spec(case), _weights(case["model"]), case["call"]
    if call == "neighbours":
        x = torch.tensor(structure.positions, dtype=torch.float64, device="cuda")
        neighbours = CellListNeighbours(structure.cell, spec.r_cut, x.device)
        neighbours.build(x)                     # the buffers a program keeps, of one size per case; each pass builds again
        atoms, degree = _sizes(case)
        neighbours.set_capacity(256 * int(1 + 1.25 * atoms * degree * ((6.0 + SKIN) / 6.0) ** 3 // 256) + 4096)
        return dict(call=call, x=x, neighbours=neighbours)
    if call == "bricks":
        return dict(call=call, simulation=DomainSimulation(spec, weights, structure, BRICKS, temperature_K=300.0, seed=seed))
    options = dict(chunk_edges=1 << 19, edge_adjoint=False) if call == "chunked" else {}
    if call in ("forces", "chunked"):
        x = torch.tensor(structure.positions, dtype=torch.float64, device="cuda")
        ff = B200ForceField(spec, weights, structure.numbers, structure.cell, compute_stress=case["stress"], positions=x,
                            **options)
        return dict(call=call, x=x, ff=ff)
    ff = B200ForceField(spec, weights, structure.numbers, structure.cell, compute_stress=case["stress"])
    if call == "evaluate":
        return dict(call=call, structure=structure, stress=case["stress"], ff=ff)
    state = SimulationState.from_structure(structure, ff.device, seed=seed, compute_stress=case["stress"])
    engine = B200Engine(ff, Langevin(state, IntegratorConfig(), temperature_K=_temperature(case)), state)
    engine.step()                               # a run in progress: the step is captured
    return dict(call=call, engine=engine, state=state)


def run(state):
    call = state["call"]
    if call == "evaluate":
        energy, forces, stress = state["ff"].evaluate(state["structure"], stress=state["stress"])
        return dict(energy=energy, forces=forces, stress=stress)
    if call in ("forces", "chunked"):
        ff = state["ff"]
        ff.compact(state["x"])
        out = ff(state["x"])
        return dict(energy=out.energy, forces=out.forces, stress=out.stress)
    if call == "step":
        state["engine"].step()
        s = state["state"]
        return dict(positions=s.positions, velocities=s.velocities, forces=s.forces, energy=s.energy, stress=s.stress)
    if call == "neighbours":
        neighbours = state["neighbours"]
        neighbours.build(state["x"])
        neighbours.compact(state["x"])
        edge_index, shifts, unit_shifts = neighbours.edges(neighbours.capacity)
        return dict(edge_index=edge_index, unit_shifts=unit_shifts, shifts=shifts, count=neighbours.count,
                    row_ptr=neighbours.edge_row_ptr)
    simulation = state["simulation"]
    simulation.step()
    positions, velocities, _ = simulation.global_state()
    forces = torch.zeros_like(positions)
    for rank in simulation.ranks:
        forces[rank.part.owned] = rank.state.forces
    return dict(positions=positions, velocities=velocities, forces=forces, energy=simulation.energy,
                stress=simulation.stress)


# ------------------------------------------------------------------------------------------------ work, tolerance


def _sizes(case):
    if case["system"] == "silica":
        return 3 * case["nx"], 60
    n = case["nx"] * case["ny"] * case["nz"] * (8 if case["system"] == "nacl" else 1)
    return n, 40 if case["system"] == "nacl" else 57     # typical neighbours within 6 Å


def work(case):
    """Bytes: inputs and outputs once (positions, species, velocities; forces; the neighbour list's pairs for a build).
    Operations of the model: per edge the radial MLPs of both layers, the last radial layer and the couplings of the
    second interaction and the outer products of the first; per atom the linears and the contraction; the gradient costs
    about twice the value."""
    n, degree = _sizes(case)
    if case["call"] == "neighbours":
        pairs = n * degree * ((6.0 + SKIN) / 6.0) ** 3
        return {"bytes": n * 28.0 + pairs * (8 + 12 + 12), "flops": n * degree * 20.0}
    lmax, c, edges = {"small": 0, "medium": 1, "large": 2}[case["model"]], 128, n * degree
    paths = {0: 4, 1: 10, 2: 17}[lmax]
    slots = {0: 16, 1: 40, 2: 71}[lmax]
    coupling = 2.0 * c * sum((2 * a + 1) * (2 * b + 1) * 1.5 for a in range(lmax + 1) for b in range(4))
    per_edge = 2 * (2.0 * (8 * 64 + 2 * 64 * 64)) + 2.0 * 64 * paths * c + coupling + 2.0 * 16 * 64
    hidden = (lmax + 1) ** 2
    per_atom = 2.0 * c * c * (16 + slots + 3 * hidden + 2) + 4.0 * c * 400 * (1 + lmax)
    flops = 3.0 * (edges * per_edge + n * per_atom)
    moved = n * (24 + 12 + 4.0) + (n * 7 * 24.0 if case["call"] in ("step", "bricks") else 0.0)
    return {"bytes": moved, "flops": flops}


def tolerance(case):
    """fp32 sums over dozens of neighbours, 128 channels and two layers: forces and stress of the random models differ
    from float64 by up to 4e-6 of their norm, energies by up to 1e-6."""
    if case["call"] == "neighbours":
        return "exact"
    return {"rel": 2e-5, "max": 8e-4}


# ------------------------------------------------------------------------------------------------ float64


def _generators(l):
    """The three rotation generators of degree l on real harmonics, in the frame the package's harmonics use: polar
    axis y for l <= 3 (the components of l = 1 are x, y, z), polar axis z above."""
    m = np.arange(-l, l + 1)
    lz = np.diag(m).astype(complex)
    up = np.zeros((2 * l + 1,) * 2, complex)
    up[np.arange(1, 2 * l + 1), np.arange(2 * l)] = np.sqrt(l * (l + 1) - m[:-1] * (m[:-1] + 1.0))
    lx, ly = (up + up.T) / 2, (up - up.T) / 2j
    real = np.zeros_like(lz)                   # rows: real harmonics, columns: complex ones
    real[l, l] = 1.0
    for k in range(1, l + 1):
        s, r = (-1.0) ** k, math.sqrt(0.5)
        real[l + k, l + k], real[l + k, l - k] = s * r, r
        real[l - k, l + k], real[l - k, l - k] = -1j * s * r, 1j * r
    x, y, z = (np.real(1j * (real @ a.T @ real.conj().T)) for a in (lx, ly, lz))
    return (y, z, x) if l <= 3 else (x, y, z)


@functools.lru_cache(maxsize=None)
def _coupling(l1, l2, l3):
    """The invariant tensor of three irreps: unit norm, first entry positive."""
    sizes = [2 * l + 1 for l in (l1, l2, l3)]
    eye = [np.eye(k) for k in sizes]
    squares = 0
    for a, b, c in zip(_generators(l1), _generators(l2), _generators(l3)):
        row = (np.kron(np.kron(a, eye[1]), eye[2]) + np.kron(np.kron(eye[0], b), eye[2])
               + np.kron(np.kron(eye[0], eye[1]), c))
        squares = squares + row.T @ row
    values, basis = np.linalg.eigh(squares)
    assert abs(values[0]) < 1e-9 and (len(values) == 1 or values[1] > 1e-3)
    t = basis[:, 0] / np.linalg.norm(basis[:, 0])
    t[np.abs(t) < 1e-12] = 0.0
    return (t if t[np.flatnonzero(np.abs(t) > 1e-9)[0]] > 0 else -t).reshape(sizes)


def _paths(lmax_in):
    """(l_in, l_edge, l_out) of the channelwise product, ordered by l_out."""
    found = [(a, b, c) for a in range(lmax_in + 1) for b in range(4) for c in range(abs(a - b), min(3, a + b) + 1)
             if (a + b + c) % 2 == 0]
    return sorted(found, key=lambda p: p[2])


@functools.lru_cache(maxsize=None)
def _trees(order, l_out):
    """Coupled products of ``order`` copies of the 16 components that end in l_out with natural parity."""
    left = []
    for l in range(4):
        block = np.zeros((2 * l + 1, 16))
        block[np.arange(2 * l + 1), l * l + np.arange(2 * l + 1)] = 1.0
        left.append((l, 0, block))              # degree, 1 where the parity is not (-1)^l, tensor
    for step in range(1, order):
        grown = []
        for la, odd, tensor in left:
            for lb in range(4):
                for lc in range(abs(la - lb), la + lb + 1):
                    new_odd = (odd + la + lb + lc) % 2
                    if step == order - 1 and (lc != l_out or new_odd):
                        continue
                    joined = np.tensordot(math.sqrt(2 * lc + 1) * _coupling(lc, la, lb), tensor, axes=([1], [0]))
                    joined = np.moveaxis(joined, 1, -1)
                    wide = np.zeros(joined.shape[:-1] + (16,))
                    wide[..., lb * lb:(lb + 1) ** 2] = joined
                    grown.append((lc, new_odd, wide))
        left = sorted(grown, key=lambda item: item[:2])
    return np.stack([t for l, odd, t in left if l == l_out and not odd])


def _harmonics(u):
    x, y, z = u.unbind(1)
    r = x * x + z * z
    zx, f = (z * z - x * x) * (math.sqrt(3) / 2), math.sqrt(3)
    a, b = math.sqrt(5 / 6), math.sqrt(3 / 8)
    l2 = [f * x * z, f * x * y, y * y - r / 2, f * y * z, zx]
    l3 = [a * (f * x * z * z + zx * x), math.sqrt(5) * f * x * z * y, b * (4 * y * y - r) * x,
          0.5 * y * (2 * y * y - 3 * r), b * z * (4 * y * y - r), math.sqrt(5) * zx * y, a * (zx * z - f * x * z * x)]
    return torch.stack([torch.ones_like(x)] + [math.sqrt(3) * v for v in (x, y, z)] + [math.sqrt(5) * v for v in l2]
                       + [math.sqrt(7) * v for v in l3], 1)


@functools.lru_cache(maxsize=None)
def _silu_scale():
    z = np.linspace(-12.0, 12.0, 240001)
    g = (z / (1 + np.exp(-z))) ** 2 * np.exp(-z * z / 2) / math.sqrt(2 * math.pi)
    return 1 / math.sqrt(float((g.sum() - (g[0] + g[-1]) / 2) * (z[1] - z[0])))


def _pairs(x, cell, cutoff):
    """(receiver, sender, shift vector) of every pair closer than the cutoff, periodic images included."""
    inverse = torch.linalg.inv(cell)
    width = 1 / torch.linalg.norm(inverse, dim=0)
    reach = [int(math.floor(cutoff / float(w))) + 1 for w in width]
    nearest = bool((width > 2 * cutoff).all())       # then only the nearest image of a pair can be in range
    base = torch.zeros(1, 3, dtype=x.dtype, device=x.device)
    if not nearest:
        # atoms may lie outside the cell: reduce the differences first, then visit the images around
        base = torch.cartesian_prod(*(torch.arange(-k, k + 1, device=x.device) for k in reach)).to(x.dtype)
    found = []
    rows = max(1, int(2e7) // len(x))
    for start in range(0, len(x), rows):
        d = x[None, :, :] - x[start:start + rows, None, :]                 # sender minus receiver
        wrap = -torch.round(d @ inverse)
        for image in base:
            s = wrap + image
            v = d + s @ cell
            hit = (v * v).sum(-1) < cutoff * cutoff
            same = (torch.arange(start, start + len(d), device=x.device)[:, None] == torch.arange(len(x), device=x.device))
            hit &= ~(same & (s == 0).all(-1))
            i, j = hit.nonzero(as_tuple=True)
            found.append((i + start, j, -s[i, j]))
    return tuple(torch.cat(parts) for parts in zip(*found))


def _model(spec, weights, x, cell, numbers, want_stress):
    """Energy, forces and stress in float64: plain torch, gradients by autograd (blocks recomputed to save memory)."""
    dev, f64, c = x.device, torch.float64, spec.channels
    w = {k: v.to(device=dev, dtype=f64) for k, v in weights.items()}
    species = torch.as_tensor(numbers, device=dev) - 1
    n = len(x)
    receiver, sender, shift = _pairs(x, cell, spec.r_cut)
    x = x.clone().requires_grad_(True)
    strain = torch.zeros(3, 3, dtype=f64, device=dev, requires_grad=True)
    sym = (strain + strain.T) / 2
    xs = x + x @ sym
    vec = xs[receiver] - xs[sender] + shift @ (cell + cell @ sym)
    r = torch.linalg.norm(vec, dim=1)
    y = _harmonics(vec / r[:, None])
    t, p, k = r / spec.r_cut, spec.cutoff_p, torch.arange(1, spec.num_bessel + 1, device=dev, dtype=f64)
    envelope = 1 - (p + 1) * (p + 2) / 2 * t ** p + p * (p + 2) * t ** (p + 1) - p * (p + 1) / 2 * t ** (p + 2)
    radial = math.sqrt(2 / spec.r_cut) * torch.sin(k * math.pi * t[:, None]) / r[:, None] * envelope[:, None]

    def silu(a):
        return _silu_scale() * torch.nn.functional.silu(a)

    def mlp(layer, a):
        for q in range(4):
            m = w[f"l{layer}.rad.{q}"]
            a = a @ m / math.sqrt(len(m))
            a = silu(a) if q < 3 else a
        return a

    def messages(layer, paths, h, yb, rb, snd, rcv):
        """The summed messages of one block of edges: one [n, 2 l + 1, C] sum per path, side by side."""
        weight = mlp(layer, rb)
        out = []
        for q, (a, b, o) in enumerate(paths):
            cg = math.sqrt(2 * o + 1) * torch.tensor(_coupling(a, b, o), device=dev)
            coupled = torch.einsum("abo,eb->eoa", cg, yb[:, b * b:(b + 1) ** 2])
            m = torch.bmm(coupled, h[snd][:, a * a:(a + 1) ** 2]) * weight[:, None, q * c:(q + 1) * c]
            out.append(torch.zeros(n, 2 * o + 1, c, dtype=f64, device=dev).index_add(0, rcv, m))
        return torch.cat(out, 1)

    def contract(layer, l_out, z, m):
        total = None
        for order in (3, 2, 1):
            u = torch.einsum("k...,kc->c...", torch.tensor(_trees(order, l_out), device=dev), w[f"l{layer}.sc.{l_out}.{order}"][z])
            mc = m.permute(2, 0, 1)                                       # [C, n, 16]
            if total is None:
                total = torch.matmul(mc, u.reshape(c, -1, 16).transpose(1, 2)).reshape(c, len(m), *u.shape[1:-1])
            else:
                total = torch.einsum("cn...i,cni->cn...", total + u[:, None], mc)
        return total.permute(1, 2, 0)                                     # [n, 2 l + 1, C]

    h = (w["emb"][species] / math.sqrt(spec.num_elements))[:, None, :]
    node = torch.zeros(n, dtype=f64, device=dev)
    for layer in range(2):
        lin_, lout = (0, spec.hidden_lmax) if layer == 0 else (spec.hidden_lmax, 0)
        block = [slice(l * l, (l + 1) ** 2) for l in range(4)]
        skip = torch.zeros(n, (lout + 1) ** 2, c, dtype=f64, device=dev)
        for l in range(min(lin_, lout) + 1):
            parts = torch.zeros(n, 2 * l + 1, c, dtype=f64, device=dev)
            for z in species.unique():
                at = (species == z).nonzero()[:, 0]
                parts = parts.index_add(0, at, h[at][:, block[l]] @ w[f"l{layer}.skip.{l}"][:, z, :])
            skip = torch.cat([skip[:, :l * l], parts / math.sqrt(c * spec.num_elements), skip[:, (l + 1) ** 2:]], 1)
        up = torch.cat([h[:, block[l]] @ w[f"l{layer}.up.{l}"] / math.sqrt(c) for l in range(lin_ + 1)], 1)
        paths, summed = _paths(lin_), 0
        size = 1 << 17
        for e in range(0, len(receiver), size):
            summed = summed + checkpoint(messages, layer, paths, up, y[e:e + size], radial[e:e + size], sender[e:e + size],
                                         receiver[e:e + size], use_reentrant=False)
        first = np.concatenate([[0], np.cumsum([2 * o + 1 for _, _, o in paths])])
        message = []
        for o in range(4):
            into = [q for q, path in enumerate(paths) if path[2] == o]
            message.append(sum(summed[:, first[q]:first[q + 1]] @ w[f"l{layer}.lin.{q}"] for q in into)
                           / math.sqrt(len(into) * c) / spec.avg_num_neighbors)
        message = torch.cat(message, 1)
        out = skip
        for l in range(lout + 1):
            part = torch.zeros(n, 2 * l + 1, c, dtype=f64, device=dev)
            for z in species.unique():
                at = (species == z).nonzero()[:, 0]
                for s in range(0, len(at), 2048):
                    rows = at[s:s + 2048]
                    part = part.index_add(0, rows, checkpoint(contract, layer, l, z, message[rows], use_reentrant=False))
            part = part @ w[f"l{layer}.prod.{l}"] / math.sqrt(c)
            out = torch.cat([out[:, :l * l], out[:, block[l]] + part, out[:, (l + 1) ** 2:]], 1)
        h = out
        if layer == 0:
            node = node + h[:, 0] @ w["l0.readout"] / math.sqrt(c)
        else:
            node = node + silu(h[:, 0] @ w["l1.readout.0"] / math.sqrt(c)) @ w["l1.readout.1"] / math.sqrt(spec.mlp_hidden)
    energy = (spec.scale * node + spec.shift).sum()
    gx, gs = torch.autograd.grad(energy, (x, strain))
    stress = (gs + gs.T) / 2 / torch.linalg.det(cell).abs() if want_stress else None
    return energy.detach().reshape(1), -gx, stress


def _langevin(case, seed, structure, forces_of):
    """Two steps of the NVT run ``prepare`` and ``run`` take together, with the host noise of the seed."""
    steps, fr, dt = 2, IntegratorConfig().friction, IntegratorConfig().timestep_fs * FS
    x, v = structure.positions.copy(), structure.velocities.copy()
    m = structure.masses[:, None]
    kt = math.sqrt(KB * _temperature(case))
    sigma = kt * np.sqrt(2 * fr / m)
    c1, c2 = dt / 2 - dt * dt * fr / 8, dt * fr / 2 - dt * dt * fr * fr / 8
    c3, c5 = sigma * (math.sqrt(dt) / 2 - dt ** 1.5 * fr / 8), sigma * dt ** 1.5 / (2 * math.sqrt(3))
    noise = np.random.default_rng(seed)
    energy, f, stress = forces_of(x)
    for _ in range(steps):
        xi, eta = noise.standard_normal((2, len(x), 3))
        rx, rv = c5 * eta, c3 * xi - fr / 2 * c5 * eta
        rx, rv = (a - (a * m).sum(0) / m.sum() for a in (rx, rv))
        v = v + c1 * f / m - c2 * v + rv
        new = x + dt * v + rx
        x, v = new, (new - x - rx) / dt
        energy, f, stress = forces_of(x)
        v = v + c1 * f / m - c2 * v + rv
    return dict(positions=x, velocities=v, forces=f, energy=energy, stress=stress)


def exact(case, seed):
    if case["call"] in ("neighbours", "bricks"):       # whole numbers; rows laid out by the decomposition
        return None
    structure, spec = _structure(case, seed), _spec(case)
    cell = torch.tensor(structure.cell, dtype=torch.float64, device="cuda")

    def forces_of(x):
        e, f, s = _model(spec, _weights(case["model"]), torch.as_tensor(x, dtype=torch.float64, device="cuda"), cell,
                         structure.numbers, case["stress"])
        return e.cpu().numpy(), f.cpu().numpy(), None if s is None else s.cpu().numpy()

    if case["call"] == "step":
        return _langevin(case, seed, structure, forces_of)
    energy, forces, stress = forces_of(structure.positions)
    if case["call"] == "evaluate":
        energy = float(energy[0])
    return dict(energy=energy, forces=forces, stress=stress)
