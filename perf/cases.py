"""The work a user of this package has it do, as cases that can be timed: energy, forces and virial of GRACE-1L / 2L / 3L
models through the public classes `System`, `Batch` and `Engine`, from single small cells (molecular dynamics or a
relaxation of a unit cell, where latency counts) to structures of a million atoms.

A case names the entry point (`api`), the model, the structure and what is asked for (`want`):

    api     system         System.compute: numpy arrays in and out, as an ASE-style calculator calls it at every step
            system_device  System.compute_device: tensors of the GPU in and out, as an MD loop on the GPU calls it
            engine         Engine.run: local and ghost atoms and a neighbour table from an MD code
            batch          Batch.compute: several structures at once, numpy arrays, buffers given back after each call
            batch_device   Batch.compute_device with kept buffers: high-throughput work on the GPU
    want    forces | energies (forces and per-atom energies) | energy_only | uq (forces and extrapolation grade)
    frames  1: the same structure again, as between two rebuilds of the neighbour list
            2: two unrelated configurations of the atoms after one another, each of which needs a new list (Monte Carlo,
               scoring a trajectory)

The models are the benchmark architectures with tables of 89 elements, written with random weights; the structures are
displaced crystals of random alloys, and for batches random triclinic cells.
"""
from __future__ import annotations

import functools
import os
import tempfile

import numpy as np
import torch

from grace_runtime_b200 import backend, modelgen, modelgen3l, structures

SKIN = 0.5
_ORDER4 = dict(modelgen.CONFIGS["1l"], max_order=4, energy_hidden=(64,))

# per model: lattice of its crystals and lattice constant; bytes of weights; flops of the dense network per atom for the
# forward pass alone and with the reverse pass; flops per bond likewise (2 lm C per message function forward, four times
# that for dE/dr and the gradient of the direction; for 3l the bond sums of two layers couple 25 harmonics with 25 message
# functions, 2 and 4 flops for each pair and channel); neighbours per atom inside 6 A
MODELS = {
    "1l": dict(lattice="bcc", a=3.2, weights=4.8e6, dense=(3.5e5, 7.4e5), bond=(1.6e3, 8.0e3), neighbours=58),
    "1l4": dict(lattice="bcc", a=3.2, weights=2.3e7, dense=(1.03e6, 2.16e6), bond=(1.6e3, 8.0e3), neighbours=58),
    "2l": dict(lattice="fcc", a=3.6, weights=2.1e7, dense=(1.40e6, 2.88e6), bond=(3.6e3, 1.8e4), neighbours=78),
    "3l": dict(lattice="bcc", a=3.2, weights=3.9e7, dense=(2.57e7, 5.30e7), bond=(1.6e5, 5.0e5), neighbours=58),
}


def _case(name, api, model, reps=(0, 0, 0), species=1, want="forces", frames=1, nsys=0, nmin=0, nmax=0):
    return dict(name=name, api=api, model=model, nx=reps[0], ny=reps[1], nz=reps[2], species=species, want=want,
                frames=frames, nsys=nsys, nmin=nmin, nmax=nmax)


def listed():
    return [
        # a unit-cell sized metal in an ASE loop: the smallest call, all latency
        _case("1l_54", "system", "1l", (3, 3, 3)),
        # the 2,000-atom tungsten supercell of the smallest benchmark configuration
        _case("1l_2k", "system", "1l", (10, 10, 10)),
        # production MD on the GPU: 128,000 atoms of a four-component alloy
        _case("1l_128k", "system_device", "1l", (40, 40, 40), species=4),
        # active learning: body order 4 and the extrapolation grade of every atom
        _case("1l4_3k_uq", "system", "1l4", (11, 12, 13), species=4, want="uq"),
        # a small alloy cell under a two-layer model
        _case("2l_108", "system", "2l", (3, 3, 3), species=3),
        # Monte Carlo: energies only, the list built anew for every configuration
        _case("2l_4k_mc", "system", "2l", (9, 10, 11), species=3, want="energy_only", frames=2),
        # the headline configuration: 1,024,000 atoms from and to host memory
        _case("2l_1m", "system", "2l", (40, 80, 80), species=3),
        # an MD code with its own list and ghost atoms, message rows exchanged through its hooks
        _case("2l_31k_engine", "engine", "2l", (19, 20, 21), species=3),
        # a few structures at once, as a workflow tool hands them over
        _case("2l_batch_24", "batch", "2l", species=89, want="energies", nsys=24, nmin=16, nmax=256),
        # high-throughput screening: the batch configuration of the benchmark
        _case("2l_batch_4096", "batch_device", "2l", species=89, nsys=4096, nmin=16, nmax=256),
        # the largest model: a small cell and the largest structure one pass keeps in memory
        _case("3l_250", "system", "3l", (5, 5, 5), species=5),
        _case("3l_31k", "system_device", "3l", (25, 25, 25), species=5),
    ]


def _log(rng, lo, hi):
    return lo * (hi / lo) ** rng.random()


def draw(rng):
    api = rng.choice(["system", "system", "system_device", "system_device", "engine", "batch", "batch_device"])
    if api.startswith("batch"):
        nsys = round(_log(rng, 4, 4096))
        nmin = rng.randint(16, 64)
        nmax = rng.randint(nmin, 256)
        want = rng.choice(["forces", "forces", "energies", "energy_only"])
        c = _case("", api, rng.choice(["1l", "2l"]), species=89, want=want, nsys=nsys, nmin=nmin, nmax=nmax)
    else:
        model = rng.choice(["1l", "2l"] if api == "engine" else ["1l", "1l4", "2l", "2l", "3l"])
        frames = 2 if api != "engine" and rng.random() < 0.25 else 1
        most = {"1l": 128000, "1l4": 64000, "2l": 1000000, "3l": 31000}[model]
        most = min(most, 32000 if api == "engine" else most) // (4 if frames == 2 else 1)
        basis = 2 if MODELS[model]["lattice"] == "bcc" else 4
        cells = _log(rng, 27, most / basis)
        edge = cells ** (1.0 / 3.0)
        nx = max(3, round(edge * (0.75 + 0.5 * rng.random())))
        ny = max(3, round(edge * (0.75 + 0.5 * rng.random())))
        nz = max(3, int(cells / (nx * ny)))
        wants = ["forces", "forces", "energies", "energy_only"] + (["uq", "uq"] if model == "1l4" else [])
        want = "forces" if api == "engine" else rng.choice(wants)
        c = _case("", api, model, (nx, ny, nz), species=rng.randint(1, 5), want=want, frames=frames)
    del c["name"]
    return c


def _atoms(case):
    if case["api"].startswith("batch"):
        return case["nsys"] * (case["nmin"] + case["nmax"]) // 2
    return case["nx"] * case["ny"] * case["nz"] * (2 if MODELS[case["model"]]["lattice"] == "bcc" else 4)


# ---- what a program has in hand ------------------------------------------------------------------------------------
@functools.lru_cache(maxsize=None)
def _file(kind):
    path = os.path.join(tempfile.mkdtemp(prefix="grace_cases_"), kind + ".npz")
    if kind == "3l":
        return modelgen3l.write_model_3l(path, elements=modelgen.ELEMENTS, lmax=4, channels=(64, 64, 64), rho_width=32,
                                         embedding=16, radial_hidden=128, energy_hidden=64, rcut=6.0, avg_neigh=58.0, seed=0)
    if kind == "1l4":
        plain = modelgen.write_model(path + ".plain.npz", elements=tuple(modelgen.ELEMENTS), seed=0, **_ORDER4)
        return modelgen.add_uq_head(plain, path, seed=0)
    return modelgen.write_config_model(path, kind, modelgen.ELEMENTS, seed=0)


@functools.lru_cache(maxsize=1)    # a program works with one model: the memory of the last one is given back
def _model(kind):
    backend.initialize(torch.cuda.current_device())
    return backend.Model(_file(kind))


def _species(k):
    return ["W"] if k == 1 else modelgen._subset(2024, k)


def _batch_structures(rng, nsys, nmin, nmax):
    """Random triclinic cells of 0.06 to 0.09 atoms per cubic Angstrom, the atoms on jittered sites of a grid so that
    none come closer than about 1.6 A; elements drawn from all 89.  The sizes are the same ones in another order."""
    natoms = rng.permutation(np.random.default_rng(nsys).integers(nmin, nmax + 1, size=nsys)).astype(np.int32)
    cells = np.zeros((nsys, 3, 3))
    positions = []
    for s, n in enumerate(int(v) for v in natoms):
        vol = n / (0.06 + 0.03 * rng.random())
        edge = vol ** (1.0 / 3.0)
        cell = np.diag(edge * (1.0 + 0.2 * (rng.random(3) - 0.5)))
        cell[1, 0], cell[2, 0], cell[2, 1] = 0.3 * edge * (rng.random(3) - 0.5)
        cell *= (vol / abs(np.linalg.det(cell))) ** (1.0 / 3.0)
        m = np.full(3, int(np.floor(n ** (1.0 / 3.0) + 1e-9)))
        while m.prod() < n:
            m[np.argmax(np.diag(cell) / m)] += 1
        site = rng.permutation(int(m.prod()))[:n]
        frac = np.stack(np.unravel_index(site, tuple(m)), 1) + 0.5 + 0.12 * (rng.random((n, 3)) - 0.5)
        positions.append(frac / m @ cell)
        cells[s] = cell
    total = int(natoms.sum())
    types = rng.integers(1, 90, size=total).astype(np.int32)
    return natoms, types, np.concatenate(positions), cells, np.ones((nsys, 3), dtype=np.uint8)


class _Rows:
    """message rows at a device address, for torch.as_tensor"""

    def __init__(self, address, rows, width):
        self.__cuda_array_interface__ = {"shape": (rows, width), "typestr": "<f4", "data": (int(address), False),
                                         "strides": None, "version": 3}


def _engine_state(case, model, species, types, pos, cell, pbc):
    """Local atoms, the ghost images their neighbours are, and the padded table of an MD code, unfolded from the
    periodic list inside the cutoff plus skin."""
    listing = backend.System(model, species, skin=SKIN)
    listing.compute(types, pos, cell, pbc, energy_only=True)
    i, j, shift = (torch.from_numpy(v).cuda() for v in listing.neighbor_list())
    n = len(types)
    key = ((shift[:, 0] + 8) * 17 + shift[:, 1] + 8) * 17 + shift[:, 2] + 8
    home = key == (8 * 17 + 8) * 17 + 8
    images, which = torch.unique(key * n + j, return_inverse=True)
    is_ghost = torch.div(images, n, rounding_mode="floor") != (8 * 17 + 8) * 17 + 8
    ghost_of = torch.cumsum(is_ghost, 0) - 1 + n
    index = torch.where(home, j, ghost_of[which]).int()
    ghosts = images[is_ghost]
    owner, k = ghosts % n, torch.div(ghosts, n, rounding_mode="floor")
    s = torch.stack([torch.div(k, 289, rounding_mode="floor"), torch.div(k, 17, rounding_mode="floor") % 17, k % 17], 1) - 8
    x = torch.from_numpy(pos).cuda()
    x = torch.cat([x, x[owner] + s.double() @ torch.from_numpy(cell).cuda()]).contiguous()
    t = torch.from_numpy(types).cuda()
    count = torch.bincount(i, minlength=n)
    width = int(count.max())
    first = torch.cumsum(count, 0) - count
    table = torch.zeros((n, width), dtype=torch.int32, device="cuda")
    order = torch.argsort(i, stable=True)
    table[i[order], torch.arange(len(i), device="cuda") - first[i[order]]] = index[order]
    nall = len(x)
    state = dict(api="engine", engine=backend.Engine(model, species), n=n, nall=nall, types=torch.cat([t, t[owner]]), x=x,
                 count=count.int(), table=table, width=width, owner=owner,
                 f=torch.zeros((nall, 3), dtype=torch.float64, device="cuda"))

    def forward(rows, floats, stream):     # the owners' message rows to their ghosts
        with torch.cuda.stream(torch.cuda.ExternalStream(stream)):
            r = torch.as_tensor(_Rows(rows, nall, floats), device="cuda")
            r[n:] = r.index_select(0, owner)

    def reverse(rows, floats, stream):     # the ghosts' gradients back to their owners
        with torch.cuda.stream(torch.cuda.ExternalStream(stream)):
            r = torch.as_tensor(_Rows(rows, nall, floats), device="cuda")
            r.index_add_(0, owner, r[n:].clone())

    two = model.layers == 2
    state.update(forward=forward if two else None, reverse=reverse if two else None)
    return state


def prepare(case, seed):
    model = _model(case["model"])
    rng = np.random.default_rng(seed)
    api, want = case["api"], case["want"]
    f64 = dict(dtype=torch.float64, device="cuda")
    ask = dict(energies=want == "energies", energy_only=want == "energy_only", uq=want == "uq")
    if api.startswith("batch"):
        natoms, types, pos, cells, pbc = _batch_structures(rng, case["nsys"], case["nmin"], case["nmax"])
        batch = backend.Batch(model, list(modelgen.ELEMENTS))
        if api == "batch":
            return dict(api=api, batch=batch, args=(natoms, types, pos, cells, pbc), ask=ask)
        batch.keep_buffers = True
        n = len(types)
        out = dict(energy=torch.zeros(len(natoms), **f64))
        if want != "energy_only":
            out.update(forces=torch.zeros((n, 3), **f64), virial=torch.zeros((len(natoms), 6), **f64))
        if want == "energies":
            out["energies"] = torch.zeros(n, **f64)
        return dict(api=api, batch=batch, out=out, energy_only=want == "energy_only",
                    args=(natoms, torch.from_numpy(types).cuda(), torch.from_numpy(pos).cuda(), cells, pbc))
    info, species = MODELS[case["model"]], _species(case["species"])
    a = 3.165 if case["species"] == 1 and info["lattice"] == "bcc" else info["a"]
    reps, sigma = (case["nx"], case["ny"], case["nz"]), 0.12 if case["frames"] == 2 else 0.08 if info["lattice"] == "fcc" else 0.05
    made = [structures.crystal(info["lattice"], a, reps, n_species=len(species), sigma=sigma, seed=int(rng.integers(1 << 31)))
            for _ in range(case["frames"])]
    types, _, cell, pbc = made[0]
    frames = [m[1] for m in made]
    if api == "engine":
        return _engine_state(case, model, species, types, frames[0], cell, pbc)
    system = backend.System(model, species, skin=SKIN)
    if api == "system":
        return dict(api=api, system=system, types=types, frames=frames, cell=cell, pbc=pbc, ask=ask)
    n, outs = len(types), []
    for _ in frames:
        out = dict(energy=torch.zeros(1, **f64))
        if want != "energy_only":
            out.update(forces=torch.zeros((n, 3), **f64), virial=torch.zeros(6, **f64))
        if want == "energies":
            out["energies"] = torch.zeros(n, **f64)
        if want == "uq":
            out.update({k: torch.zeros(n, **f64) for k in ("gamma", "atomic_sigma", "gmm_cluster")})
        outs.append(out)
    return dict(api=api, system=system, types=torch.from_numpy(types).cuda(), frames=[torch.from_numpy(x).cuda() for x in frames],
                cell=cell, pbc=pbc, outs=outs, energy_only=want == "energy_only")


def run(state):
    s = state
    if s["api"] == "system":
        return [s["system"].compute(s["types"], x, s["cell"], s["pbc"], **s["ask"]) for x in s["frames"]]
    if s["api"] == "system_device":
        for x, out in zip(s["frames"], s["outs"]):
            s["system"].compute_device(s["types"], x, s["cell"], s["pbc"], energy_only=s["energy_only"], **out)
        return s["outs"]
    if s["api"] == "batch":
        return s["batch"].compute(*s["args"], **s["ask"])
    if s["api"] == "batch_device":
        s["batch"].compute_device(*s["args"], energy_only=s["energy_only"], **s["out"])
        return s["out"]
    s["f"].zero_()                              # the engine adds to the caller's forces, on a stream of its own
    torch.cuda.current_stream().synchronize()
    energy, virial = s["engine"].run(s["n"], s["nall"], s["types"], s["x"], s["count"], s["table"], s["width"], s["f"],
                                     forward=s["forward"], reverse=s["reverse"])
    f, n = s["f"], s["n"]
    f.index_add_(0, s["owner"], f[n:].clone())  # the ghosts' forces back to their owners
    return [energy, virial, f[:n]]


def work(case):
    """Positions and types in, results out, the weights once; the dense network and the bond sums."""
    m, n, reverse = MODELS[case["model"]], _atoms(case) * case["frames"], case["want"] != "energy_only"
    per_atom = 28 + (24 if reverse else 0) + {"energies": 8, "uq": 24}.get(case["want"], 0)
    if case["api"] == "engine":
        per_atom += 4 * (m["neighbours"] + 1)
    return {"bytes": per_atom * n + m["weights"], "flops": n * (m["dense"][reverse] + m["neighbours"] * m["bond"][reverse])}


def tolerance(case):
    # fp32 networks under fp64 geometry and sums: a few 1e-6 of the forces between two orders of summation, more for the
    # distances of the extrapolation grade and through the three layers of the largest model
    return {"rel": 3e-5 if case["want"] == "uq" or case["model"] == "3l" else 1e-5}
