"""The calls this library is timed on: energy, forces and stress through its public entry points.

A case names a model (architecture, channels and the options of its file), a structure and the way a program drives the
evaluation.  Structures are the perturbed SrTiO3 supercells and the ten-element disordered solid of ``bench.py`` and the
tests, with atoms removed where the size is to be odd; models are the seeded ones of ``modelgen``.  The model file stays
the same for every seed (a program keeps its model), positions and velocities are made from the seed.

Keys of a case
    mode      calculate  ``Calculator.calculate`` on host arrays, the neighbor list is reused from call to call
              screen     the same on a list of different structures, so that every call builds a list
              committee  ``EnsembleCalculator.calculate`` over several models
              md         one velocity-Verlet step of ``NVEIntegrator`` (positions stay on the GPU)
              device     ``MACEB200.compute_positions_device`` on positions that stay on the GPU, optionally tiled
              ghosts     ``DistributedCalculator.calculate`` on one rank: owned atoms, ghost atoms, three phases
    arch      small (32x0e, 5 A), medium (128x0e+128x1o, 6 A), large (128x0e+128x1o+128x2e, 6 A)
    channels  width, 0 for the architecture's own
    options   comma-separated: agnesi, zbl, scaled (density scaling of both layers), pairs (stored pair splines)
    cells     "nx,ny,nz" SrTiO3 unit cells, or the number of atoms of the disordered solid
    drop      atoms removed from the structure
    tile      receivers per tile, 0 for the whole graph at once
    members   structures of a screen, models of a committee
    pbc       periodic axes
    fixed     True for the reproducible mode (fixed order of every sum)
"""
from __future__ import annotations

import atexit
import math
import shutil
import tempfile
from pathlib import Path

import numpy as np
import torch

from __graft_entry__ import load_package

SKIN = 0.5
TEN_ELEMENTS = (1, 6, 8, 13, 14, 22, 26, 38, 56, 79)
SOLID_DENSITY = 0.085
MODEL_SEED = 17

_models = {}
_folder = None


def _case(mode, arch, cells, **other):
    case = {"mode": mode, "arch": arch, "channels": 0, "options": "", "cells": str(cells), "drop": 0, "tile": 0,
            "members": 1, "pbc": "111", "fixed": False}
    case.update(other)
    return case


def listed():
    return [
        # one unit cell doubled along each axis: relaxations, phonon displacements and tests; launches and latency count
        _case("calculate", "medium", "2,2,2", name="cell_40"),
        # the small model on the 4x4x4 supercell, the size of a training-set structure
        _case("calculate", "small", "4,4,4", name="small_320"),
        # a data set worked through: sixteen structures of different size, a neighbor list for each
        _case("screen", "medium", "4,3,2", members=16, name="screen_16"),
        # uncertainty from three models on one structure
        _case("committee", "medium", "4,4,4", members=3, drop=3, name="committee_317"),
        # a model with the file options of the published force fields: distance transform, repulsion, density scaling
        _case("calculate", "medium", "5,6,4", options="agnesi,zbl,scaled", drop=1, name="options_599"),
        # a slab: two periodic axes, host-built list with a reference geometry
        _case("calculate", "medium", "8,8,3", pbc="110", drop=7, name="slab_953"),
        # molecular dynamics of a medium-sized cell, everything on the GPU
        _case("md", "medium", "9,8,6", name="md_2160"),
        # one rank of a decomposed run: owned atoms and ghosts, three phases
        _case("ghosts", "medium", "8,8,8", name="ghosts_2560"),
        # regression runs that ask for the same bits every time
        _case("calculate", "medium", "6,6,6", fixed=True, name="fixed_1080"),
        # the 5,000-atom supercell that the benchmark quotes
        _case("calculate", "medium", "10,10,10", name="bulk_5000"),
        # the higher-order model on the ten-element disordered solid
        _case("calculate", "large", "20000", name="solid_20000"),
        # a large cell in tiles with a reusable workspace
        _case("device", "medium", "30,30,30", tile=32768, name="tiled_135000"),
    ]


def draw(rng):
    mode = rng.choice(("calculate", "calculate", "calculate", "screen", "committee", "md", "device", "device", "ghosts"))
    arch = rng.choice(("small", "medium", "medium", "medium", "large"))
    most = {"calculate": 8000, "screen": 400, "committee": 2000, "md": 8000, "device": 60000, "ghosts": 5000}[mode]
    if arch == "large":
        most = min(most, 16000)
    least = 64 if mode in ("md", "ghosts") else 20
    atoms = math.exp(rng.uniform(math.log(least), math.log(most)))
    case = _case(mode, arch, "1,1,1")
    if arch == "large" and rng.random() < 0.5 and mode in ("calculate", "device"):
        case["cells"] = str(max(50, int(atoms)))
    else:
        edge = (atoms / 5.0) ** (1.0 / 3.0)
        sides = [max(1, round(edge * rng.uniform(0.75, 1.33))) for _ in range(3)]
        if mode == "ghosts":      # a brick has to be wider than a ghost layer's overlap with itself
            sides = [max(4, s) for s in sides]
        case["cells"] = ",".join(str(s) for s in sides)
        case["drop"] = rng.randrange(0, max(1, sides[0] * sides[1] * sides[2] // 4) + 1)
    if arch == "medium" and rng.random() < 0.25:
        case["channels"] = 64
    case["options"] = rng.choice(("", "", "", "zbl", "agnesi", "scaled", "pairs", "agnesi,zbl,scaled"))
    if case["cells"].isdigit():
        case["options"] = rng.choice(("", "zbl"))       # tables of a hundred species pairs take long to make
    elif case["options"] == "pairs" and arch != "small":
        case["options"] = ""                            # a file of a hundred megabytes takes long to write
    if mode in ("screen", "committee"):
        case["members"] = rng.randrange(2, 9 if mode == "screen" else 4)
    if mode == "device" and rng.random() < 0.5:
        case["tile"] = rng.randrange(64, 32769)
    if mode == "calculate" and "," in case["cells"] and rng.random() < 0.15:
        case["pbc"] = rng.choice(("110", "100", "000"))
    elif mode == "calculate" and arch != "large" and "scaled" not in case["options"] and atoms < 4000 and rng.random() < 0.15:
        case["fixed"] = True
    return case


# ---------------------------------------------------------------------------------------- structures and models
def _sides(case):
    return tuple(int(s) for s in case["cells"].split(","))


def _model_file(case, member=0):
    global _folder
    solid = case["cells"].isdigit()
    key = (case["arch"], case["channels"], case["options"], solid, member)
    if key not in _models:
        if _folder is None:
            _folder = tempfile.mkdtemp(prefix="sxb_cases_")
            atexit.register(shutil.rmtree, _folder, ignore_errors=True)
        on = [o for o in case["options"].split(",") if o]
        path = Path(_folder) / f"model_{len(_models)}.json"
        kwargs = {"atomic_numbers": TEN_ELEMENTS} if solid else {}
        load_package().modelgen.write_model(
            path, case["arch"], seed=MODEL_SEED + member, channels=case["channels"] or None, agnesi="agnesi" in on,
            zbl="zbl" in on, a0_scaled="scaled" in on, a1_scaled="scaled" in on,
            radial="pair-splines" if "pairs" in on else "compact", **kwargs)
        _models[key] = path
    return _models[key]


def _solid(atoms, rng):
    """Disordered solid at SOLID_DENSITY: a face-centred lattice 1.4 times as dense, a random share of its sites
    occupied, every atom displaced by up to 0.2 A along each axis (no pair closer than about 1.8 A)."""
    side = math.ceil((1.4 * atoms / 4.0) ** (1.0 / 3.0))
    length = (atoms / SOLID_DENSITY) ** (1.0 / 3.0)
    grid = np.stack(np.meshgrid(*[np.arange(side)] * 3, indexing="ij"), axis=-1).reshape(-1, 3)
    basis = np.array([[0, 0, 0], [0.5, 0.5, 0], [0.5, 0, 0.5], [0, 0.5, 0.5]])
    sites = (grid[:, None, :] + basis).reshape(-1, 3) * (length / side)
    chosen = np.sort(rng.permutation(len(sites))[:atoms])
    pos = sites[chosen] + rng.uniform(-0.2, 0.2, size=(atoms, 3))
    return pos, np.eye(3) * length, rng.integers(0, len(TEN_ELEMENTS), size=atoms).astype(np.int32)


def _structure(case, seed, sides=None):
    rng = np.random.default_rng([seed, 5])
    if case["cells"].isdigit():
        return _solid(int(case["cells"]), rng)
    pos, cell, types = load_package().modelgen.srtio3(sides or _sides(case), 0.05, seed)
    if case["drop"]:
        keep = np.sort(rng.permutation(len(pos))[case["drop"]:])
        pos, types = pos[keep], types[keep]
    return pos, cell, types


def _screen_sides(case):
    """Sizes of the structures of a screen: the given cell with its axes lengthened one after the other."""
    sides = list(_sides(case))
    out = []
    for i in range(case["members"]):
        out.append((sides[0] + (i % 3 == 1), sides[1] + (i % 4 == 2), sides[2] + (i % 2)))
    return out


def prepare(case, seed):
    pkg = load_package()
    mode = case["mode"]
    pbc = tuple(c == "1" for c in case["pbc"])
    if mode == "screen":
        structures = [_structure(case, 1000 * seed + i, sides) for i, sides in enumerate(_screen_sides(case))]
        return {"mode": mode, "calc": pkg.Calculator(_model_file(case), skin=SKIN), "structures": structures}
    pos, cell, types = _structure(case, seed)
    state = {"mode": mode, "pos": pos, "cell": cell, "types": types, "pbc": pbc}
    if mode == "committee":
        state["calc"] = pkg.EnsembleCalculator([_model_file(case, m) for m in range(case["members"])], skin=SKIN)
        state["calc"].calculate(pos, cell, types, pbc)
    elif mode == "calculate":
        calc = pkg.Calculator(_model_file(case), skin=SKIN)
        if case["fixed"]:
            calc.evaluator.set_deterministic(True)
        calc.calculate(pos, cell, types, pbc)
        state["calc"] = calc
        # the call that is timed moves the atoms a little, so that the list is reused as it is in a relaxation
        state["pos"] = pos + np.random.default_rng([seed, 6]).uniform(-0.05, 0.05, size=pos.shape)
    elif mode == "md":
        ev = pkg.MACEB200(_model_file(case))
        masses = np.array([pkg.md.MASSES[z] for z in (8, 22, 38)])[types]
        velocities = pkg.md.maxwell_boltzmann(masses, 300.0, seed)
        state["md"] = pkg.md.NVEIntegrator(ev, pos, cell, types, masses, velocities, dt_fs=1.0, skin=SKIN)
    elif mode == "device":
        ev = pkg.MACEB200(_model_file(case))
        ev.set_tile_size(case["tile"])
        result = ev._prepare_periodic_factorized_graph(types, pos, cell, np.linalg.inv(cell), ev.r_cut + SKIN)
        state.update(ev=ev, generation=result["generation"], device_pos=torch.from_numpy(pos).cuda())
    elif mode == "ghosts":
        calc = pkg.distributed.DistributedCalculator(_model_file(case), pkg.MACEB200, skin=SKIN)
        calc.prepare(pos, cell, types, (1, 1, 1))
        state["calc"] = calc
        state["owned"] = calc.owned_positions.clone()
    return state


def _view(pointer, count, like):
    class Array:
        __cuda_array_interface__ = {"shape": (count,), "typestr": "<f8", "data": (int(pointer), False), "version": 2}

    return torch.as_tensor(Array(), device=like.device)


def run(state):
    mode = state["mode"]
    if mode == "screen":
        return [state["calc"].calculate(*structure) for structure in state["structures"]]
    if mode in ("calculate", "committee"):
        return state["calc"].calculate(state["pos"], state["cell"], state["types"], state["pbc"])
    if mode == "md":
        md = state["md"]
        energy = md.step()
        return {"energy": energy, "positions": md.x, "velocities": md.v, "forces": md.f}
    if mode == "device":
        ev, n = state["ev"], len(state["pos"])
        ev.compute_positions_device(state["generation"], state["device_pos"].data_ptr())
        _energy, forces, virial = ev.device_results()
        # copies, as the integrator takes them: the evaluator's buffers hold the next result soon, and go with it
        return {"energy": ev.energy, "forces": _view(forces, 3 * n, state["device_pos"]).clone(),
                "virial": _view(virial, 9, state["device_pos"]).clone()}
    out = state["calc"].calculate(state["owned"])
    return {"energy": out["energy"], "stress": out["stress"], "forces": out["forces"].clone()}


# ---------------------------------------------------------------------------------------- work and tolerance
_SHAPE = {  # arch: channels, cutoff, hidden components, paths, rows, output components, monomials, source components over the paths
    "small": (32, 5.0, 1, 4, 16, 16, 188, 4),
    "medium": (128, 6.0, 4, 10, 88, 40, 516, 22),
    "large": (128, 6.0, 9, 17, 243, 71, 981, 57),
}


def _atoms_and_edges(case):
    """(atoms, edges in the list, edges inside the cutoff) over everything one pass evaluates."""
    r_cut = _SHAPE[case["arch"]][1]
    if case["cells"].isdigit():
        atoms, density = int(case["cells"]), SOLID_DENSITY
    else:
        cells = [_sides(case)] if case["mode"] != "screen" else _screen_sides(case)
        full = sum(5 * a * b * c for a, b, c in cells)
        atoms = full - case["drop"] * len(cells)
        density = 5.0 / 3.905 ** 3 * atoms / full
    neighbors = 4.0 / 3.0 * math.pi * density * r_cut ** 3
    listed_share = ((r_cut + SKIN) / r_cut) ** 3
    members = case["members"] if case["mode"] == "committee" else 1
    return atoms * members, atoms * members * neighbors * listed_share, atoms * members * neighbors


def work(case):
    C, _r, NH, NP, NR, NE, monomials, sources = _SHAPE[case["arch"]]
    C = case["channels"] or C
    atoms, edges, active = _atoms_and_edges(case)
    elements = len(TEN_ELEMENTS) if case["cells"].isdigit() else 3
    # per active edge: layer 0 on the 64 radial basis functions (value; value and slope in the reverse pass) times 16
    # harmonics, layer 1 per channel: radial cubics, coupling rows (once forward, twice in reverse)
    per_edge = 2.0 * 64 * 16 * 3 + C * 2.0 * (3 * NP + sources + NR + 5 * NP + 2 * sources + 2 * NR)
    # per atom: contraction (one multiply-add per monomial forward, three in reverse), linears (forward and reverse)
    per_atom = C * 2.0 * 4 * monomials + 2 * 2.0 * C * C * (NH + NE + 2) + 2 * 2.0 * 64 * 16 * C
    weights = 4.0 * (C * C * (round(math.sqrt(NH)) + 10 + 2 * elements) + elements * monomials * C + 255 * 4 * 64 * 2
                     + 64 * C * (NP + 4 * elements * elements))
    # positions, types and graph (source and image of every edge) in, energies and forces out
    return {"bytes": atoms * (24 + 4 + 32) + edges * 16 + weights, "flops": active * per_edge + atoms * per_atom}


def tolerance(case):
    # against the float64 oracle on small systems of every architecture: energies 1e-6, forces 3e-6 (largest 1.3e-5 of
    # the root mean square), stress 3e-6, total energies 7e-6 where the atoms' energies nearly cancel; four times that
    return {"rel": 3e-5, "max": 6e-5}
