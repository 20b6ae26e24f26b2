"""GPU parity tests: the CUDA path through the C ABI against the oracles on identical inputs.

Tolerances of the force path: |dE| <= 1e-5 eV/atom, |dF| <= 1e-4 eV/A per component,
|dsigma| <= 1e-6 eV/A^3; the neighbor list must be bit-exact.
"""
import json
from pathlib import Path

import numpy as np
import pytest

from conftest import csr_from_positions
from oracle import mace_numpy, neighbor, ref

pytestmark = pytest.mark.gpu

TOL_E, TOL_F, TOL_S = 1e-5, 1e-4, 1e-6

STAGES = ["A0", "M0", "H1", "Phi1", "A1", "M1", "H2", "H2_adj", "A1_adj", "dPhi1", "H1_adj", "M0_adj", "A0_adj"]


def _edge_set(first, src, shifts):
    recv = np.repeat(np.arange(len(first) - 1), np.diff(first))
    return np.stack([recv, src, shifts[:, 0], shifts[:, 1], shifts[:, 2]], axis=1)


@pytest.mark.parametrize("n,sigma,cutoff,seed", [(3, 0.05, 5.5, 0), (4, 0.05, 5.5, 1), (4, 0.3, 6.5, 2), (2, 0.05, 6.5, 3)])
def test_neighbor_graph_bit_exact(pkg, model_path, n, sigma, cutoff, seed):
    pos, cell, types = pkg.modelgen.srtio3(n, sigma, seed)
    ev = pkg.MACEB200(model_path("small"))
    res = ev._prepare_periodic_factorized_graph(types, pos, cell, np.linalg.inv(cell), cutoff)
    first, src, shifts = ev.graph(res["generation"])
    ofirst, osrc, oshifts = neighbor.build_neighbor_graph(pos, cell, cutoff)
    assert res["num_edges"] == len(osrc)
    # identical order, not only identical sets
    assert np.array_equal(first, ofirst)
    assert np.array_equal(src, osrc)
    assert np.array_equal(shifts, oshifts)


def test_neighbor_graph_triclinic_and_wrapped(pkg, model_path):
    rng = np.random.default_rng(7)
    cell = np.array([[9.0, 0.0, 0.0], [2.5, 8.0, 0.0], [-1.0, 1.5, 10.0]])
    pos = rng.random((60, 3)) @ cell + rng.integers(-2, 3, size=(60, 3)) @ cell  # atoms outside the home cell
    types = rng.integers(0, 3, size=60).astype(np.int32)
    ev = pkg.MACEB200(model_path("small"))
    res = ev._prepare_periodic_factorized_graph(types, pos, cell, np.linalg.inv(cell), 4.0)
    first, src, shifts = ev.graph(res["generation"])
    ofirst, osrc, oshifts = neighbor.build_neighbor_graph(pos, cell, 4.0)
    assert np.array_equal(first, ofirst) and np.array_equal(src, osrc) and np.array_equal(shifts, oshifts)
    brute = neighbor.brute_force_edges(pos, cell, 4.0, max_image=6)
    mine = set(map(tuple, _edge_set(first, src, shifts).tolist()))
    assert mine == brute


NEIGHBOR_EDGES = [("lattice", 8, 4.0), ("lattice", 10, 4.0), ("lattice", 12, 4.0), ("lattice", 14, 4.0), ("lattice", 8, 3.999),
                  ("one", 1, 7.0), ("skewed", 1, 3.0), ("skewed", 40, 3.0), ("skewed", 700, 5.0), ("slab", 90, 6.5)]


@pytest.mark.parametrize("kind,n,cutoff", NEIGHBOR_EDGES)
def test_neighbor_graph_where_the_stencil_is_cut_short(pkg, model_path, kind, n, cutoff):
    """Bins that a receiver's neighbors cannot reach are passed over and rows are dealt to 8, 4, 2 or 1 warps (592, 1,184 and
    2,368 receivers): atoms exactly on the planes between bins with pairs exactly at the cutoff, cells far smaller than the
    cutoff, strongly skewed cells, flat cells.  Bit for bit, order included."""
    rng = np.random.default_rng(n)
    if kind == "lattice":                    # spacing 2, bins of exactly one cutoff
        pos = 2.0 * np.stack(np.meshgrid(*[np.arange(n)] * 3, indexing="ij"), axis=-1).reshape(-1, 3)
        cell = 2.0 * n * np.eye(3)
    elif kind == "one":
        pos, cell = np.array([[0.3, -0.2, 9.0]]), np.diag([2.0, 2.5, 30.0])
    else:
        cell = {"skewed": np.array([[6.0, 0.0, 0.0], [5.5, 7.0, 0.0], [-6.5, 5.0, 8.0]]) * max(1.0, (n / 40.0) ** (1 / 3)),
                "slab": np.array([[22.0, 0.0, 0.0], [9.0, 18.0, 0.0], [1.0, 2.0, 3.5]])}[kind]
        pos = rng.random((n, 3)) @ cell
    types = rng.integers(0, 3, size=len(pos)).astype(np.int32)
    ev = pkg.MACEB200(model_path("small"))
    res = ev._prepare_periodic_factorized_graph(types, pos, cell, np.linalg.inv(cell), cutoff)
    first, src, shifts = ev.graph(res["generation"])
    ofirst, osrc, oshifts = neighbor.build_neighbor_graph(pos, cell, cutoff)
    assert np.array_equal(first, ofirst) and np.array_equal(src, osrc) and np.array_equal(shifts, oshifts)


@pytest.mark.parametrize("far", [1e12, -1e12, 1e300, -1e300, float("nan"), float("-inf")])
def test_neighbor_graph_refuses_positions_it_cannot_wrap(pkg, model_path, far):
    """A coordinate whose count of cells does not fit 32 bits (a diverged trajectory is full of them) is an error like one that
    is not finite, on either side of the cell; the evaluator stays usable.  A million cells away is still the same crystal."""
    pos, cell, types = pkg.modelgen.srtio3(2, 0.05, 4)
    ev = pkg.MACEB200(model_path("small"))
    inverse = np.linalg.inv(cell)
    bad = pos.copy()
    bad[7, 1] = far
    with pytest.raises(ValueError, match="positions"):
        ev._prepare_periodic_factorized_graph(types, bad, cell, inverse, 5.5)
    edges = ev._prepare_periodic_factorized_graph(types, pos, cell, inverse, 5.5)["num_edges"]
    moved = pos + np.array([1e6, -1e6, 0.0]) @ cell
    assert abs(ev._prepare_periodic_factorized_graph(types, moved, cell, inverse, 5.5)["num_edges"] - edges) <= 2


# with density scaling the device keeps Phi1 already divided by 1 + rho and A1_adj / dPhi1 / A0_adj
# not yet divided (the division is folded into the next kernel's load), so those stages differ by
# design from the serial evaluator's intermediates and are left to the energy / force comparison
SCALED_STAGES = ["A0", "M0", "H1", "A1", "M1", "H2", "H2_adj", "H1_adj", "M0_adj"]


@pytest.mark.parametrize("arch,n,scaled", [("small", 3, False), ("medium", 2, False), ("medium", 2, True), ("small", 3, True), ("large", 2, False), ("large", 2, True)])
def test_stage_tensors_match_oracle(pkg, model_path, arch, n, scaled):
    path = model_path(arch, a0_scaled=scaled, a1_scaled=scaled)
    pos, cell, types = pkg.modelgen.srtio3(n, 0.05, 11)
    cutoff = pkg.modelgen.ARCHITECTURES[arch]["r_cut"]
    first, src, shifts, xyz = csr_from_positions(pos, cell, cutoff)
    ev = pkg.MACEB200(path)
    ev.compute_node_energies_forces(len(pos), types, np.diff(first), src, types[src], xyz)
    oracle = mace_numpy.NumpyMACE(str(path))
    oracle.compute(types, first, src, xyz)
    for name in (SCALED_STAGES if scaled else STAGES):
        got = ev.stage(name)
        want = oracle.stage[name].reshape(-1)
        scale = max(1.0, np.abs(want).max())
        assert np.abs(got - want).max() <= 2e-5 * scale, name
    de = np.abs(ev.node_energies - oracle.stage["node_energies"]).max()
    df = np.abs(ev.node_forces.reshape(-1, 3) - oracle.stage["node_forces"]).max()
    assert de <= TOL_E and df <= TOL_F


@pytest.mark.parametrize("arch,n,seed,scaled,zbl,agnesi", [("small", 4, 0, False, False, False), ("medium", 3, 1, False, False, False),
                                                           ("medium", 3, 2, True, False, False), ("large", 2, 3, False, False, False),
                                                           ("small", 3, 4, False, True, False), ("medium", 2, 5, True, True, False),
                                                           ("small", 3, 6, False, False, True), ("medium", 2, 7, True, True, True),
                                                           ("large", 2, 8, False, False, True)])
def test_energy_forces_stress_vs_reference_evaluator(pkg, model_path, arch, n, seed, scaled, zbl, agnesi):
    """Against the reference's own serial evaluator (MACECPU<double> and <float>)."""
    if not ref.available():
        pytest.skip("oracle/_ref was not built")
    path = model_path(arch, a0_scaled=scaled, a1_scaled=scaled, zbl=zbl, agnesi=agnesi)
    pos, cell, types = pkg.modelgen.srtio3(n, 0.05, seed)
    calc = pkg.Calculator(path, skin=0.5)
    out = calc.calculate(pos, cell, types)
    r_cut = calc.evaluator.r_cut
    # exact-cutoff graph for the reference (skin edges contribute exactly zero on the device path)
    first, src, shifts, xyz = csr_from_positions(pos, cell, r_cut)
    volume = abs(np.linalg.det(cell))
    for double in (True, False):
        m = ref.ReferenceMACE(str(path), double=double)
        m.compute(types, np.diff(first), src, xyz)
        F, S = ref.reduce_forces_stress(len(pos), np.diff(first), src, m.get("node_forces"), xyz, volume)
        e = m.get("node_energies")
        assert abs(out["energy"] - e.sum()) / len(pos) <= TOL_E
        assert np.abs(out["energies"] - e).max() <= TOL_E
        assert np.abs(out["forces"] - F).max() <= TOL_F
        assert np.abs(out["stress"] - S).max() <= TOL_S


def _reference_efs(path, pos, cell, types, r_cut, double=False):
    """Energy per node, atom forces and stress of the reference's serial evaluator on the exact-cutoff graph."""
    first, src, shifts, xyz = csr_from_positions(pos, cell, r_cut)
    m = ref.ReferenceMACE(str(path), double=double)
    m.compute(types, np.diff(first), src, xyz)
    F, S = ref.reduce_forces_stress(len(pos), np.diff(first), src, m.get("node_forces"), xyz, abs(np.linalg.det(cell)))
    return m.get("node_energies"), F, S


def _assert_matches_reference(out, e, F, S, natoms, node_tol=TOL_E):
    assert abs(out["energy"] - e.sum()) / natoms <= TOL_E
    assert np.abs(out["energies"] - e).max() <= node_tol
    assert np.abs(out["forces"] - F).max() <= TOL_F
    assert np.abs(out["stress"] - S).max() <= TOL_S


@pytest.mark.parametrize("arch,n,scaled,zbl", [("small", 3, False, False), ("small", 2, True, True), ("medium", 2, False, False)])
def test_pair_spline_models_vs_reference_evaluator(pkg, model_path, arch, n, scaled, zbl):
    """The stored pair-spline radial representation (nodal values and derivatives per unordered element
    pair instead of radial networks), with and without density splines and the pair repulsion."""
    if not ref.available():
        pytest.skip("oracle/_ref was not built")
    path = model_path(arch, seed=23, radial="pair-splines", num_spline_points=96, a0_scaled=scaled, a1_scaled=scaled, zbl=zbl)
    pos, cell, types = pkg.modelgen.srtio3(n, 0.05, 29)
    calc = pkg.Calculator(path, skin=0.5)
    out = calc.calculate(pos, cell, types)
    for double in (True, False):
        e, F, S = _reference_efs(path, pos, cell, types, calc.evaluator.r_cut, double=double)
        _assert_matches_reference(out, e, F, S, len(pos))


@pytest.mark.parametrize("arch,n,kwargs", [("small", 3, {}), ("medium", 2, {"a0_scaled": True}), ("large", 2, {"zbl": True}),
                                           ("small", 2, {"radial": "pair-splines", "num_spline_points": 96})])
def test_single_layer_models_vs_reference_evaluator(pkg, model_path, arch, n, kwargs):
    """Models with one interaction (single_layer_readout): the readout polynomial acts on H1 and there is no second
    message step (libsymmetrix/source/mace.cpp:265-283), for hidden irreps up to l = 0, 1 and 2; untiled and tiled."""
    if not ref.available():
        pytest.skip("oracle/_ref was not built")
    path = model_path(arch, seed=41, single_layer=True, **kwargs)
    pos, cell, types = pkg.modelgen.srtio3(n, 0.05, 43)
    calc = pkg.Calculator(path, skin=0.5)
    assert calc.evaluator.single_layer_readout
    out = calc.calculate(pos, cell, types)
    for double in (True, False):
        e, F, S = _reference_efs(path, pos, cell, types, calc.evaluator.r_cut, double=double)
        _assert_matches_reference(out, e, F, S, len(pos))
    tiled = pkg.Calculator(path, skin=0.5)
    tiled.evaluator.set_tile_size(16)
    out_tiled = tiled.calculate(pos, cell, types)
    _assert_matches_reference(out_tiled, e, F, S, len(pos))
    with pytest.raises(ValueError):
        rep = pkg.MACEB200(path)
        rep.set_deterministic(True)
        rep._prepare_periodic_factorized_graph(types, pos, cell, np.linalg.inv(cell), rep.r_cut + 0.5)


@pytest.mark.parametrize("arch,n,kwargs", [("small", 3, {}), ("medium", 2, {"a0_scaled": True, "a1_scaled": True}),
                                           ("medium", 2, {"radial": "pair-splines", "num_spline_points": 64}),
                                           ("small", 2, {"single_layer": True})])
def test_old_basis_models_vs_reference_evaluator(pkg, model_path, arch, n, kwargs):
    """Format version 2 (and 1): the first readout and the H1 -> H2 skip act on the scalar block of H1, after the linear
    (libsymmetrix/source/h1_affine_schema.hpp:5-30, mace.cpp:2516-2557); untiled and tiled.  The reference's own float and
    double evaluators differ by up to 8e-6 eV in single node energies on these models, hence the wider per-node bound."""
    if not ref.available():
        pytest.skip("oracle/_ref was not built")
    path = model_path(arch, seed=71, format_version=2, **kwargs)
    pos, cell, types = pkg.modelgen.srtio3(n, 0.05, 29 if n == 3 else 43)
    calc = pkg.Calculator(path, skin=0.5)
    assert calc.evaluator.h1_affine_mode == "legacy"
    out = calc.calculate(pos, cell, types)
    e, F, S = _reference_efs(path, pos, cell, types, calc.evaluator.r_cut, double=True)
    _assert_matches_reference(out, e, F, S, len(pos), node_tol=3e-5)
    tiled = pkg.Calculator(path, skin=0.5)
    tiled.evaluator.set_tile_size(16)
    _assert_matches_reference(tiled.calculate(pos, cell, types), e, F, S, len(pos), node_tol=3e-5)


@pytest.mark.parametrize("arch,n,kwargs", [("small", 3, {}), ("medium", 2, {"first_residual": True}),
                                           ("large", 2, {"first_residual": True, "a0_scaled": True, "a1_scaled": True})])
def test_pre_linear_up_models_vs_reference_evaluator(pkg, model_path, arch, n, kwargs):
    """Format 4 in the pre_linear_up basis: the first readout and the skip act on x = M0[l=0] P0 (+ the scalar block of the
    first-interaction residual), and an element-dependent constant R U joins H1 (libsymmetrix/source/mace.cpp:1759-1888);
    untiled and tiled."""
    if not ref.available():
        pytest.skip("oracle/_ref was not built")
    path = model_path(arch, seed=61, pre_linear_up=True, **kwargs)
    pos, cell, types = pkg.modelgen.srtio3(n, 0.05, 63)
    calc = pkg.Calculator(path, skin=0.5)
    assert calc.evaluator.h1_affine_mode == "pre_linear_up"
    out = calc.calculate(pos, cell, types)
    e, F, S = _reference_efs(path, pos, cell, types, calc.evaluator.r_cut, double=True)
    _assert_matches_reference(out, e, F, S, len(pos), node_tol=3e-5)
    tiled = pkg.Calculator(path, skin=0.5)
    tiled.evaluator.set_tile_size(16)
    _assert_matches_reference(tiled.calculate(pos, cell, types), e, F, S, len(pos), node_tol=3e-5)


GOLDEN = Path(__file__).resolve().parent / "golden"
GOLDEN_CASES = {"small": ("small", {}), "medium": ("medium", {}), "medium_scaled": ("medium", {"a0_scaled": True, "a1_scaled": True}),
                "large": ("large", {}), "small_zbl": ("small", {"zbl": True}),
                "small_scaled_zbl_agnesi": ("small", {"a0_scaled": True, "a1_scaled": True, "zbl": True, "agnesi": True})}
GOLDEN_CASES.update({"variant_" + k: tuple(v) for k, v in json.loads((GOLDEN / "variants.json").read_text()).items()
                     if not k.startswith("_")})


@pytest.mark.parametrize("name", sorted(GOLDEN_CASES))
def test_committed_golden_vectors_of_the_reference_evaluator(pkg, model_path, name):
    """Energies, forces and stress against the committed vectors of the reference's MACECPU<double> (tests/golden/,
    written by make_golden.py): the standard models and every model-file variant; needs no reference build."""
    arch, kwargs = GOLDEN_CASES[name]
    g = np.load(GOLDEN / f"reference_evaluator_{name}.npz")
    path = model_path(arch, seed=101, **kwargs)
    pos, cell, types = pkg.modelgen.srtio3(2, 0.05, 202)
    assert np.array_equal(pos, g["positions"])
    out = pkg.Calculator(path, skin=0.5).calculate(pos, cell, types)
    xyz = neighbor.edge_vectors(pos, cell, g["first"], g["sources"], g["shifts"])
    F, S = ref.reduce_forces_stress(len(pos), np.diff(g["first"]), g["sources"], g["edge_forces"], xyz, abs(np.linalg.det(cell)))
    # bounds: the tolerances of the force path, or eight times the deviation of the reference's own float evaluator
    # from these double vectors on the same input (stored beside them), whichever is larger: on a 40-atom cell the
    # FP32 resolution of the model itself can come close to the stress tolerance
    floor = 8.0 * g["float_deviation"]
    assert abs(out["energy"] - g["node_energies"].sum()) / len(pos) <= TOL_E
    assert np.abs(out["energies"] - g["node_energies"]).max() <= max(TOL_E, floor[0])
    assert np.abs(out["forces"] - F).max() <= max(TOL_F, floor[1])
    assert np.abs(out["stress"] - S).max() <= max(TOL_S, floor[2])


def test_headline_configuration_vs_reference_evaluator(pkg, model_path):
    """The configuration the throughput is quoted on, at full size: OMAT-0-medium architecture,
    10x10x10 SrTiO3 (5,000 atoms, sigma 0.05 A), 0.5 A skin, against MACECPU<float>."""
    if not ref.available():
        pytest.skip("oracle/_ref was not built")
    path = model_path("medium", seed=17)
    pos, cell, types = pkg.modelgen.srtio3(10, 0.05, 17)
    calc = pkg.Calculator(path, skin=0.5)
    out = calc.calculate(pos, cell, types)
    e, F, S = _reference_efs(path, pos, cell, types, calc.evaluator.r_cut)
    _assert_matches_reference(out, e, F, S, len(pos))


DISORDERED_ELEMENTS = (1, 6, 8, 13, 14, 22, 26, 38, 56, 79)


def test_disordered_ten_element_solid_vs_reference_evaluator(pkg, model_path):
    """Hidden irreps 0e+1o+2e, ten elements, a 2,000-atom cut of the seeded Poisson-disk solid
    (0.085 atoms/A^3, 1.8 A minimum separation: irregular neighbor counts) against MACECPU<float>."""
    if not ref.available():
        pytest.skip("oracle/_ref was not built")
    path = model_path("large", seed=17, atomic_numbers=DISORDERED_ELEMENTS)
    pos, cell, types = pkg.modelgen.random_solid(2000, 0.085, 1.8, len(DISORDERED_ELEMENTS), 17)
    calc = pkg.Calculator(path, skin=0.5)
    out = calc.calculate(pos, cell, types)
    assert len(np.unique(types)) == len(DISORDERED_ELEMENTS)
    e, F, S = _reference_efs(path, pos, cell, types, calc.evaluator.r_cut)
    _assert_matches_reference(out, e, F, S, len(pos))


@pytest.mark.parametrize("arch,options", [("medium", {}), ("small", dict(a0_scaled=True, a1_scaled=True, zbl=True, agnesi=True))])
def test_inactive_element_slots(pkg, model_path, arch, options):
    """A model with ten element slots of which three non-adjacent ones (1, 4, 8) occur in the
    structure: the active-type tables must skip the unused slots."""
    if not ref.available():
        pytest.skip("oracle/_ref was not built")
    path = model_path(arch, seed=5, atomic_numbers=DISORDERED_ELEMENTS, **options)
    pos, cell, base_types = pkg.modelgen.srtio3(3, 0.05, 9)
    types = np.array([1, 4, 8], dtype=np.int32)[base_types]
    calc = pkg.Calculator(path, skin=0.5)
    out = calc.calculate(pos, cell, types)
    for double in (True, False):
        e, F, S = _reference_efs(path, pos, cell, types, calc.evaluator.r_cut, double=double)
        _assert_matches_reference(out, e, F, S, len(pos))
    # a second structure that uses other slots on the same evaluator: the tables are rebuilt
    types2 = np.array([0, 9, 4], dtype=np.int32)[base_types]
    out2 = calc.calculate(pos, cell, types2)
    e, F, S = _reference_efs(path, pos, cell, types2, calc.evaluator.r_cut)
    _assert_matches_reference(out2, e, F, S, len(pos))


def test_multi_head_model_uses_the_selected_head(pkg, model_path, tmp_path):
    """Two prediction heads: the default head against the reference's evaluator (which applies the
    same selection), and the other head gives a different energy."""
    if not ref.available():
        pytest.skip("oracle/_ref was not built")
    path = model_path("small", seed=8, heads=("pbe", "omat"), zbl=True)
    pos, cell, types = pkg.modelgen.srtio3(3, 0.05, 2)
    calc = pkg.Calculator(path, skin=0.5)
    assert calc.evaluator.head == "omat" and calc.evaluator.selected_head == "omat"
    assert calc.evaluator.available_heads == ["pbe", "omat"] and calc.evaluator.supports_factorized
    out = calc.calculate(pos, cell, types)
    e, F, S = _reference_efs(path, pos, cell, types, calc.evaluator.r_cut)
    _assert_matches_reference(out, e, F, S, len(pos))
    other = pkg.Calculator(path, skin=0.5, head="pbe").calculate(pos, cell, types)
    assert abs(other["energy"] - out["energy"]) > 1e-3


def test_tiny_systems_and_isolated_atoms(pkg, model_path):
    """3..9 atoms (tile-boundary sizes of the reference's tests) and an atom with no neighbors."""
    path = model_path("small")
    oracle = mace_numpy.NumpyMACE(str(path))
    rng = np.random.default_rng(3)
    for natoms in (3, 4, 5, 8, 9):
        cell = np.eye(3) * 14.0
        pos = rng.random((natoms, 3)) * 5.0 + 1.0
        pos[0] = [12.0, 12.0, 12.0] if natoms > 3 else pos[0]   # far from the others: empty neighbor list
        # keep a sane minimum distance
        for i in range(1, natoms):
            while i > 0 and np.min(np.linalg.norm(pos[:i] - pos[i], axis=1)) < 1.5:
                pos[i] = rng.random(3) * 5.0 + 1.0
        types = rng.integers(0, 3, size=natoms).astype(np.int32)
        calc = pkg.Calculator(path, skin=0.5)
        out = calc.calculate(pos, cell, types)
        first, src, shifts = neighbor.build_neighbor_graph(pos, cell, calc.evaluator.r_cut + 0.5)
        e, energies, F, S = oracle.energy_forces_stress(types, pos, cell, first, src, shifts)
        assert abs(out["energy"] - e) / natoms <= TOL_E
        assert np.abs(out["forces"] - F).max() <= TOL_F
        assert np.abs(out["stress"] - S).max() <= TOL_S


def test_skin_graph_matches_exact_graph_and_is_reused(pkg, model_path):
    """Skin 0.5 vs exact graph, and no rebuild after a 0.1 A move
    (reference: symmetrix/test/test_mace_streamed_edges.py:4592-4676)."""
    path = model_path("small")
    pos, cell, types = pkg.modelgen.srtio3(3, 0.05, 2)
    skin = pkg.Calculator(path, skin=0.5)
    exact = pkg.Calculator(path, skin=0.0)
    a, b = skin.calculate(pos, cell, types), exact.calculate(pos, cell, types)
    assert abs(a["energy"] - b["energy"]) / len(pos) <= 1e-6
    assert np.abs(a["forces"] - b["forces"]).max() <= 1e-5
    moved = pos + np.random.default_rng(0).normal(scale=0.03, size=pos.shape)
    a2 = skin.calculate(moved, cell, types)
    assert skin.rebuilds == 1
    b2 = pkg.Calculator(path, skin=0.0).calculate(moved, cell, types)
    assert abs(a2["energy"] - b2["energy"]) / len(pos) <= 1e-6
    assert np.abs(a2["forces"] - b2["forces"]).max() <= 1e-5


def test_stale_generation_and_bad_inputs_raise(pkg, model_path):
    ev = pkg.MACEB200(model_path("small"))
    pos, cell, types = pkg.modelgen.srtio3(2, 0.05, 0)
    with pytest.raises(ValueError):
        ev._compute_prepared_factorized_positions(1, pos)            # nothing prepared
    res = ev._prepare_periodic_factorized_graph(types, pos, cell, np.linalg.inv(cell), 5.5)
    ev._compute_prepared_factorized_positions(res["generation"], pos)
    res2 = ev._prepare_periodic_factorized_graph(types, pos, cell, np.linalg.inv(cell), 5.5)
    assert res2["generation"] > res["generation"]
    with pytest.raises(ValueError):
        ev._compute_prepared_factorized_positions(res["generation"], pos)   # stale token
    with pytest.raises(ValueError):
        ev._prepare_periodic_factorized_graph(types, pos, cell, np.linalg.inv(cell) * 2.0, 5.5)  # inconsistent inverse
    with pytest.raises(ValueError):
        ev._prepare_periodic_factorized_graph(types + 7, pos, cell, np.linalg.inv(cell), 5.5)     # type out of range
    bad = pos.copy()
    bad[1] = bad[0]                                                     # zero-length edge
    res3 = ev._prepare_periodic_factorized_graph(types, pos, cell, np.linalg.inv(cell), 5.5)
    with pytest.raises(ValueError):
        ev._compute_prepared_factorized_positions(res3["generation"], bad)


@pytest.mark.parametrize("scaled,zbl,agnesi", [(False, False, False), (True, False, False), (False, True, False), (True, False, True)])
def test_forces_are_energy_gradient(pkg, model_path, scaled, zbl, agnesi):
    """Finite-difference check (reference: symmetrix/test/test_mace.py:74-85)."""
    path = model_path("small", a0_scaled=scaled, a1_scaled=scaled, zbl=zbl, agnesi=agnesi)
    pos, cell, types = pkg.modelgen.srtio3(2, 0.05, 4)
    calc = pkg.Calculator(path, skin=0.5)
    base = calc.calculate(pos, cell, types)
    h = 2e-3
    for atom, axis in ((0, 0), (7, 1), (13, 2)):
        p, m = pos.copy(), pos.copy()
        p[atom, axis] += h
        m[atom, axis] -= h
        ep = calc.calculate(p, cell, types)["energy"]
        em = calc.calculate(m, cell, types)["energy"]
        fd = -(ep - em) / (2 * h)
        assert abs(fd - base["forces"][atom, axis]) <= 5e-3 * max(1.0, abs(fd))


def test_graphless_force_and_stress_reduction(pkg, model_path):
    """Directed forces reduced from explicit edge lists (reference: _reduce_atom_forces /
    _reduce_stress with execution_graph_generation = 0) agree with the fused reduction."""
    path = model_path("small")
    pos, cell, types = pkg.modelgen.srtio3(3, 0.05, 6)
    first, src, shifts, xyz = csr_from_positions(pos, cell, 5.0)
    ev = pkg.MACEB200(path)
    gen = ev.compute_node_energies_forces(len(pos), types, np.diff(first), src, types[src], xyz)
    volume = abs(np.linalg.det(cell))
    fused_f = ev._reduce_atom_forces(len(pos), execution_graph_generation=gen)
    fused_s = ev._reduce_stress(volume, execution_graph_generation=gen)
    recv = np.repeat(np.arange(len(pos)), np.diff(first))
    f, s = pkg.reduce_edge_forces(len(pos), recv, src, ev.node_forces, xyz, volume)
    want_f, want_s = ref.reduce_forces_stress(len(pos), np.diff(first), src, ev.node_forces, xyz, volume)
    assert np.abs(f - want_f).max() < 1e-12 and np.abs(s - want_s).max() < 1e-14
    assert np.abs(f - fused_f).max() < 1e-6 and np.abs(s - fused_s).max() < 1e-8
    with pytest.raises(ValueError):
        pkg.reduce_edge_forces(len(pos), recv, src + 1000, ev.node_forces, xyz, volume)


@pytest.mark.parametrize("arch,cells,tile,scaled", [("small", (2, 2, 2), 4, False), ("small", (3, 2, 2), 7, False),
                                                    ("medium", (2, 2, 2), 16, False), ("medium", (3, 2, 2), 32, False),
                                                    ("medium", (2, 2, 2), 16, True), ("large", (2, 2, 2), 16, False)])
def test_tiled_streaming_matches_untiled(pkg, model_path, arch, cells, tile, scaled):
    """Tiled streaming with a reusable workspace against the one-tile evaluation
    (reference: symmetrix/test/test_dual_layer_fixed_workspace.py:104-146, rtol 2e-4 / atol 2e-5)."""
    path = model_path(arch, a0_scaled=scaled, a1_scaled=scaled)
    pos, cell, types = pkg.modelgen.srtio3(cells, 0.05, 12)
    plain = pkg.Calculator(path, skin=0.5)
    a = plain.calculate(pos, cell, types)
    h1_adj = plain.evaluator.stage("H1_adj")
    tiled = pkg.Calculator(path, skin=0.5)
    tiled.evaluator.set_tile_size(tile)
    b = tiled.calculate(pos, cell, types)
    b = tiled.calculate(pos, cell, types)         # the workspace is reused across evaluations
    assert abs(a["energy"] - b["energy"]) / len(pos) <= 1e-7
    assert np.abs(a["energies"] - b["energies"]).max() <= 1e-6
    assert np.abs(a["forces"] - b["forces"]).max() <= 1e-5
    assert np.abs(a["stress"] - b["stress"]).max() <= 1e-8
    got = tiled.evaluator.stage("H1_adj")
    assert np.abs(got - h1_adj).max() <= 2e-5 * max(1.0, np.abs(h1_adj).max())
    with pytest.raises(ValueError):
        tiled.evaluator.stage("Phi1")
    if ref.available():      # and directly against the reference's evaluator
        e, F, S = _reference_efs(path, pos, cell, types, tiled.evaluator.r_cut)
        _assert_matches_reference(b, e, F, S, len(pos))


def test_tile_boundary_sizes(pkg, model_path):
    """3, 4, 5, 8 and 9 atoms with a tile capacity of 4 (the reference's tile-boundary cases)."""
    path = model_path("small")
    rng = np.random.default_rng(5)
    for natoms in (3, 4, 5, 8, 9):
        cell = np.eye(3) * 9.0
        pos = rng.random((natoms, 3)) * 9.0
        for i in range(1, natoms):
            while np.min(np.linalg.norm(pos[:i] - pos[i], axis=1)) < 1.6:
                pos[i] = rng.random(3) * 9.0
        types = rng.integers(0, 3, size=natoms).astype(np.int32)
        a = pkg.Calculator(path, skin=0.5).calculate(pos, cell, types)
        calc = pkg.Calculator(path, skin=0.5)
        calc.evaluator.set_tile_size(4)
        b = calc.calculate(pos, cell, types)
        assert abs(a["energy"] - b["energy"]) <= 1e-6
        assert np.abs(a["forces"] - b["forces"]).max() <= 1e-5


@pytest.mark.parametrize("arch,zbl", [("medium", False), ("small", True)])
def test_reproducible_mode_gives_identical_bits(pkg, model_path, arch, zbl):
    """Fixed-order accumulation over the source schedule (the reference's source-sorted schedule,
    libsymmetrix/source/mace_kokkos_factorized_lifecycle.cpp:2133-2195): repeated evaluations, and a second
    evaluator, give bit-identical energies, forces, stress and source adjoints; the values agree with the
    default (atomic) mode and with the reference's evaluator within the tolerances."""
    path = model_path(arch, seed=12, zbl=zbl)
    pos, cell, types = pkg.modelgen.srtio3(3, 0.05, 31)
    runs = []
    for instance in range(2):
        calc = pkg.Calculator(path, skin=0.5)
        calc.evaluator.set_deterministic(True)
        for repeat in range(2):
            out = calc.calculate(pos, cell, types)
            runs.append((out["energy"], out["energies"].copy(), out["forces"].copy(), out["stress"].copy(),
                         calc.evaluator.stage("H1_adj")))
    for other in runs[1:]:
        assert other[0] == runs[0][0]
        for a, b in zip(other[1:], runs[0][1:]):
            assert np.array_equal(a, b)
    plain = pkg.Calculator(path, skin=0.5).calculate(pos, cell, types)
    assert abs(plain["energy"] - runs[0][0]) / len(pos) <= 1e-7
    assert np.abs(plain["forces"] - runs[0][2]).max() <= 1e-5
    assert np.abs(plain["stress"] - runs[0][3]).max() <= 1e-8
    if ref.available():
        e, F, S = _reference_efs(path, pos, cell, types, calc.evaluator.r_cut)
        _assert_matches_reference({"energy": runs[0][0], "energies": runs[0][1], "forces": runs[0][2], "stress": runs[0][3]}, e, F, S,
                                  len(pos))
    scaled = pkg.Calculator(model_path("small", a0_scaled=True, a1_scaled=True), skin=0.5)
    scaled.evaluator.set_deterministic(True)
    with pytest.raises(ValueError):
        scaled.calculate(pos, cell, types)


@pytest.mark.parametrize("arch,channels", [("medium", 128), ("medium", 64), ("small", 32)])
def test_reproducible_bits_do_not_depend_on_tiles_or_skin(pkg, model_path, arch, channels):
    """Energies and forces of the reproducible mode are sums over the edges inside the cutoff, in list order: the number of
    skin edges between them and the size of the tiles change no bit (one bin along each axis, so that every list has its edges
    in the same order).  Tiled evaluations add the direct adjoint of M0 last and the untiled one first: their forces are
    compared among themselves.  40 atoms are dealt out to parts."""
    path = model_path(arch, seed=12, channels=channels)
    pos, cell, types = pkg.modelgen.srtio3(2, 0.05, 31)
    pos = pos + 0.25 * cell.sum(axis=0) / 2
    edges, results = set(), {}
    for tile, skin in ((0, 0.5), (0, 0.0), (0, 0.9), (7, 0.5), (16, 0.2), (20, 0.5), (1, 0.0)):
        ev = pkg.MACEB200(path)
        ev.set_deterministic(True)
        ev.set_tile_size(tile)
        res = ev._prepare_periodic_factorized_graph(types, pos, cell, np.linalg.inv(cell), ev.r_cut + skin)
        ev._compute_prepared_factorized_positions(res["generation"], pos)
        edges.add(res["num_edges"])
        forces = ev._reduce_atom_forces(len(pos), execution_graph_generation=res["generation"]).copy()
        results.setdefault(tile > 0, []).append((ev.node_energies.copy(), ev.energy, ev.stage("H1_adj").copy(), forces))
    assert len(edges) > 2
    first = results[False][0]
    for run in results[False] + results[True]:
        assert np.array_equal(run[0], first[0]) and run[1] == first[1] and np.array_equal(run[2], first[2])
    for runs in results.values():
        for run in runs:
            assert np.array_equal(run[3], runs[0][3])


def test_nve_energy_conservation(pkg, model_path):
    """20 velocity-Verlet steps of 1 fs at 300 K: total energy is conserved to integrator accuracy."""
    path = model_path("small")
    pos, cell, types = pkg.modelgen.srtio3(3, 0.05, 3)
    z = np.array([8, 22, 38])[types]
    masses = np.array([pkg.md.MASSES[int(v)] for v in z])
    vel = pkg.md.maxwell_boltzmann(masses, 300.0, 3)
    ev = pkg.MACEB200(path)
    md = pkg.md.NVEIntegrator(ev, pos, cell, types, masses, vel, dt_fs=1.0, skin=0.5)
    e = md.run(20)
    drift = np.abs(e - e[0]).max() / len(pos)
    assert drift < 2e-4, drift          # eV/atom over 20 fs
    assert md.kinetic() > 0


@pytest.mark.parametrize("channels,scale", [(128, 1.0), (128, 0.9), (64, 0.9)])
def test_records_of_the_paired_gradient_match_its_atomic_sums(pkg, model_path, channels, scale):
    """The reproducible mode's records against the default build of the same kernel: one chunk of edges per receiver, and a
    compressed cell with more than a chunk holds (96); in few parts and in many (40 and 320 receivers).  The two differ in the
    order of FP32 sums of about 100 edges: bounds of 2^-24 times the terms of a sum times the largest row, with room for the
    linears behind it.  Bits do not depend on the list's skin."""
    for copies in (2, 4):
        pos, cell, types = pkg.modelgen.srtio3(copies, 0.05, 8)
        pos, cell = pos * scale, cell * scale
        runs = []
        for fixed, skin in ((False, 0.5), (True, 0.5), (True, 0.2)):
            calc = pkg.Calculator(model_path("medium", seed=5, channels=channels), skin=skin)
            calc.evaluator.set_deterministic(fixed)
            runs.append(calc.calculate(pos, cell, types))
        bound = 100 * 2.0 ** -24 * max(1.0, np.abs(runs[0]["forces"]).max())
        assert np.abs(runs[1]["forces"] - runs[0]["forces"]).max() <= bound
        assert np.abs(runs[1]["stress"] - runs[0]["stress"]).max() <= 0.1 * bound
        assert np.array_equal(runs[1]["forces"], runs[2]["forces"]) and runs[1]["energy"] == runs[2]["energy"]


@pytest.mark.parametrize("n", [1, 128, 129, 592 * 128 + 1])
def test_advance_kernel_is_the_tensor_expression(pkg, model_path, n):
    """Kick and drift bit for bit as the tensor expressions (one rounding per operation), a block's edge and more atoms than
    the grid has threads; the largest squared displacement, also with a NaN among the atoms (it wins, as in max())."""
    import torch

    ev = pkg.MACEB200(model_path("small"))
    gen = torch.Generator("cuda").manual_seed(n)
    x, v, f, x_ref = (torch.randn((n, 3), dtype=torch.float64, device="cuda", generator=gen) for _ in range(4))
    m = 1.0 + torch.rand((n, 1), dtype=torch.float64, device="cuda", generator=gen)
    for bad in (False, True):
        if bad:
            f[n // 2, 1] = float("nan")
        want_v = v + 0.37 * f / m
        want_x = x + 0.9 * want_v
        want = ((want_x - x_ref) ** 2).sum(dim=1).max().item()
        got = ev.md_advance(torch.cuda.current_stream().cuda_stream, n, 0.9, 0.37, x.data_ptr(), v.data_ptr(), f.data_ptr(),
                            m.data_ptr(), x_ref.data_ptr())
        assert torch.equal(v.nan_to_num(7.0), want_v.nan_to_num(7.0)) and torch.equal(x.nan_to_num(7.0), want_x.nan_to_num(7.0))
        assert np.isnan(got) if bad else abs(got - want) <= 4 * 2.0 ** -53 * want          # three squares, two sums


def test_first_step_of_an_evaluator_on_a_side_stream(pkg, model_path):
    """The workspace of the step is cleared in the order of the caller's stream, which does not wait for the default one."""
    import torch

    n = 129
    gen = torch.Generator("cuda").manual_seed(n)
    x_ref, v, f = (torch.randn((n, 3), dtype=torch.float64, device="cuda", generator=gen) for _ in range(3))
    m = torch.ones((n, 1), dtype=torch.float64, device="cuda")
    x = x_ref + 0.01 * v
    moved = ((x + 0.9 * (v + 0.37 * f) - x_ref) ** 2).sum(dim=1).max().item()
    for _ in range(4):
        ev = pkg.MACEB200(model_path("small"))
        stream = torch.cuda.Stream()
        state = [t.clone() for t in (x, v)]
        stream.wait_stream(torch.cuda.current_stream())
        got = ev.md_advance(stream.cuda_stream, n, 0.9, 0.37, state[0].data_ptr(), state[1].data_ptr(), f.data_ptr(), m.data_ptr(),
                            x_ref.data_ptr())
        assert abs(got - moved) <= 16 * 2.0 ** -53 * moved


@pytest.mark.parametrize("drop", [0, 6, 7, 8])
def test_step_kernels_match_the_tensor_step(pkg, model_path, drop):
    """The same trajectory from the two kernels and from tensor expressions, in the reproducible mode (equal forces for equal
    positions): bit for bit, and the energies to the order of a sum of 3n squares.  127 to 135 atoms; lists are rebuilt."""
    class Tensors(pkg.md.NVEIntegrator):
        def kinetic(self):                      # a subclass with its own energy keeps the tensor step
            return super().kinetic()

    path = model_path("small")
    pos, cell, types = pkg.modelgen.srtio3(3, 0.05, 3)
    pos, types = pos[drop:], types[drop:]
    masses = np.array([pkg.md.MASSES[z] for z in (8, 22, 38)])[types]
    vel = pkg.md.maxwell_boltzmann(masses, 300.0, 3)
    runs = []
    for cls in (pkg.md.NVEIntegrator, Tensors):
        ev = pkg.MACEB200(path)
        ev.set_deterministic(True)
        md = cls(ev, pos, cell, types, masses, vel, dt_fs=1.0, skin=0.02)
        assert md._plain() == (cls is pkg.md.NVEIntegrator)
        runs.append((md.run(8), md.x.cpu().numpy(), md.v.cpu().numpy(), md.f.cpu().numpy(), md.rebuilds, md.kinetic()))
    for a, b in zip(runs[0][1:5], runs[1][1:5]):
        assert np.array_equal(a, b)
    assert runs[0][4] > 1
    bound = 3 * len(pos) * 2.0 ** -53
    assert abs(runs[0][5] - runs[1][5]) <= bound * runs[1][5]
    assert np.abs(runs[0][0] - runs[1][0]).max() <= bound * runs[1][5] + 2.0 ** -52 * np.abs(runs[1][0]).max()


@pytest.mark.parametrize("way", ["evaluator subclass", "evaluator object", "evaluator instance", "evaluator class", "integrator subclass",
                                 "integrator instance", "integrator class", "time step"])
def test_forces_of_ones_own_steer_the_step(pkg, model_path, monkeypatch, way):
    """Forces that an evaluator or an integrator puts in the place of the computed ones (here: none, the atoms fly straight) are
    those of the step, as is a time step for each atom."""
    import torch

    pos, cell, types = pkg.modelgen.srtio3(1, 0.05, 3)
    masses = np.array([pkg.md.MASSES[z] for z in (8, 22, 38)])[types]
    vel = pkg.md.maxwell_boltzmann(masses, 300.0, 3)
    zeros = torch.zeros((len(pos), 3), dtype=torch.float64, device="cuda")
    results = pkg.MACEB200.device_results

    def device_results(self):
        energy, _forces, virial = results(getattr(self, "inner", self))
        return energy, zeros.data_ptr(), virial

    class Wrapper:
        def __init__(self, inner):
            self.inner = inner

        def __getattr__(self, name):
            if name.startswith("md_"):
                raise AttributeError(name)
            return getattr(self.inner, name)

    Wrapper.device_results = device_results
    ev = pkg.MACEB200(model_path("small"))
    kind, place = way.split()
    if way == "evaluator object":
        ev = Wrapper(ev)
    elif way == "evaluator subclass":
        ev.__class__ = type("Own", (pkg.MACEB200,), {"device_results": device_results})
    elif way == "evaluator instance":
        ev.device_results = device_results.__get__(ev)
    elif way == "evaluator class":
        monkeypatch.setattr(pkg.MACEB200, "device_results", device_results)
    md = pkg.md.NVEIntegrator(ev, pos, cell, types, masses, vel, dt_fs=1.0)
    if kind == "integrator":
        def forces(self):
            self._evaluate(0.0)
            return zeros.clone(), self.ev.energy

        md.f = zeros.clone()
        if place == "instance":
            md._forces = forces.__get__(md)
        elif place == "class":
            monkeypatch.setattr(pkg.md.NVEIntegrator, "_forces", forces)
        else:
            md.__class__ = type("Own", (pkg.md.NVEIntegrator,), {"_forces": forces})
    if way == "time step":
        md.dt = torch.full((len(pos), 1), 0.5, dtype=torch.float64, device="cuda")
        md.f = zeros.clone()
    before, v = md.x.clone(), md.v.clone()
    energy = md.step()
    assert torch.equal(md.x, before + (0.5 if way == "time step" else 1.0) * v)
    if way != "time step":
        assert torch.equal(md.v, v) and torch.equal(md.f, zeros)
    assert np.isfinite(energy)


@pytest.mark.gpu
@pytest.mark.parametrize("arch,copies", [("medium", (2, 1, 1)), ("medium", (4, 2, 2)), ("small", (4, 2, 1)), ("large", (2, 2, 1))])
def test_parts_of_a_receiver_add_up(pkg, model_path, arch, copies):
    """A receiver's edges are dealt to more blocks and warps, and the linears' column tiles get narrower, the fewer receivers
    there are: a cell of 38 atoms (most parts) against the oracle, and its periodic copies (fewer parts; undivided receivers
    are in test_every_division_of_receivers) against the cell.  Bounds: those of the oracle comparison; the copies differ from
    the cell by the order of float sums alone."""
    from oracle import mace_numpy, neighbor

    path = model_path(arch, 31)
    pos, cell, types = pkg.modelgen.srtio3(2, 0.05, 12)
    pos, types = pos[2:], types[2:]
    calc = pkg.Calculator(path, skin=0.5)
    out = calc.calculate(pos, cell, types)
    first, src, shifts = neighbor.build_neighbor_graph(pos, cell, calc.evaluator.r_cut + 0.5)
    _e, energies, forces, _s = mace_numpy.NumpyMACE(str(path)).energy_forces_stress(types, pos, cell, first, src, shifts)
    assert np.abs(out["energies"] - energies).max() <= TOL_E
    assert np.abs(out["forces"] - forces).max() <= TOL_F
    grid = np.stack(np.meshgrid(*[np.arange(c) for c in copies], indexing="ij"), axis=-1).reshape(-1, 3)
    many = (pos[None] + (grid @ cell)[:, None]).reshape(-1, 3)
    big = pkg.Calculator(path, skin=0.5).calculate(many, cell * np.array(copies)[:, None], np.tile(types, len(grid)))
    assert np.abs(big["energies"].reshape(len(grid), -1) - out["energies"]).max() <= TOL_E
    assert np.abs(big["forces"].reshape(len(grid), -1, 3) - out["forces"]).max() <= TOL_F


@pytest.mark.gpu
@pytest.mark.parametrize("arch,counts", [("medium", (1, 1, 1)), ("medium", (3, 17, 15)), ("small", (33, 1, 2)), ("large", (31, 2, 34))])
def test_contraction_runs_of_elements(pkg, model_path, arch, counts):
    """The contraction kernels walk runs of equal elements, two nodes per warp: runs of one, odd runs, runs that end inside a
    block and runs that fill it exactly, for stage tensors against the oracle (bounds of the stage comparison)."""
    from oracle import mace_numpy, neighbor

    path = model_path(arch, 33)
    rng = np.random.default_rng(5)
    n = sum(counts)
    side = int(np.ceil(n ** (1 / 3)))
    grid = np.stack(np.meshgrid(*[np.arange(side)] * 3, indexing="ij"), axis=-1).reshape(-1, 3)[:n]
    pos = 2.4 * grid + rng.uniform(-0.2, 0.2, (n, 3))
    cell = np.eye(3) * max(2.4 * side, 4.8)
    types = np.repeat(np.arange(3), counts).astype(np.int32)
    ev = pkg.MACEB200(path)
    res = ev._prepare_periodic_factorized_graph(types, pos, cell, np.linalg.inv(cell), ev.r_cut)
    ev._compute_prepared_factorized_positions(res["generation"], pos)
    first, src, shifts = neighbor.build_neighbor_graph(pos, cell, ev.r_cut)
    oracle = mace_numpy.NumpyMACE(str(path))
    _e, energies, forces, _s = oracle.energy_forces_stress(types, pos, cell, first, src, shifts)
    assert np.abs(ev.node_energies - energies).max() <= TOL_E
    got = ev._reduce_atom_forces(n, execution_graph_generation=res["generation"])
    assert np.abs(got - forces).max() <= TOL_F * max(1.0, np.abs(forces).max())
    for name in ("M0", "M1", "A1_adj", "A0_adj"):      # what the four contraction kernels leave
        want = oracle.stage[name]
        assert np.abs(ev.stage(name).reshape(want.shape) - want).max() <= 2e-5 * max(1.0, np.abs(want).max()), name


@pytest.mark.gpu
@pytest.mark.parametrize("channels,options", [(128, {}), (64, {}), (64, {"a0_scaled": True, "a1_scaled": True}), (128, {"agnesi": True})])
def test_layer1_gradient_widths_and_odd_edge_counts(pkg, model_path, channels, options):
    """The layer-1 gradient takes two edges at a time: receivers without, with one and with an odd number of active edges, and a
    dense cell whose 120 list edges a receiver are dealt to eight parts, at both compiled widths, against the oracle.  (Chunks
    filled more than once: test_every_division_of_receivers.)"""
    from oracle import mace_numpy, neighbor

    path = model_path("medium", 35, channels=channels, **options)
    rng = np.random.default_rng(9)
    blob = rng.uniform(0.0, 1.0, (26, 3)) * np.array([9.0, 9.0, 4.0])
    keep = [0]
    for i in range(1, len(blob)):
        if all(np.linalg.norm(blob[i] - blob[j]) > 1.6 for j in keep):
            keep.append(i)
    pos = np.concatenate([blob[keep], [[30.0, 30.0, 30.0], [45.0, 30.0, 30.0], [45.0, 33.0, 30.0]]])
    cell = np.eye(3) * 60.0
    types = (np.arange(len(pos)) % 3).astype(np.int32)
    dense_pos, dense_cell, dense_types = pkg.modelgen.srtio3(2, 0.05, 3)
    calc = pkg.Calculator(path, skin=0.5)
    for p, c, t in ((pos, cell, types), (dense_pos, dense_cell * 0.93, dense_types)):
        out = calc.calculate(p, c, t)
        first, src, shifts = neighbor.build_neighbor_graph(p, c, calc.evaluator.r_cut + 0.5)
        _e, energies, forces, _s = mace_numpy.NumpyMACE(str(path)).energy_forces_stress(t, p, c, first, src, shifts)
        assert np.abs(out["energies"] - energies).max() <= TOL_E
        assert np.abs(out["forces"] - forces).max() <= TOL_F * max(1.0, np.abs(forces).max())


@pytest.mark.gpu
@pytest.mark.parametrize("arch,channels,options,copies,layer0,parts", [
    # layer 0 on the folded table: parts of a receiver in the layer-0 sums, the layer-1 sums, the layer-1 and the layer-0 gradient; on
    # the radial functions, whose sums are never divided: layer-1 sums, layer-1 and layer-0 gradient
    ("medium", 128, {}, (1, 1, 1), "table", (4, 8, 4, 8)),
    ("medium", 128, {}, (2, 2, 2), "table", (4, 1, 2, 4)),
    ("medium", 128, {}, (3, 3, 3), "functions", (1, 1, 3)),
    ("medium", 128, {"a0_scaled": True, "a1_scaled": True}, (3, 3, 4), "functions", (1, 1, 3)),
    ("medium", 128, {"a0_scaled": True, "a1_scaled": True}, (3, 3, 6), "functions", (1, 1, 1)),
    ("medium", 128, {"radial_hidden": (64, 64, 32)}, (3, 3, 3), "table", (4, 1, 1, 4)),
    ("medium", 128, {"radial_hidden": (64, 64, 32), "a0_scaled": True}, (7, 4, 4), "table", (1, 1, 1, 1)),
    ("medium", 64, {}, (1, 1, 1), "table", (4, 8, 4, 8)),
    ("medium", 64, {}, (3, 3, 3), "functions", (1, 1, 3)),
    ("medium", 64, {"a0_scaled": True, "a1_scaled": True}, (3, 3, 9), "functions", (1, 1, 1)),
    ("medium", 64, {"radial_hidden": (64, 64, 32)}, (3, 3, 3), "table", (4, 1, 1, 2)),
    ("medium", 64, {"radial_hidden": (64, 64, 32), "a0_scaled": True}, (7, 4, 4), "table", (1, 1, 1, 1)),
    ("large", 128, {}, (1, 1, 1), "table", (4, 8, 2, 8)),
    ("large", 128, {}, (3, 3, 2), "functions", (1, 1, 3)),
    ("small", 32, {}, (1, 1, 1), "table", (4, 8, 8, 8)),
    ("small", 32, {}, (4, 3, 3), "table", (4, 1, 2, 2)),
    ("small", 32, {}, (6, 5, 4), "table", (1, 1, 1, 1)),
])
def test_every_division_of_receivers(pkg, model_path, part_rule, arch, channels, options, copies, layer0, parts):
    """Each build that the part rules can choose, from the most parts to undivided receivers whose 97 list edges (small: 58)
    fill the 64-edge chunks of the layer-1 kernels and the 32-edge ones of layer 0 more than once: periodic copies of a 40-atom
    cell, atom by atom against the oracle of the cell (bounds of the oracle comparison).  The parts are asserted by the rules that the
    launches call, so that a changed rule cannot leave a build out unnoticed."""
    import torch

    path = model_path(arch, 37, channels=channels, **options)
    pos, cell, types = pkg.modelgen.srtio3(2, 0.05, 14)
    calc = pkg.Calculator(path, skin=0.5)
    first, src, shifts = neighbor.build_neighbor_graph(pos, cell, calc.evaluator.r_cut + 0.5)
    _e, energies, forces, _s = mace_numpy.NumpyMACE(str(path)).energy_forces_stress(types, pos, cell, first, src, shifts)
    grid = np.stack(np.meshgrid(*[np.arange(c) for c in copies], indexing="ij"), axis=-1).reshape(-1, 3)
    many = (pos[None] + (grid @ cell)[:, None]).reshape(-1, 3)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    shape = {"small": 0, "medium": 1, "large": 2}[arch]
    rule = lambda kernel: part_rule(kernel, sms, channels, shape, len(src) / len(pos), len(many))
    functions = channels in (64, 128) and "radial_hidden" not in options and rule("layer0_on_basis")
    kernels = ("l1_forward", "l1_reverse", "l0_moments_reverse") if functions else ("l0_forward", "l1_forward", "l1_reverse", "l0_reverse")
    assert (layer0, parts) == ("functions" if functions else "table", tuple(rule(kernel) for kernel in kernels))
    calc.evaluator.set_profiling(True)
    out = calc.calculate(many, cell * np.array(copies)[:, None], np.tile(types, len(grid)))
    assert ("gemm_a0" in {name for name, _ms, _launches in calc.evaluator.profile()}) == bool(functions)
    assert np.abs(out["energies"].reshape(len(grid), -1) - energies).max() <= TOL_E
    assert np.abs(out["forces"].reshape(len(grid), -1, 3) - forces).max() <= TOL_F


@pytest.mark.gpu
def test_a_graph_that_failed_to_install_ends_the_handle_before(pkg, model_path):
    """Installation that throws after extents and tables have been replaced (the reproducible mode's records would take more than
    16 GB): the handle before is refused, results are gone, and the calculator builds its list again, with the same bits.  Types
    that are refused at once leave the handle as it was."""
    calc = pkg.Calculator(model_path("medium"), skin=0.5)
    calc.evaluator.set_deterministic(True)
    ev = calc.evaluator
    pos, cell, types = pkg.modelgen.srtio3(2, 0.05, 6)
    first = calc.calculate(pos, cell, types)
    generation = calc._generation
    bad = types.copy()
    bad[3] = 3
    with pytest.raises(ValueError):
        ev._prepare_periodic_factorized_graph(bad, pos, cell, np.linalg.inv(cell), 6.5)
    ev._compute_prepared_factorized_positions(generation, pos)
    assert np.array_equal(ev.node_energies, first["energies"])
    many, big, of = pkg.modelgen.srtio3((27, 26, 26), 0.05, 6)             # 91,260 atoms, 8.8 million edges
    for _ in range(2):
        with pytest.raises(ValueError, match="16 GB"):
            calc.calculate(many, big, np.where(of == 2, 1, of).astype(np.int32))
        with pytest.raises(ValueError, match="stale"):
            ev._compute_prepared_factorized_positions(generation, pos)
        with pytest.raises((RuntimeError, ValueError)):         # no results, or a buffer of the old extent
            ev.node_energies
    again = calc.calculate(pos, cell, types)
    assert again["energy"] == first["energy"] and np.array_equal(again["forces"], first["forces"])


def test_types_refused_half_way_are_refused_again(pkg, model_path, tmp_path):
    """The repulsion's radii are missing for one element: a preparation with it throws after other tables have been made.  The
    same types throw again instead of passing for prepared, and the elements that are covered evaluate as in a whole file."""
    whole = model_path("small", 3, zbl=True)
    model = json.loads(Path(whole).read_text())
    model["zbl_covalent_radii"] = model["zbl_covalent_radii"][:30]          # up to Zn: not Sr
    cut = tmp_path / "cut.json"
    cut.write_text(json.dumps(model))
    pos, cell, types = pkg.modelgen.srtio3(2, 0.05, 4)
    few = np.where(types == 2, 1, types).astype(np.int32)
    calc = pkg.Calculator(cut, skin=0.5)
    for _ in range(2):
        with pytest.raises(ValueError, match="radii"):
            calc.calculate(pos, cell, types)
    out = calc.calculate(pos, cell, few)
    with pytest.raises(ValueError, match="radii"):
        calc.calculate(pos, cell, types)
    again, want = calc.calculate(pos, cell, few), pkg.Calculator(whole, skin=0.5).calculate(pos, cell, few)
    for got in (out, again):          # the order of atomic sums differs
        assert np.abs(got["energies"] - want["energies"]).max() <= 2e-6
        assert np.abs(got["forces"] - want["forces"]).max() <= 2e-5 * max(1.0, np.abs(want["forces"]).max())
