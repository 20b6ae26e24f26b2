"""Layer 0 on the functions of the radial network's last hidden layer, and the kernels that only larger graphs reach."""
import ctypes
import subprocess
import sysconfig
from pathlib import Path

import numpy as np
import pytest

ROOT = Path(__file__).resolve().parent.parent

HARNESS = r"""
#include <algorithm>
#include <cmath>
#include "%s"
// Largest difference between the folded table and the functions times the folded map, over all ordered pairs of active types, all
// intervals at four places and all channels, relative to the largest value of the pair; -1 when the model has no such functions.
extern "C" double difference(const char* path, const int* types, int n, int* width)
{
    using namespace sxb;
    const HostModel m = load_model(path);
    const std::vector<int> active(types, types + n);
    const int H = *width = radial_basis_width(m, "R0"), C = m.channels, L = m.l_max + 1, F = L * C;
    if (H == 0) return -1.0;
    int pair_types[2];
    const auto lanes = build_r0_basis(m, active, &pair_types[0], false), steps = build_r0_basis(m, active, &pair_types[1], true);
    const auto table = fold_r0_table(m, active);
    const int intervals = m.spline_points - 1, pt = pair_types[0];
    if (pair_types[1] != pt || lanes.size() != steps.size()) return 1e30;
    double worst = 0.0;
    for (int ai = 0; ai < n; ++ai)
        for (int l = 0; l < L; ++l) {
            const auto G = fold_r0_mixing(m, active, ai, l);
            for (int aj = 0; aj < n; ++aj) {
                const int a = std::min(ai, aj), b = std::max(ai, aj), pair = pt > 1 ? a * (2 * pt - a - 1) / 2 + b : 0;
                double largest = 0.0, difference = 0.0;
                for (int i = 0; i < intervals; ++i)
                    for (int place = 0; place < 4; ++place) {
                        const double x = m.spline_h * place / 4.0;
                        std::vector<double> phi(H);
                        for (int h = 0; h < H; ++h) {
                            const float* row = lanes.data() + (static_cast<std::size_t>(pair) * intervals + i) * 4 * H;
                            const float* step = steps.data() + ((static_cast<std::size_t>(pair) * intervals + i) * (H / 4) + h %% (H / 4)) * 16 + 4 * (h / (H / 4));
                            double c[4];
                            for (int q = 0; q < 4; ++q) {
                                c[q] = row[(q / 2) * 2 * H + (h / 2) * 4 + (q %% 2) * 2 + h %% 2];
                                if (static_cast<float>(c[q]) != step[q]) return 1e30;
                            }
                            phi[h] = c[0] + x * (c[1] + x * (c[2] + x * c[3]));
                        }
                        for (int k = 0; k < C; ++k) {
                            const float* t = table.data() + (static_cast<std::size_t>(ai * n + aj) * intervals + i) * 4 * F + l * C + k;
                            const double want = t[0] + x * (t[F] + x * (t[2 * F] + x * static_cast<double>(t[3 * F])));
                            double got = 0.0;
                            for (int h = 0; h < H; ++h) got += phi[h] * G[(static_cast<std::size_t>(aj) * H + h) * C + k];
                            largest = std::max(largest, std::abs(want));
                            difference = std::max(difference, std::abs(got - want));
                        }
                    }
                worst = std::max(worst, difference / largest);
            }
        }
    return worst;
}
"""


@pytest.fixture(scope="module")
def difference(tmp_path_factory):
    folder = tmp_path_factory.mktemp("layer0")
    csrc = ROOT / "symmetrix-xl_b200" / "csrc"
    (folder / "harness.cpp").write_text(HARNESS % (csrc / "model.cpp"))
    include = Path(sysconfig.get_paths()["purelib"]) / "include" / "cudnn_frontend" / "thirdparty"
    subprocess.run(["g++", "-std=c++17", "-O2", "-shared", "-fPIC", "-I", str(csrc), "-I", str(include), "-o", str(folder / "harness.so"),
                    str(folder / "harness.cpp")], check=True)
    lib = ctypes.CDLL(str(folder / "harness.so"))
    lib.difference.restype = ctypes.c_double

    def call(path, types):
        width = ctypes.c_int(0)
        value = lib.difference(str(path).encode(), (ctypes.c_int * len(types))(*types), len(types), ctypes.byref(width))
        return value, width.value

    return call


@pytest.mark.parametrize("kwargs,types,width", [(dict(channels=64), (0, 1, 2), 64), (dict(channels=64), (2,), 64),
                                                (dict(channels=64, agnesi=True, a0_scaled=True), (0, 2), 64),
                                                (dict(channels=64, radial_hidden=(32, 64)), (1, 2), 64),
                                                (dict(channels=32, radial_hidden=(64, 32)), (0, 1), 32),
                                                (dict(channels=32, radial="pair-splines"), (0, 1), 0)])
def test_functions_and_map_give_the_folded_table(difference, model_path, kwargs, types, width):
    """Both are made in double and rounded once: coefficients and map to 6e-8 each, 64 products of either sign."""
    value, found = difference(model_path("medium" if "radial" not in kwargs else "small", **kwargs), types)
    assert found == width
    assert value == -1.0 if width == 0 else value <= 1e-6


def test_choice_of_layer0(tmp_path):
    """The functions need enough receivers per type; ten types at most."""
    header = ROOT / "symmetrix-xl_b200" / "csrc" / "part_rules.hpp"
    (tmp_path / "rule.cpp").write_text(f'#include "{header}"\nextern "C" int rule(int channels, long receivers, int types)\n'
                                       "{ return sxb::PartRules{148, channels, 1, 97.0}.layer0_on_basis(receivers, types); }\n"
                                       'extern "C" int parts(long receivers, int types)\n'
                                       "{ return sxb::PartRules{148, 128, 1, 97.0}.l0_moments_reverse(receivers, types); }\n"
                                       'extern "C" int pairs(long receivers, int resident)\n'
                                       "{ return sxb::PartRules{148, 128, 1, 97.0}.l1_reverse_pairs(receivers, resident); }\n")
    subprocess.run(["g++", "-std=c++17", "-shared", "-fPIC", "-o", str(tmp_path / "rule.so"), str(tmp_path / "rule.cpp")], check=True)
    lib = ctypes.CDLL(str(tmp_path / "rule.so"))
    assert [lib.rule(128, ctypes.c_long(n), 3) for n in (40, 449, 450, 10 ** 7)] == [0, 0, 1, 1]
    assert [lib.rule(64, ctypes.c_long(n), 3) for n in (689, 690)] == [0, 1]
    assert [lib.rule(128, ctypes.c_long(10 ** 6), t) for t in (1, 10, 11, 200)] == [1, 1, 0, 0]
    for types in (1, 2, 3, 10):
        for receivers in (1, 150, 450, 1775, 1776, 10 ** 7):
            parts = lib.parts(ctypes.c_long(receivers), types)
            assert parts == 1 if receivers >= 1776 else parts % types == 0 and 1 <= parts // types <= 4
    assert [lib.pairs(ctypes.c_long(n), 2) for n in (40, 160, 320, 600, 5000)] == [4, 4, 2, 1, 1]
    assert [lib.pairs(ctypes.c_long(n), 1) for n in (1, 160, 2 ** 31 - 1)] == [8, 2, 1]


# a perturbed cell of 40 atoms alone (layer 0 on the folded table, its edges in four parts, M1 to the readout in one kernel) and
# repeated: 480 atoms (functions, a warp per run), 1,800 (functions, a warp per receiver, the gradient's edges undivided), 3,240
# (M1 to the readout in five launches); the compressed cells have up to 112 edges a receiver, more than one chunk of 96 of the
# layer-1 gradient
@pytest.mark.gpu
@pytest.mark.parametrize("repeat,a,kwargs", [((3, 2, 2), 3.905, {}), ((5, 3, 3), 3.905, dict(agnesi=True, zbl=True, a0_scaled=True, a1_scaled=True)),
                                             ((9, 3, 3), 3.5, {}), ((6, 3, 3), 3.5, dict(channels=64)), ((4, 2, 2), 3.905, dict(one_type=True)),
                                             ((4, 2, 2), 3.5, dict(arch="large"))])
def test_repeated_cell_gives_the_energies_and_forces_of_the_cell(pkg, model_path, repeat, a, kwargs):
    """FP32 sums in another order and linears on another unit: energies and forces agree to 1e-6 of their size per operation
    chain (measured against the float64 oracle: 5e-7 and 1.2e-6), five times that."""
    kwargs = dict(kwargs)
    arch, one_type = kwargs.pop("arch", "medium"), kwargs.pop("one_type", False)
    path = model_path(arch, **kwargs)
    pos, cell, types = pkg.modelgen.srtio3((2, 2, 2), 0.05, 21, a)
    if one_type:
        types = np.full_like(types, 1)
    shifts = np.stack(np.meshgrid(*[np.arange(n) for n in repeat], indexing="ij"), axis=-1).reshape(-1, 3) @ cell
    small = pkg.Calculator(path, skin=0.5).calculate(pos, cell, types)
    copies = len(shifts)
    large = pkg.Calculator(path, skin=0.5).calculate((pos[None] + shifts[:, None]).reshape(-1, 3), cell * np.array(repeat)[:, None],
                                                     np.tile(types, copies))
    for key, scale in (("energies", np.abs(small["energies"]).max()), ("forces", np.abs(small["forces"]).max()),
                       ("stress", np.abs(small["stress"]).max())):
        got = np.asarray(large[key]).reshape((copies,) + small[key].shape) if key != "stress" else large[key][None]
        assert np.abs(got - small[key][None]).max() <= 6e-6 * scale, key


@pytest.mark.gpu
def test_forward_tensors_repeat_bit_for_bit(pkg, model_path):
    """No atomics up to the row adjoints: a difference between evaluations of the same positions is a race.  8,640 receivers keep
    every stage of the persistent linears busy, with tiles of 128, 126, 125 and 126 rows and K of 128 to 384."""
    pos, cell, types = pkg.modelgen.srtio3((12, 12, 12), 0.05, 3)
    calc = pkg.Calculator(model_path("medium"), skin=0.5)
    first = None
    for _ in range(6):
        calc.calculate(pos, cell, types)
        stages = {name: calc.evaluator.stage(name).copy() for name in ("A0", "H1", "A1", "dPhi1")}
        if first is None:
            first = stages
        for name, tensor in stages.items():
            assert np.array_equal(tensor, first[name]), name


@pytest.mark.gpu
@pytest.mark.parametrize("channels,options,tile,receivers", [(128, {}, 0, 193), (128, {}, 0, 1), (128, {}, 320, 100),
                                                             (64, dict(a0_scaled=True, a1_scaled=True, agnesi=True), 0, 211),
                                                             (64, dict(a0_scaled=True), 450, 499)])
def test_slices_of_the_sums_over_the_functions(pkg, model_path, channels, options, tile, receivers):
    """Layer 0 in slices that end inside an element's run of receivers (750 atoms: 450, 150 and 150 of a type), of one receiver, smaller
    and larger than a tile, against all at once.  A receiver's sums do not depend on the slice: A0 has the same bits.  Of the
    gradient a slice decides how many warps take a run, and the order of the atomic sums has no fixed order in the first place: the
    bounds of the tiled evaluation."""
    path = model_path("medium", channels=channels, **options)
    pos, cell, types = pkg.modelgen.srtio3((6, 5, 5), 0.05, 7)
    whole, sliced = pkg.Calculator(path, skin=0.5), pkg.Calculator(path, skin=0.5)
    with pytest.raises(ValueError):
        sliced.evaluator.set_moment_bytes(0)
    sliced.evaluator.set_moment_bytes(receivers * 3 * 16 * 64 * 4)
    sliced.evaluator.set_tile_size(tile)
    sliced.evaluator.set_profiling(True)
    a = whole.calculate(pos, cell, types)
    b = sliced.calculate(pos, cell, types)
    used = [c.evaluator.execution_plan_report["candidates"][0]["estimated_bytes"] for c in (whole, sliced)]
    assert used[0] - used[1] >= (len(pos) - receivers) * 3 * 16 * 64 * 4
    names = {name for name, _ms, _launches in sliced.evaluator.profile()}     # A0 made again for the reverse sweep has names of its own
    again = {"l0_forward_recompute", "gemm_a0_recompute"}
    assert {"l0_forward", "gemm_a0"} <= names and names & again == (again if tile else set())
    if tile == 0:
        assert np.array_equal(sliced.evaluator.stage("A0"), whole.evaluator.stage("A0"))
    assert np.abs(a["energies"] - b["energies"]).max() <= 1e-6
    assert np.abs(a["forces"] - b["forces"]).max() <= 1e-5
    assert np.abs(a["stress"] - b["stress"]).max() <= 1e-8


def layer0_gradient_error(pkg, path, cells):
    """Edge forces of a model with one interaction (nothing but layer 0) against float64 from the same adjoints of A0: the error's 2-norm
    and its part along the forces, both over the 2-norm of the forces."""
    from conftest import csr_from_positions
    from oracle import mace_numpy

    pos, cell, types = pkg.modelgen.srtio3(cells, 0.05, 11)
    first, src, shifts, xyz = csr_from_positions(pos, cell, 6.0)
    ev = pkg.MACEB200(path)
    ev.compute_node_energies_forces(len(pos), types, np.diff(first), src, types[src], xyz)
    oracle = mace_numpy.NumpyMACE(str(path))
    C, l_of_lm = oracle.C, np.array([0] + [1] * 3 + [2] * 5 + [3] * 7)
    adj = ev.stage("A0_adj").reshape(len(pos), 16, C)
    mixed = np.empty(adj.shape)                   # adjoint of the sums before the receiver's mixing matrix (mace.cpp:1486-1503)
    for a in range(oracle.A):
        for lm in range(16):
            mixed[types == a, lm] = adj[types == a, lm] @ oracle.WA0[a, l_of_lm[lm]].T
    recv = np.repeat(np.arange(len(pos)), np.diff(first))
    want = np.empty((len(src), 3))
    for e0 in range(0, len(src), 2000):
        e = slice(e0, e0 + 2000)
        r = np.linalg.norm(xyz[e], axis=1)
        Y, grad = mace_numpy.harmonics(3, xyz[e])
        R, dR = (v.reshape(-1, 4, C)[:, l_of_lm] for v in oracle._radial("R0", types[recv[e]], types[src[e]], r))
        weighted = mixed[recv[e]] * oracle.H0[types[src[e]]][:, None]
        along = ((weighted * dR).sum(axis=2) * Y).sum(axis=1)
        want[e] = -along[:, None] * xyz[e] / r[:, None] - np.einsum("em,edm->ed", (weighted * R).sum(axis=2), grad)
    error = ev.node_forces.reshape(-1, 3) - want
    return np.sqrt((error ** 2).sum() / (want ** 2).sum()), (error * want).sum() / (want ** 2).sum()


@pytest.mark.gpu
@pytest.mark.parametrize("channels,seed,cells,bound", [(128, 1, (6, 4, 4), 4e-8), (64, 2, (6, 6, 4), 1.2e-7)])
def test_gradient_on_the_functions_is_not_pulled_towards_zero(pkg, model_path, channels, seed, cells, bound):
    """A unit that truncates where FP32 rounds pulls each sum by 4e-8 an addition, in products with the functions and in the linear
    before them 1.7e-7 and 2.3e-7 here; errors that are rounded to nearest have no direction (some 1e5 components of 4e-7: 1e-9).
    Bounds: half a truncation for what the average in the linear leaves, and at 64 channels what the rounded coefficients of this model
    do (-1e-7 on the folded table too).  480 and 720 receivers are on the functions."""
    error, pull = layer0_gradient_error(pkg, model_path("medium", seed=seed, channels=channels, single_layer=True), cells)
    assert error <= 6e-7
    assert abs(pull) <= bound
