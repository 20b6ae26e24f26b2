import ctypes
import subprocess
import sys
from pathlib import Path

import numpy as np
import pytest

ROOT = Path(__file__).resolve().parents[1]
if str(ROOT) not in sys.path:
    sys.path.insert(0, str(ROOT))

import __graft_entry__ as graft  # noqa: E402


def pytest_configure(config):
    config.addinivalue_line("markers", "gpu: needs a CUDA device (B200)")


@pytest.fixture(scope="session")
def pkg():
    return graft.load_package()


@pytest.fixture(scope="session")
def model_dir(tmp_path_factory):
    return tmp_path_factory.mktemp("models")


@pytest.fixture(scope="session")
def model_path(pkg, model_dir):
    """Returns a function (arch, seed) -> path of a generated model JSON (cached per session)."""
    cache = {}

    def get(arch="small", seed=1, **kwargs):
        key = (arch, seed, tuple(sorted(kwargs.items())))
        if key not in cache:
            path = model_dir / f"{arch}_{seed}_{len(cache)}.json"
            pkg.modelgen.write_model(path, arch, seed=seed, **kwargs)
            cache[key] = path
        return cache[key]

    return get


@pytest.fixture(scope="session")
def part_rule(tmp_path_factory):
    """rule(kernel, sms, channels, shape, edges, receivers, types=3) -> parts, compiled from the library's header: the calls that the
    launches make.  "layer0_on_basis" is 1 where layer 0 runs on the radial functions and "l0_moments_reverse" gives its parts."""
    folder = tmp_path_factory.mktemp("part_rules")
    header = ROOT / "symmetrix-xl_b200" / "csrc" / "part_rules.hpp"
    kernels = {"l0_forward": "receivers", "l1_forward": "receivers", "l1_reverse": "receivers", "l0_reverse": "receivers",
               "layer0_on_basis": "receivers, types", "l0_moments_reverse": "receivers, types"}
    (folder / "rules.cpp").write_text(
        f'#include "{header}"\n'
        'extern "C" int rule(int kernel, int sms, int channels, int shape, double edges, long receivers, int types)\n'
        "{\n    const sxb::PartRules r{sms, channels, shape, edges};\n    switch (kernel) {\n"
        + "".join(f"    case {i}: return r.{name}({args});\n" for i, (name, args) in enumerate(kernels.items()))
        + "    }\n    return 0 * types;\n}\n")
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-Werror", "-shared", "-fPIC", "-o", str(folder / "rules.so"),
                    str(folder / "rules.cpp")], check=True)
    lib = ctypes.CDLL(str(folder / "rules.so"))
    lib.rule.argtypes = [ctypes.c_int] * 4 + [ctypes.c_double, ctypes.c_long, ctypes.c_int]
    return lambda kernel, *args, types=3: lib.rule(list(kernels).index(kernel), *args, types)


def csr_from_positions(positions, cell, cutoff):
    from oracle import neighbor

    first, src, shifts = neighbor.build_neighbor_graph(positions, cell, cutoff)
    xyz = neighbor.edge_vectors(positions, cell, first, src, shifts)
    return first, src, shifts, xyz
