"""The rules that deal a receiver's edges to blocks and warps (csrc/part_rules.hpp), against measured kernel times."""
import ctypes
import re
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]

# (hidden shape, channels, list edges, kernel): receivers -> us at 1, 2, 4, 8 parts (layer-0 sums: 1 and 4 parts) on 148 SMs, one
# launch of each kernel by CUDA events, medians of seven.  Layer 0 with more than some hundred receivers runs on the table where the
# model has no 64 radial functions, or more than ten types.
MEASURED = {
    (1, 128, 96.6, "l0_forward"): {40: (46, 20), 600: (51, 38), 1080: (59, 46), 2160: (76, 82), 2560: (111, 97), 3240: (133, 117),
                                   4500: (138, 157), 6480: (195, 215), 7200: (222, 238), 7560: (238, 250)},
    (1, 64, 96.6, "l0_forward"): {40: (55, 25), 1500: (68, 48), 2160: (73, 64), 3240: (77, 85), 3600: (79, 88), 4500: (85, 106),
                                  6480: (133, 144), 7560: (137, 166)},
    (0, 32, 58.5, "l0_forward"): {40: (23, 13), 1500: (31, 24), 2560: (32, 29), 4500: (39, 45), 8640: (66, 73)},
    (1, 128, 96.6, "l0_reverse"): {40: (66, 39, 25, 17), 320: (70, 41, 31, 33), 1080: (82, 76, 74, 76), 2160: (138, 119, 123, 142),
                                   5000: (243, 248, 271, 312), 7560: (369, 365, 398, 465)},
    (1, 64, 96.6, "l0_reverse"): {40: (50, 29, 19, 15), 600: (52, 35, 37, 35), 1500: (68, 68, 64, 70), 5000: (179, 171, 177, 201)},
    (0, 32, 58.5, "l0_reverse"): {40: (31, 19, 15, 11), 600: (35, 25, 21, 23), 1080: (35, 29, 31, 33), 2160: (48, 50, 48, 58)},
    (1, 128, 96.6, "l1_forward"): {40: (39, 35, 23, 18), 80: (39, 37, 25, 29), 320: (51, 64, 64, 70), 1080: (111, 144, 164, 199)},
    (1, 64, 96.6, "l1_forward"): {80: (39, 37, 25, 19), 160: (39, 37, 27, 31), 600: (49, 66, 66, 70)},
    (0, 32, 58.5, "l1_forward"): {40: (21, 17, 12, 10), 160: (21, 17, 13, 15), 320: (21, 18, 19, 21), 600: (21, 27, 27, 31),
                                  1080: (23, 31, 35, 47)},
    (0, 128, 58.5, "l1_forward"): {40: (25, 21, 15, 13), 160: (27, 21, 17, 21), 320: (29, 23, 27, 29), 600: (29, 37, 37, 45)},
    (1, 128, 96.6, "l1_reverse"): {40: (38, 25, 23, 23), 160: (50, 44, 44, 50), 320: (72, 66, 70, 87), 600: (111, 109, 119, 154),
                                   1080: (173, 179, 204, 267), 5000: (699, 762, 904, 1308)},
    (1, 64, 96.6, "l1_reverse"): {40: (23, 17, 17, 19), 320: (44, 42, 50, 68), 1080: (97, 105, 136, 199)},
    (2, 128, 96.6, "l1_reverse"): {40: (56, 35, 37, 38), 160: (85, 80, 83, 103), 600: (220, 236, 275, 359)},
    (0, 32, 58.5, "l1_reverse"): {40: (31, 21, 15, 13), 600: (35, 33, 33, 35), 1080: (37, 39, 45, 56), 1500: (60, 54, 60, 72),
                                  2160: (68, 72, 80, 99)},
    (0, 128, 58.5, "l1_reverse"): {40: (31, 21, 17, 13), 320: (39, 41, 39, 43), 1080: (86, 91, 99, 117)},
}


@pytest.mark.parametrize("key", list(MEASURED), ids=lambda k: f"{k[3]}-shape{k[0]}-{k[1]}")
def test_parts_chosen_are_among_the_fastest(part_rule, key):
    """No slower than the undivided kernel and within a twelfth of the fastest (2 us: the grain of the event times)."""
    shape, channels, edges, kernel = key
    for receivers, times in MEASURED[key].items():
        by_parts = dict(zip((1, 4) if kernel == "l0_forward" else (1, 2, 4, 8), times))
        took = by_parts[part_rule(kernel, 148, channels, shape, edges, receivers)]
        assert took <= by_parts[1] + 2, (receivers, by_parts)
        assert took <= min(times) * 13 / 12 + 2, (receivers, by_parts)


def test_parts_stay_within_the_builds(part_rule):
    """Layer-0 sums have builds for one and four warps per receiver, clusters at most eight blocks; a graph without edges, or
    one receiver, is dealt out within those limits at every width."""
    for channels in (32, 64, 96, 128, 160, 192, 224, 256):
        for shape in (0, 1):
            for receivers in (1, 2, 7, 40, 1000, 123457, 2 ** 31 - 1):
                for edges in (0.0, 1.0, 58.5, 400.0):
                    args = (148, channels, shape, edges, receivers)
                    assert part_rule("l0_forward", *args) in (1, 4)
                    for kernel in ("l1_forward", "l1_reverse", "l0_reverse"):
                        assert part_rule(kernel, *args) in (1, 2, 4, 8)
                    assert part_rule("l1_forward", *args) * receivers <= max(receivers, 148 * 5)


def test_tables_of_a_preparation_that_threw_are_made_by_the_next(tmp_path):
    """Bookkeeping of the type-dependent tables (csrc/type_tables.hpp): whichever of the uploads throws, the next preparation with
    the same types makes what is missing, and other types make everything again."""
    header = ROOT / "symmetrix-xl_b200" / "csrc" / "type_tables.hpp"
    (tmp_path / "tables.cpp").write_text(
        f'#include "{header}"\n#include <stdexcept>\n#include <string>\n'
        "static sxb::TypeTables t;\nstatic int made[3];      // type that basis, folded table and pair tables were made for\n"
        'extern "C" int prepare(int type, int on_basis, int fail)\n{\n    try {\n'
        "        t.request({type});\n"
        "        const auto make = [&](int table, bool& stands) {\n"
        '            if (stands) return;\n            made[table] = -1;\n            if (fail == table) throw std::runtime_error("");\n'
        "            made[table] = type;\n            stands = true;\n        };\n"
        "        on_basis ? make(0, t.basis) : make(1, t.folded);\n        make(2, t.pairs);\n"
        "    } catch (const std::runtime_error&) { return -1; }\n"
        "    return made[on_basis ? 0 : 1] == type && made[2] == type;\n}\n")
    subprocess.run(["g++", "-std=c++17", "-Wall", "-Werror", "-shared", "-fPIC", "-o", str(tmp_path / "tables.so"),
                    str(tmp_path / "tables.cpp")], check=True)
    lib = ctypes.CDLL(str(tmp_path / "tables.so"))
    for on_basis in (0, 1):
        for fail in (1 - on_basis, 2):
            assert lib.prepare(7, on_basis, -1) == 1
            assert lib.prepare(8, on_basis, fail) == -1
            assert lib.prepare(8, on_basis, fail) == -1       # the same types again: not taken for prepared
            assert lib.prepare(8, on_basis, -1) == 1
            assert lib.prepare(8, 1 - on_basis, -1) == 1
            assert lib.prepare(7, on_basis, fail) == -1 and lib.prepare(7, on_basis, -1) == 1


def test_row_batches_are_taken_in_order():
    """The layer-1 gradient on channel pairs asks for batch b + 1 of the row adjoints when it takes batch b (csrc/edge_kernels_pairs.cuh):
    an edge's body takes every batch that is stored, once and in order, and leaves none outstanding."""
    text = (ROOT / "symmetrix-xl_b200" / "csrc" / "generated" / "structures.h").read_text()
    for name in ("S1", "S2"):
        batches = int(re.search(rf"#define SXB_{name}_ROW_BATCHES (\d+)", text).group(1))
        body = re.search(rf"#define SXB_{name}_L1_REVERSE_EDGE_BODY (.*?[^\\])\n(?!\s)", text, re.S).group(1)
        stored = re.search(rf"#define SXB_{name}_L1_ADJOINT_ROWS (.*?[^\\])\n(?!\s)", text, re.S).group(1)
        assert [int(b) for b in re.findall(r"\bROWS\((\d+)\)", body)] == list(range(batches))
        assert [int(b) for b in re.findall(r"\bSTORE\((\d+)\)", stored)] == list(range(batches))
