"""The rows that a Y sweep's blocks march when they are sized for the device, against measured sweeps: the rule is compiled from
sweep_table.cuh and has to choose among the measured segment lengths one whose time is near the best."""
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
NVCC = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
SMS = 148

# (model, nx = ny, block width TX, TY, resident blocks per SM): us a sweep by rows, on a B200
MEASURED = {
    ("euler_multiphysics", 2048, 128, 32, 5): {2: 1464, 4: 1210, 8: 1080, 14: 1069, 17: 1022, 24: 1009, 32: 1107, 45: 964,
                                               56: 1002, 76: 1106, 90: 1289, 114: 1479, 128: 1652},
    ("euler_multiphysics", 1024, 128, 32, 5): {2: 379, 4: 319, 6: 296, 8: 331, 11: 366, 14: 276, 17: 319, 28: 383, 45: 594,
                                               56: 678, 76: 908, 128: 1504},
    ("mhd_intermediate", 1024, 64, 64, 4): {2: 750, 4: 600, 8: 592, 14: 505, 17: 587, 24: 784, 28: 490, 32: 555, 38: 637, 45: 729,
                                            64: 975, 128: 1909},
    ("hpr_solid", 1024, 64, 64, 4): {2: 1499, 4: 1265, 8: 1204, 14: 1083, 20: 1364, 28: 1001, 32: 1149, 38: 1341, 45: 1539,
                                     64: 1941, 128: 3727},
    ("two_material_mixed", 2048, 128, 32, 5): {2: 1024, 8: 782, 17: 753, 24: 742, 38: 931, 45: 700, 56: 734, 76: 875, 128: 1299},
    ("hpr", 1024, 64, 64, 4): {2: 516, 6: 401, 14: 350, 20: 455, 28: 336, 32: 372, 38: 438, 56: 546, 128: 1034},
    ("mhd", 2048, 64, 64, 4): {2: 488, 8: 304, 17: 273, 28: 263, 45: 261, 56: 257, 64: 289, 76: 266, 90: 307, 114: 261, 128: 289},
    ("euler", 130, 64, 64, 8): {2: 13.8, 3: 13.8, 4: 15.7, 8: 20.5, 17: 28.7, 32: 42.8, 64: 75.3},
    ("mhd_mixed", 2048, 128, 32, 5): {2: 217, 8: 158, 17: 151, 28: 153, 45: 143, 56: 149, 76: 173, 90: 202, 128: 257},
}


@pytest.fixture(scope="module")
def chosen(tmp_path_factory):
    """The rule's rows for every entry."""
    d = tmp_path_factory.mktemp("rule")
    calls = "".join(f'    std::printf("%d\\n", vg::y_segment_rows({97 if n == 130 else n}, {-(-n // tx)}, {tx}, {res * SMS}L, {SMS}, {ty}));\n'
                    for _, n, tx, ty, res in MEASURED)
    (d / "rule.cu").write_text('#include <cstdio>\n#include "sweep_table.cuh"\nint main() {\n' + calls + "}\n")
    env = {k: v for k, v in os.environ.items() if k not in ("CXX", "CC")}
    subprocess.run([NVCC, "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", "-ccbin", "g++", "-I",
                    os.path.join(HERE, "..", "vanguard_b200", "csrc"), "-o", str(d / "rule"), str(d / "rule.cu")],
                   check=True, env=env)
    rows = subprocess.run([str(d / "rule")], capture_output=True, text=True, check=True).stdout.split()
    return dict(zip(MEASURED, map(int, rows)))


@pytest.mark.parametrize("key", list(MEASURED), ids=lambda k: f"{k[0]}_{k[1]}")
def test_rule_is_near_the_best(chosen, key):
    """Within 1.1 of the best measured length, the chosen one's time read off between its measured neighbours."""
    t, rows = MEASURED[key], chosen[key]
    lo, hi = max(r for r in t if r <= rows), min(r for r in t if r >= rows)
    assert max(t[lo], t[hi]) <= 1.1 * min(t.values()), (rows, lo, hi)
