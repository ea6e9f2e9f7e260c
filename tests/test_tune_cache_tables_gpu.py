"""Saved tunings name the shape table that their indices belong to: a line of an earlier table is not applied."""
import os
import re
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))
SCRIPT = """
import vanguard_b200 as vg
from vanguard_b200 import workloads as wl
nx, ny = 300, 200
with vg.Solver(vg.EULER, nx, ny, wl.euler_params()) as s:
    s.upload(wl.euler_quadrants_2d(nx, ny, seed=3))
    s.autotune(1.0 / nx, 0.8, limiter=0, measure=False)
    print(*s.launch_config(), s.schedule())
"""


def _apply(cache):
    env = dict(os.environ, VG_TUNE_CACHE=str(cache), PYTHONPATH=os.path.dirname(HERE))
    out = subprocess.run([sys.executable, "-c", SCRIPT], env=env, capture_output=True, text=True, timeout=300)
    assert out.returncode == 0, out.stderr[-2000:]
    return out.stdout.split(), [ln.split() for ln in cache.read_text().splitlines()]


def test_lines_of_another_table_are_tuned_again(tmp_path):
    cache = tmp_path / "tune.txt"
    cache.write_text("")
    _, (line,) = _apply(cache)
    key = line[0]
    assert re.fullmatch(r"v\d+_p\d+_b\d+_\d+x\d+_sm\d+_k\d+r\d+", key)
    # this table's line is applied as it stands
    other = [key, "3", "2", "1", "0"]
    cache.write_text(" ".join(other) + "\n")
    chosen, lines = _apply(cache)
    assert lines == [other] and chosen[:2] == ["3", "2"] and chosen[-1] == "1"
    # a line without the table, and one of an earlier revision of it, are not
    for stale in (re.sub(r"_k\d+r\d+$", "", key), re.sub(r"r\d+$", "r1", key)):
        cache.write_text(f"{stale} 3 2 1 0\n")
        _, lines = _apply(cache)
        assert [ln[0] for ln in lines] == [stale, key]


def test_names_give_the_register_caps(gpu):
    """Index 0 of the exact models' tables, whose caps differ by the length of the state."""
    from vanguard_b200 import workloads as wl
    names = []
    for model, W, prm in ((gpu.EULER, wl.euler_quadrants_2d(40, 30, seed=1), wl.euler_params()),
                          (gpu.EULER_REDUCED, wl.reduced_bubble_2d(40, 30), wl.reduced_params()),
                          (gpu.MHD, wl.mhd_vortex_2d(40, 30, seed=1), wl.mhd_params())):
        if model == gpu.MHD:
            W[3] = 0.1  # all nine planes
        with gpu.Solver(model, 40, 30, prm) as s:
            s.upload(W)
            s.set_launch_config(0, 0)
            names.append(s.launch_config()[2:])
    assert names == [("P128xL1/min7", "TX64xTY64/min8"), ("P128xL1/min7", "TX64xTY64"), ("P128xL1/min4", "TX64xTY64")]
