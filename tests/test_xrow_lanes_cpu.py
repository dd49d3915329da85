"""The x stage's warp code on the CPU, its lanes in several orders between the warp-wide
synchronisations: at every compiled length, with any number of the warp's rows
present, the CFL maxima are those of the rows (evaluated term by term) and no result
depends on the order."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_lanes_may_run_in_any_order(tmp_path):
    (tmp_path / "cuda_runtime.h").write_text("#pragma once\n#include <stddef.h>\n")  # the types are the program's own
    exe = str(tmp_path / "xrow_lanes")
    subprocess.run(["g++", "-std=c++17", "-O1", "-w", f"-I{tmp_path}",
                    f"-I{os.path.join(ROOT, 'final-single-block-_b200', 'csrc')}", "-o", exe,
                    os.path.join(ROOT, "tests", "xrow_lanes.cpp")], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
