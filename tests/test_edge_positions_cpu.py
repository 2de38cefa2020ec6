"""CPU tests of the kernels' arithmetic on edge positions, which reach
2^31 - 2: the host build of include/pm/pm_edges.cuh walks rows that end there,
and no kernel steps through a row with an int32 position."""
import os
import re
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "polymer_b200", "csrc")
INC = os.path.join(ROOT, "include", "pm")


def test_rows_near_the_last_position(tmp_path):
    exe = str(tmp_path / "edge_positions")
    src = os.path.join(ROOT, "tests", "cpp", "edge_positions.cpp")
    subprocess.run(["g++", "-O2", "-std=c++17", "-x", "c++", "-I" + INC, src, "-o", exe], check=True)
    p = subprocess.run([exe], capture_output=True, text=True)
    assert p.returncode == 0, p.stdout
    assert int(p.stdout) > 3000


def test_no_kernel_steps_an_int32_position():
    # over the adjacency itself; the degree-sorted copies refuse m above 2^31 - 8192
    step = re.compile(r"for \((?:const )?int(?:32_t)? (e|b|o|base|x)\b[^)]*;[^;]*;[^)]*\+=")
    copies = {"pm_sorted.cu", "pm_sorted.cuh"}
    for folder in (CSRC, INC):
        for name in sorted(os.listdir(folder)):
            if name in copies or not name.endswith((".cu", ".cuh")):
                continue
            for i, line in enumerate(open(os.path.join(folder, name)), 1):
                hit = step.search(line)
                # a count from 0 is not a position
                assert not hit or "= 0;" in hit.group(0), "%s:%d: %s" % (name, i, line.strip())
