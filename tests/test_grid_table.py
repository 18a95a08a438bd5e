"""The fixed table of kernel grid sizes (bulbit_b200/csrc/grid_table.h), which
queries that must not allocate consult: tests/cpp/grid_table_test.cpp, compiled
here. The library asks no growing container in its place."""
import os
import shutil
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "bulbit_b200", "csrc")


def test_grid_table(tmp_path):
    exe = str(tmp_path / "grid_table_test")
    cmd = [shutil.which("g++") or "g++", "-std=c++20", "-O2", "-pthread", "-I", CSRC, "-o", exe,
           os.path.join(ROOT, "tests", "cpp", "grid_table_test.cpp")]
    built = subprocess.run(cmd, capture_output=True, text=True)
    assert built.returncode == 0, built.stderr[-2000:]
    p = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert p.returncode == 0 and p.stdout.endswith("0 failures\n"), p.stdout[-2000:]


def test_grids_come_from_the_table():
    code = open(os.path.join(CSRC, "accel.cu")).read()
    body = code[code.index("int PersistentGrid("):]
    body = body[:body.index("\n}\n")]
    assert "static GridTable" in body
    assert "std::" not in body.replace("std::max", "")
