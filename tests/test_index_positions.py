"""The GPU index build's minimizers of long nodes, base by base (index_walk.cuh: minimizers_at),
compiled for the host and checked against the walk that its other nodes take, on random nodes with
many equal hashes and non-ACGT bases (tests/harness/index_positions.cpp)."""
import os
import subprocess

ROOT = os.path.abspath(os.path.join(os.path.dirname(__file__), ".."))


def test_minimizers_base_by_base_match_the_walk(tmp_path):
    exe = str(tmp_path / "index_positions")
    subprocess.run(["g++", "-std=c++17", "-O2", "-Wall", "-Wno-unknown-pragmas", "-Werror", "-o", exe,
                    os.path.join(ROOT, "tests", "harness", "index_positions.cpp")], check=True)
    out = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert out.returncode == 0 and out.stdout.startswith("ok"), out.stdout + out.stderr
