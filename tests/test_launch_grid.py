"""A launch shape's blocks_per_sm caps every kernel of a pass (csrc/launch_grid.h), the second fill's
one-warp blocks included (tests/harness/launch_grid.cpp)."""
import os
import subprocess

ROOT = os.path.abspath(os.path.join(os.path.dirname(__file__), ".."))


def test_blocks_stay_within_the_cap(tmp_path):
    exe = str(tmp_path / "launch_grid")
    subprocess.run(["g++", "-std=c++17", "-O2", "-Wall", "-Werror", "-fsanitize=undefined", "-fno-sanitize-recover", "-o", exe,
                    os.path.join(ROOT, "tests", "harness", "launch_grid.cpp")], check=True)
    out = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert out.returncode == 0 and out.stdout.startswith("ok"), out.stdout + out.stderr
