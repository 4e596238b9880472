"""The traceback's step bits (csrc/wordslice.cuh: diagonal_rows, up_run), compiled for the host
and checked cell by cell against the scores of the columns they come from
(tests/harness/walk_props.cpp)."""
import os
import subprocess

ROOT = os.path.abspath(os.path.join(os.path.dirname(__file__), ".."))


def test_step_bits_match_the_scores(tmp_path):
    exe = str(tmp_path / "walk_props")
    subprocess.run(["g++", "-std=c++17", "-O2", "-Wall", "-Werror", "-o", exe,
                    os.path.join(ROOT, "tests", "harness", "walk_props.cpp")], check=True)
    out = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert out.returncode == 0 and out.stdout.startswith("ok"), out.stdout + out.stderr
