"""The lookup of bigraph node ids (gaf_format.cuh: IdTable), dense and hashed, compiled for the host and
checked against a std::map on both sides of the rule between them (tests/harness/id_table.cpp)."""
import os
import subprocess

ROOT = os.path.abspath(os.path.join(os.path.dirname(__file__), ".."))


def test_id_lookup_matches_a_map(tmp_path):
    exe = str(tmp_path / "id_table")
    subprocess.run(["g++", "-std=c++17", "-O2", "-Wall", "-Wno-unknown-pragmas", "-Werror", "-fsanitize=undefined", "-fno-sanitize-recover", "-o", exe,
                    os.path.join(ROOT, "tests", "harness", "id_table.cpp")], check=True)
    out = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert out.returncode == 0 and out.stdout.startswith("ok"), out.stdout + out.stderr
