"""The wavefronts' edge values (xfluid_b200/csrc/xfp_edges.h): a block waits for exactly
the groups that its neighbours send, or it would wait until its time is up."""
import subprocess
from pathlib import Path

ROOT = Path(__file__).resolve().parents[1]


def test_blocks_wait_for_what_is_sent(tmp_path):
    exe = tmp_path / "edges"
    cxx = "/usr/bin/g++" if Path("/usr/bin/g++").exists() else "g++"
    subprocess.run([cxx, "-std=c++17", "-O1", "-Wall", "-Werror", str(ROOT / "tests" / "cpp" / "edges_main.cpp"),
                    "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stderr
