"""The PCG loop's host side (xfluid_b200/csrc/xfp_loop.h), which reads the scalars while
the next launch of its graph runs, against a CUDA runtime of the test's own."""
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]


@pytest.fixture(scope="module")
def loop(tmp_path_factory):
    exe = tmp_path_factory.mktemp("loop") / "loop_main"
    cxx = "/usr/bin/g++" if Path("/usr/bin/g++").exists() else "g++"
    subprocess.run([cxx, "-std=c++17", "-O1", "-Wall", "-Werror", "-I/usr/local/cuda/include",
                    str(ROOT / "tests" / "cpp" / "loop_main.cpp"), "-o", str(exe)], check=True)
    return exe


@pytest.mark.parametrize("case", ["half", "expired", "both", "endless", "refused", "kinds", "check_every"])
def test_reads_beside_a_running_launch(loop, case):
    r = subprocess.run([str(loop), case], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stderr


def test_done_is_the_kernels_last_store():
    """What the second read relies on: every kernel that ends a solve does it through
    end_solve, which fences before it sets the flag."""
    csrc = ROOT / "xfluid_b200" / "csrc"
    stores = [line.strip() for f in sorted(csrc.glob("*.cu*")) for line in f.read_text().splitlines()
              if "done" in line and "= 1;" in line]
    assert stores == ["*(volatile int*)&sc->done = 1;"]
    common = (csrc / "xfp_common.cuh").read_text()
    body = common[common.index("void end_solve("):]
    assert body.index("sc->status = status;") < body.index("__threadfence_system();") < body.index("sc->done = 1;")


def test_a_context_allocates_no_page_locked_memory():
    """cudaHostAlloc takes longer than all else that creating a context does."""
    capi = (ROOT / "xfluid_b200" / "csrc" / "xfp_capi.cu").read_text()
    create = capi[capi.index("int xfp_create("):capi.index("int xfp_destroy(")]
    assert "cudaHostAlloc" not in create and "cudaMallocHost" not in create
