"""A warp's waits end in all its lanes together (xfluid_b200/csrc/xfp_warp_wait.h):
run on the host with lanes whose looks disagree, and required of every wait of the
wavefront kernel that a collective of the whole warp follows."""
import re
import subprocess
from pathlib import Path

ROOT = Path(__file__).resolve().parents[1]
WAVE = (ROOT / "xfluid_b200" / "csrc" / "xfp_wave.cu").read_text()


def test_lanes_that_see_different_answers_leave_together(tmp_path):
    exe = tmp_path / "warp_wait"
    cxx = "/usr/bin/g++" if Path("/usr/bin/g++").exists() else "g++"
    subprocess.run([cxx, "-std=c++17", "-O1", "-Wall", "-Werror", "-pthread",
                    str(ROOT / "tests" / "cpp" / "warp_wait_main.cpp"), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stderr


def test_the_kernels_waits_are_votes():
    """No lane of the wavefront kernel looks at a mbarrier outside warp_wait, and a
    warp's count of free consumer slots is one lane's look."""
    code = re.sub(r"//[^\n]*", "", WAVE)
    tries = [m.start() for m in re.finditer(r"\bmbar_try\(", code)][1:]   # (after its definition)
    assert tries
    for at in tries:
        assert "warp_wait(" in code[max(0, at - 120):at], code[at - 120:at + 60]
    compute = code[code.index("compute) {"):code.index("helper) {")]
    for m in re.finditer(r"room = ", compute):
        assert "__shfl_sync(" in compute[m.start():m.start() + 60] or compute[m.start():].startswith("room = 0;")
