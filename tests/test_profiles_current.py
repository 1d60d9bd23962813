"""Committed profiles and the bench's line name kernels that exist."""
import re
from pathlib import Path

ROOT = Path(__file__).resolve().parents[1]


def test_profiled_kernels_exist():
    source = "\n".join(f.read_text() for f in sorted((ROOT / "xfluid_b200" / "csrc").glob("*.cu")))
    known = set(re.findall(r"\b(\w+_kernel)\(", source))
    for f in [ROOT / "bench.py", *sorted((ROOT / "profiles").iterdir())]:
        gone = set(re.findall(r"\b(\w+_kernel)\b", f.read_text())) - known
        assert not gone, (f.name, sorted(gone))


def test_the_bench_reads_no_profile():
    assert "profiles" not in (ROOT / "bench.py").read_text()
