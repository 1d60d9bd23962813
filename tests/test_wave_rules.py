"""Orderings that the wavefront kernel (xfluid_b200/csrc/xfp_wave.cu) owes the PTX
memory model and that no run can prove: read off its source."""
import re
from pathlib import Path

CODE = re.sub(r"//[^\n]*", "", (Path(__file__).resolve().parents[1] / "xfluid_b200" / "csrc" / "xfp_wave.cu").read_text())


def test_slots_are_refilled_behind_a_proxy_fence():
    """A slot that ordinary stores have written (results, cleared edges) is refilled by
    a bulk copy: of the async proxy, so the copying lane fences first, after the
    warp's barrier that collects the other lanes' accesses."""
    assert "fence.proxy.async.shared::cta" in CODE
    copies = [m.start() for m in re.finditer(r"\bbulk_load\(", CODE)][1:]   # (after its definition)
    assert copies
    for at in copies:
        before = CODE[max(0, at - 500):at]
        assert "fence_bulk();" in before
        assert "__syncwarp();" in before[:before.rindex("fence_bulk();")]
