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


def test_an_expired_wait_leaves_no_copies_behind():
    """Only a wait inside a cluster ends a loop early, and then the CTAs of the cluster
    leave after the copies to their slots: the courier goes on, and no sleep stands
    for a wait."""
    courier = CODE[CODE.index("courier) {"):CODE.index("if constexpr (!FACTOR) {\n      if (!skip")]
    expired = courier[courier.index("sp.step(g.ctl, g.spin_limit)"):]
    assert "late = true;" in expired and "break;" not in expired
    end = CODE[CODE.index("if (*(volatile int*)&s_broken != 0) {"):]
    assert end.index("mbar_try(") < end.index("cluster_sync();") < end.index("break;")
    assert "__nanosleep" not in CODE


def test_free_slots_are_told_with_release_and_read_with_acquire():
    """A block writes edge values into a neighbour's slot once the neighbour has told it
    that the slot is free; what the neighbour read from the slot has to come first."""
    assert "st.release.cta.shared::cluster" in CODE and "ld.acquire.cluster.shared" in CODE
    told = [line for line in CODE.splitlines() if "if (told)" in line]
    assert told and all("st_release_s32(" in line for line in told)
    looks = re.findall(r"room = [^;]*(?:limit|freed)[^;]*;", CODE)
    assert len(looks) >= 3 and all("ld_acquire_s32(" in look for look in looks)
