"""Memory orderings of the tensor-core GEMM that no run can be relied on to show (without them the results are
right on most days), read from the kernel's source."""

from pathlib import Path

SOURCE = (Path(__file__).resolve().parents[1] / "fused-dequantisation-kernels_b200" / "csrc" / "gemm_lut_tc.cu").read_text()


def between(first: str, last: str) -> str:
    start = SOURCE.index(first)
    return SOURCE[start: SOURCE.index(last, start)]


def test_partial_sums_are_read_after_every_lanes_acquire():
    """One lane per share polls its flag, all lanes read the share: a vote in between implies no memory ordering,
    `__syncwarp` does."""
    assert "__syncwarp();" in between("ld.acquire.gpu.global", "__ldcg(theirs")


def test_flags_are_published_after_every_lanes_stores():
    hand_over = between("if (begin != 0) {  // publish", "st.relaxed.gpu.global")
    assert 0 <= hand_over.index("__syncwarp();") < hand_over.index("__threadfence();")


def test_code_slots_are_handed_back_behind_a_proxy_fence():
    """Plain reads and the bulk copy that refills the slot go through different proxies."""
    release = between("auto release = [&] {", "mbar_arrive(held)")
    assert release.index("fence.proxy.async.shared::cta") < release.index("__syncwarp();")


def test_only_narrow_tiles_carry_the_eight_column_form():
    """Compiled into the other forms it cost them registers that they spilled, and large products 2 % of their time."""
    assert SOURCE.count("tmem_load8(") == 2  # its definition, and the one use
    assert "if (FORM == kTcNarrow && parts > 1" in between("Several shares of a tile", "tmem_load8(taddr")
