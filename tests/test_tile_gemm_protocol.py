"""Who may touch the row scales of the tile GEMMs when, read from the source: the warps that read what a bulk copy brought wait on
the barrier that the copy completes on, and their hand-back, behind which a slot may be copied into again, releases their reads."""
import re

from test_dependency_wait import CSRC, code_of


def test_row_scales_are_read_between_their_copy_and_the_hand_back():
    code = code_of(CSRC / "gemm.cu")
    split = code.index("setmaxnreg_inc_promo()")
    producer, readers = code[code.index("setmaxnreg_dec_aux()"):split], code[split:code.index("#undef ACC")]
    copy = re.search(r"bulk_load\(smem_u32\(&aux->row_scale.*?,\s*(\w+)\);", producer, re.S)
    barriers = re.findall(r"&aux->(\w+)\[", re.findall(rf"\b{copy.group(1)} = ([^;]*);", producer[:copy.start()])[-1])
    assert barriers
    for bar in barriers:
        assert re.search(rf"mbar_wait_all\(smem_u32\(&aux->{bar}\[", readers), f"nobody who reads row_scale waits for {bar}"
    for signal in ("drained", "handed"):
        call = re.search(rf"__syncwarp\(\);\s*if \(lane == 0\) (\w+)\([^;]*&?aux->{signal}\[", readers)
        assert call and "_release_" in call.group(1), f"{signal} orders no reads"
    common = code_of(CSRC / "common.cuh")
    for poll in ("ld_acquire_shared", "flags_equal"):
        body = common[common.index(f" {poll}("):]
        assert "ld.acquire.cta" in body[:body.index("}\n")]
