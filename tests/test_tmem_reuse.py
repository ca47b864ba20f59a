"""Tensor memory that an MMA still reads is not written by the next one before the first has completed.

S of tile t + 2 goes into the buffer whose P the MMA of tile t reads. PTX orders two MMAs of one thread only where they have the same
accumulator and shape, which S = Q K^T and O += P V have not, so the issuing warp has to see P V complete first. A missing wait shows in no
result, it depends on the hardware's own order, so the rule is checked on the source."""
import importlib
import os
import re


def _issuer(pkg):
    bld = importlib.import_module(pkg.__name__ + ".build")
    text = re.sub(r"//[^\n]*", "", open(os.path.join(bld.CSRC, "attn_kernel.cuh")).read())
    return text[text.index("} else if (warp == WARP_MMA) {"):]


def test_s_waits_for_the_pv_that_reads_its_buffer(pkg):
    text = _issuer(pkg)
    issue = text[text.index("auto issue_s ="):text.index("return true;")]
    wait = re.search(r"if \(tt >= 2 && !uniform_i32\(ptx::mbar_wait\(BAR\(B_PV_DONE \+ b\), \(\(tt >> 1\) - 1\) & 1, abort_flag\)\)\) return false;", issue)
    assert wait, "S is issued without a wait for the P V of the tile before last"
    assert wait.end() < issue.index("tc_fence_after") < issue.index("mma_ts_s8_warp")
    # every S goes through it: no other place of the kernel issues one
    assert len(re.findall(r"\bmma_ts_s8_warp\b", text)) == 1
