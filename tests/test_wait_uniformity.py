"""A role that goes on to warp-wide instructions leaves its waits with one answer per warp.

The kernels' waits are bounded and an abort flag releases them. Evaluated lane by lane, a wait can then end with "complete" in some
lanes of a warp and "give up" in others; if the next step is a warp-wide instruction (elect.sync in front of an MMA or a commit, a
tensor-memory load or store, __syncwarp, a vote) the lanes would meet at different ones, which may hang. Running such a case needs
a kernel that fails, so the rule is checked on the sources: in every role (and every function called by one) that has a warp-wide
instruction, each wait is a warp's, made uniform at once, one that no flag releases (its flag is `never`), or one that no lane leaves
by: the lane notes its answer (`ok = wait`, or `alive = false` where the loop around it votes on `alive`) and walks on. That the warp's
wait itself has one answer is shown on the device by llattn_wait_selftest."""
import importlib
import os
import re

import pytest

WARP_WIDE = re.compile(r"\b(tmem_(ld|st|wait)\w*|mma_\w+|__syncwarp|__shfl\w*|__any_sync|__all_sync)\s*(<[^>]*>)?\(")
LANE_WAIT = re.compile(r"\b(mbar_wait|filled|emptied)\s*\(")


def _source(pkg, name):
    bld = importlib.import_module(pkg.__name__ + ".build")
    text = open(os.path.join(bld.CSRC, name)).read()
    return re.sub(r"//[^\n]*", "", text)


def _block(text, at):
    """The {...} block that opens at or behind `at`, and where it ends."""
    start = text.index("{", at)
    depth = 0
    for i in range(start, len(text)):
        depth += {"{": 1, "}": -1}.get(text[i], 0)
        if depth == 0:
            return text[start:i + 1], i + 1
    raise ValueError("unbalanced braces")


def _roles(text, first):
    """The blocks of the if / else if / else chain that begins with `first`."""
    at, out = text.index(first), []
    while True:
        block, end = _block(text, at)
        out.append(block)
        if not re.match(r"\s*else\b", text[end:]):
            return out
        at = end


def _lane_waits(block):
    """Waits of a block with warp-wide instructions by whose answer some lanes of a warp may part from others."""
    if not WARP_WIDE.search(block):
        return []
    bad = []
    for m in LANE_WAIT.finditer(block):
        call = block[m.start():block.index(";", m.start())]
        before = block[:m.start()].rstrip()
        uniform = before.endswith(("uniform_i32(ptx::", "__all_sync(0xffffffffu, ptx::"))
        rest = block[m.start():block.index("\n", m.start())]
        votes = "for (int ii = i0; ii < i1 && __all_sync(0xffffffffu, alive); ++ii)" in block
        stays = before.endswith("    ok = ptx::") or (votes and rest.endswith("{ alive = false; errbits |= ERR_WAIT_SOFTMAX; }"))
        if not uniform and not stays and "&never" not in call:
            bad.append(call[:100])
    return bad


def test_projection_roles(pkg):
    roles = _roles(_source(pkg, "dense_i8.cuh"), "if (warp < DW_FOLD_WARPS)")
    assert len(roles) == 5 and sum(bool(WARP_WIDE.search(r)) for r in roles) == 3          # fold, producer, MMA issue
    assert [w for r in roles for w in _lane_waits(r)] == []


def test_attention_roles(pkg):
    text = _source(pkg, "attn_kernel.cuh")
    roles = _roles(text, "if (warp < SOFTMAX_WARPS)")
    assert len(roles) == 5 and sum(bool(WARP_WIDE.search(r)) for r in roles) == 4          # all but the dequantising warps
    called = [_block(text, text.index(f))[0] for f in ("float raise_reference(", "float2 raise_reference_rows16(")]
    assert [w for r in roles + called for w in _lane_waits(r)] == []


def test_the_check_itself():
    lane = "{ if (!ptx::mbar_wait(BAR(0), 0, abort_flag)) break;\n ptx::tmem_ld16(t, r); }"
    assert len(_lane_waits(lane)) == 1
    assert _lane_waits(lane.replace("mbar_wait(", "mbar_wait_warp(")) == []
    assert _lane_waits(lane.replace("ptx::tmem_ld16(t, r);", "")) == []
    assert len(_lane_waits("{ if (!ptx::mbar_wait(B, 0, f)) { alive = false; errbits |= ERR_WAIT_SOFTMAX; }\n ptx::tmem_ld16(t, r); }")) == 1
