"""Every kernel that is launched as a dependent one waits for the kernel ahead of it on every way through it, before it reads or writes
anything: a way out in front of the wait would let the kernels behind it start while that one still runs. Checked on the sources, the
way out is one that no test can take (a base of shared memory that is not aligned)."""
import importlib
import os
import re

KERNEL = re.compile(r"__global__ void\s+__launch_bounds__\((?:[^()]|\([^()]*\))*\)\s*(\w+)\s*\(")
BEFORE_IT = re.compile(r"\breturn;|\breport_error\(|\batomic\w+\(|\b__ld\w+\(|\b__st\w+\(|\bbulk_g2s\(|\bcp_async16\(|\w+_(body|tiles)\b\s*[<(]")


def _kernels(pkg):
    bld = importlib.import_module(pkg.__name__ + ".build")
    for name in sorted(os.listdir(bld.CSRC)):
        if name.endswith(".cuh"):
            text = re.sub(r"//[^\n]*", "", open(os.path.join(bld.CSRC, name)).read())
            for m in KERNEL.finditer(text):
                start = text.index("{", m.end())
                depth, end = 0, start
                while True:
                    depth += {"{": 1, "}": -1}.get(text[end], 0)
                    end += 1
                    if depth == 0:
                        break
                yield m.group(1), text[start:end]


def _misses(body):
    """What happens in front of the wait (None: there is no wait). A block that leaves the kernel and begins with a wait of its own is none of it."""
    body = re.sub(r"\bif \([^{}]*\) \{\s*ptx::grid_dependency_wait\(\);[^{}]*\breturn;\s*\}", "", body)
    at = body.find("ptx::grid_dependency_wait();")
    if at < 0:
        return None
    m = BEFORE_IT.search(body[:at])
    return m.group(0) if m else ""


def test_every_kernel_waits_first(pkg):
    found = dict(_kernels(pkg))
    assert set(found) == {"attn_tile_kernel", "dense_strip_kernel", "dense_tile_kernel", "dense_wide_kernel", "kv_commit_kernel", "combine_ref_kernel", "qkv_prepare_kernel"}
    assert {k: _misses(b) for k, b in found.items()} == dict.fromkeys(found, "")


def test_the_check_itself():
    assert _misses("{ if (x) { report_error(p, 1); return; } ptx::grid_dependency_wait(); }") == "report_error("
    assert _misses("{ if (x) return; ptx::grid_dependency_wait(); }") == "return;"
    assert _misses("{ if (x) { ptx::grid_dependency_wait(); return; } ptx::grid_dependency_wait(); }") == ""
    assert _misses("{ if (x) { ptx::grid_dependency_wait(); return; } f(); }") is None and _misses("{ return; }") is None
    assert _misses("{ if (x) { ptx::grid_dependency_wait(); return; } __ldg(p); ptx::grid_dependency_wait(); }") == "__ldg("
