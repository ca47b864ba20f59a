"""The library built with other values of its compile-time options gives the default build's numbers. Compiled here:
LLATTN_NRAW=8: a ring of eight records in flight instead of ten in the attention kernel (its slots and phases then fall differently on the tiles);
LLATTN_DW_LAUNCH_REGS=96: the projection's tcgen05 kernels, built with 80 registers a thread, have fewer than their roles are to divide."""
import importlib
import importlib.util
import os
import re
import shutil
import subprocess
import sys

import numpy as np
import pytest

torch = pytest.importorskip("torch")
OPTIONS = {"LLATTN_NRAW": 8, "LLATTN_DW_LAUNCH_REGS": 96}


def test_the_options_exist(pkg):
    """A define that no source reads would test the default build against itself."""
    bld = importlib.import_module(pkg.__name__ + ".build")
    text = "".join(open(f).read() for f in bld.sources())
    for name, value in OPTIONS.items():
        default = re.search(rf"#ifndef {name}\n#define {name} (\d+)\n", text)
        assert default and int(default.group(1)) != value and len(re.findall(rf"\b{name}\b", text)) > 2, name


@pytest.fixture(scope="module")
def other(pkg, tmp_path_factory):
    nvcc = os.environ.get("NVCC") or shutil.which("nvcc")
    if nvcc is None:
        pytest.skip("needs nvcc: the options are compile-time ones")
    bld = importlib.import_module(pkg.__name__ + ".build")
    lib = str(tmp_path_factory.mktemp("other") / "libllattn_other.so")
    subprocess.check_call([nvcc] + bld.NVCC_FLAGS + [f"-D{k}={v}" for k, v in OPTIONS.items()] + [os.path.join(bld.CSRC, "llattn.cu"), "-o", lib])
    old = os.environ.get("LLATTN_LIB")
    os.environ["LLATTN_LIB"] = lib                             # read when the module is loaded
    try:
        spec = importlib.util.spec_from_file_location("llattn_api_other", os.path.join(bld.HERE, "api.py"))
        api = sys.modules[spec.name] = importlib.util.module_from_spec(spec)
        spec.loader.exec_module(api)
    finally:
        os.environ.pop("LLATTN_LIB")
        if old is not None:
            os.environ["LLATTN_LIB"] = old
    assert api.lib()._name == lib
    return api


@pytest.mark.gpu
@pytest.mark.parametrize("nblocks,nctas", [(0, 0), (3, 4), (5, 8), (33, 3), (130, 0)])
@pytest.mark.parametrize("precise", [False, True])
def test_other_build_matches_the_oracle(other, pkg, orc, nblocks, nctas, precise):
    wl = pkg.workload
    Q, Kf, Vf = wl.query_blocks(1, seq=nblocks)
    cache = np.zeros((4, nblocks + 1, orc.REC_BYTES), np.uint8)
    if nblocks:
        Kc, Vc = wl.context_blocks(nblocks, seq=nblocks)
        orc.kv_commit(Kc, Vc, cache, nblocks + 1, 0)
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    want, lse = orc.attention(Q, Kf, Vf, cache, nblocks + 1, nblocks, dq_mode=1)
    ctx = other.Context(0)
    cached = dev(cache)
    plan = ctx.plan([other.Seq(cache=cached, nblocks=nblocks)], nctas)
    O, L = torch.zeros((32, 16, 128), device="cuda"), torch.zeros((32, 16), device="cuda")
    ctx.attention(plan, dev(Q), dev(Kf), dev(Vf), O32=O, LSE=L, precise=precise)
    assert ctx.device_status() == 0
    rms = np.sqrt((want.astype(np.float64) ** 2).mean())
    # the bounds of the default build's tests: 2e-3 up to 8 blocks and with precise, 5e-3 above (fp16 rounding of P); LSE 1e-3
    assert np.abs(O.cpu().numpy() - want).max() <= (2e-3 if precise or nblocks <= 8 else 5e-3) * rms
    assert np.abs(L.cpu().numpy() - lse).max() <= 1e-3
    plan.close(); ctx.close()


# The sizes of the tcgen05 form; without the registers for it the mma.sync tiles take the call, same bits.
@pytest.mark.gpu
@pytest.mark.parametrize("ntokens", [160, 577])
def test_too_few_registers_for_the_split(other, pkg, orc, ntokens):
    wl = pkg.workload
    strips, _, _, _ = wl.dense_weights(2048, 2048, 81)
    q, s, qsum = wl.int8_activations(ntokens, 2048, 82)
    assert other.dense_preview(2048, 2048, ntokens, 148)[0] == other.DENSE_TCGEN05
    want = np.random.default_rng(83).normal(size=(ntokens, 2048)).astype(np.float32)
    Y = torch.from_numpy(want.copy()).cuda()
    orc.dense_w4a8(strips, q, s, qsum, want)
    other.dense_w4a8(*(torch.from_numpy(np.ascontiguousarray(x)).cuda() for x in (strips, q, s, qsum)), Y)
    assert other.dense_status() == 0 and np.array_equal(Y.cpu().numpy().view(np.uint32), want.view(np.uint32))
