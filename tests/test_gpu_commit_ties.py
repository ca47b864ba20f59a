"""The quantiser's codes where (value - minimum) / scale lies on or next to a tie, where the range is empty, and next to
the clamp: there the product with the reciprocal may not stand in for the division. Byte-equal to the oracle."""
import ctypes
import importlib
import os
import shutil
import subprocess

import numpy as np
import pytest

torch = pytest.importorskip("torch")


@pytest.mark.gpu
@pytest.mark.parametrize("seed,step,lo", [(0, 0.5, 0.0), (1, 0.5, -7.5), (2, 0.25, 3.0), (3, 1.5, -100.0), (4, 2.0 ** -14, 0.0), (5, 1000.0, -15000.0)])
def test_codes_on_ties(orc, pkg, seed, step, lo):
    api = importlib.import_module(pkg.__name__ + ".api")
    g = np.random.default_rng(seed)
    nb = 5                                                        # 15 steps of 2 between the extremes: odd multiples of `step` are ties
    k = g.integers(0, 31, (2, nb, 32, 4, 128))
    k[..., 0] = 0; k[..., 1] = 30                                 # V: both extremes in every token
    k[0][:, 0] = 0; k[0][:, 1] = 30                               # K: in every channel
    x = (lo + step * k).astype(np.float16)
    bits = x.view(np.uint16)
    near = g.random(x.shape) < 0.3                                # a third of the values one fp16 step beside the tie
    bits[near & (k > 0) & (k < 30)] += 1
    x[:, nb - 1] = lo                                             # an empty range
    want = np.zeros((4, nb, orc.REC_BYTES), np.uint8)
    orc.kv_commit(x[0], x[1], want, nb, 0)
    cache = torch.zeros((4, nb, orc.REC_BYTES), dtype=torch.uint8, device="cuda")
    api.kv_commit(torch.from_numpy(x[0]).cuda(), torch.from_numpy(x[1]).cuda(), cache, nb, 0)
    torch.cuda.synchronize()
    assert np.array_equal(cache.cpu().numpy(), want)


def _blocks(g, nb):
    """nb blocks, a third each: values on and beside ties, N(0,1) with outlier channels, and one of many scales per block."""
    k = g.integers(0, 31, (2, nb, 32, 4, 128))
    k[..., 0] = 0; k[..., 1] = 30
    k[0][:, 0] = 0; k[0][:, 1] = 30
    step = 2.0 ** g.integers(-12, 8, (1, nb, 1, 1, 1))
    x = ((k - g.integers(0, 31, (1, nb, 1, 1, 1))) * step).astype(np.float16)
    bits = x.view(np.uint16)
    bits[(g.random(x.shape) < 0.2) & (np.abs(x) > 1e-3) & (np.abs(x) < 6e4)] += 1
    n = g.normal(size=x.shape)
    n[0][..., [5, 37, 70, 101]] *= 8
    kind = g.integers(0, 3, nb)
    x[:, kind == 1] = n[:, kind == 1].astype(np.float16)
    x[:, kind == 2] = (n * step)[:, kind == 2].astype(np.float16)
    return x[0], x[1]


@pytest.mark.gpu
@pytest.mark.parametrize("nb", [111, 112, 128, 129, 296, 297, 600])
def test_large_commits_byte_for_byte(orc, pkg, nb):
    """Block counts on both sides of the change of launch shape and of full waves: every record equals the oracle's, contiguous and
    paged, and no byte beside them changes."""
    api = importlib.import_module(pkg.__name__ + ".api")
    g = np.random.default_rng(nb)
    K, V = _blocks(g, nb)
    want = np.full((4, nb + 3, orc.REC_BYTES), 0xAB, np.uint8)
    orc.kv_commit(K, V, want, nb + 3, 2)
    dK, dV = torch.from_numpy(K).cuda(), torch.from_numpy(V).cuda()
    got = torch.full((4, nb + 3, orc.REC_BYTES), 0xAB, dtype=torch.uint8, device="cuda")
    api.kv_commit(dK, dV, got, nb + 3, 2)
    pages = g.permutation(4 * nb + 20)[:4 * nb].astype(np.int32).reshape(nb, 4)
    pool = torch.full((4 * nb + 20, orc.REC_BYTES), 0xCD, dtype=torch.uint8, device="cuda")
    api.kv_commit_paged(dK, dV, pool, torch.from_numpy(pages).cuda())
    torch.cuda.synchronize()
    assert np.array_equal(got.cpu().numpy(), want)
    expect = np.full((4 * nb + 20, orc.REC_BYTES), 0xCD, np.uint8)
    expect[pages.T] = want[:, 2:2 + nb]
    assert np.array_equal(pool.cpu().numpy(), expect)


@pytest.mark.gpu
@pytest.mark.parametrize("nb", [1, 7, 200])
def test_source_shim_commit_byte_for_byte(orc, pkg, tmp_path, nb):
    """attn::kv_commit of the source shim keeps the reference's launch of 128 threads, a split of the same routine that the
    library's own launches do not use."""
    nvcc = os.environ.get("NVCC") or shutil.which("nvcc")
    if nvcc is None:
        pytest.skip("needs nvcc: the shim is source")
    bld = importlib.import_module(pkg.__name__ + ".build")
    lib = _shim_library(nvcc, bld, tmp_path)
    K, V = _blocks(np.random.default_rng(1000 + nb), nb)
    want = np.full((4, nb + 2, orc.REC_BYTES), 0xAB, np.uint8)
    orc.kv_commit(K, V, want, nb + 2, 1)
    dK, dV = torch.from_numpy(K).cuda(), torch.from_numpy(V).cuda()
    got = torch.full((4, nb + 2, orc.REC_BYTES), 0xAB, dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    assert lib.commit(ctypes.c_void_p(dK.data_ptr()), ctypes.c_void_p(dV.data_ptr()), ctypes.c_void_p(got.data_ptr()), nb + 2, 1, nb) == 0
    assert np.array_equal(got.cpu().numpy(), want)


_shim = []


def _shim_library(nvcc, bld, tmp_path):
    if not _shim:
        src, so = tmp_path / "shim_commit.cu", tmp_path / "shim_commit.so"
        src.write_text('#include "attn_shim.cuh"\n'
                       'extern "C" int commit(const void* K, const void* V, void* cache, int max_blocks, int blk, int nb) {\n'
                       '    attn::kv_commit<<<dim3(4, nb), 128>>>((const half*)K, (const half*)V, (uint8_t*)cache, max_blocks, blk);\n'
                       '    return int(cudaDeviceSynchronize());\n}\n')
        subprocess.check_call([nvcc] + bld.NVCC_FLAGS + ["-I", bld.CSRC, str(src), "-o", str(so)])
        _shim.append(ctypes.CDLL(str(so)))
    return _shim[0]
