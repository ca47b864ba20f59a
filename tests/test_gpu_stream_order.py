"""Calls one after the other on a stream, without waiting in between, give what the same calls give one at a time: a launch that starts
before the kernel ahead of it is done waits before it reads or writes anything. Every call's inputs are the outputs of the one before, and
buffers are written again while their readers may still be running."""
import importlib

import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def api(pkg):
    return importlib.import_module(pkg.__name__ + ".api")


@pytest.mark.parametrize("nq,nblocks,own_stream", [(1, 5, False), (2, 40, True), (4, 9, False)])
def test_back_to_back_calls(api, pkg, nq, nblocks, own_stream):
    wl, T = pkg.workload, 32 * nq
    g = torch.Generator(device="cuda"); g.manual_seed(11)
    strips, _, _, _ = wl.dense_weights(2048, 2048, 12)
    W = torch.from_numpy(strips).cuda()
    pos = torch.arange(T, device="cuda", dtype=torch.int32) + 32 * nblocks
    gain, freq = torch.ones(128, device="cuda"), torch.from_numpy(api.inv_freq()).cuda()
    qkv0 = torch.randn((T, 3072), generator=g, device="cuda")
    cache0 = torch.zeros((4, nblocks + 2 * nq, 4736), dtype=torch.uint8, device="cuda")
    api.kv_commit(torch.randn((nblocks, 32, 4, 128), generator=g, device="cuda").half(), torch.randn((nblocks, 32, 4, 128), generator=g, device="cuda").half(),
                  cache0, nblocks + 2 * nq, 0)
    bpc = api.pick_bpc(nblocks + nq - 1, nq)
    nch = api.chunks_for(nblocks + nq - 1, bpc)

    def chain(between):
        qkv, cache = qkv0.clone(), cache0.clone()
        q, k, v = (torch.zeros((T, n, 128), dtype=torch.half, device="cuda") for n in (16, 4, 4))
        Y, q8 = torch.zeros((T, 2048), device="cuda"), torch.zeros((T, 2048), dtype=torch.int8, device="cuda")
        s8, sum8 = torch.zeros((T, 16), device="cuda"), torch.zeros((T, 16), dtype=torch.int32, device="cuda")
        args = api.Args(Q=q.view(nq, 32, 16, 128), Kf=k.view(nq, 32, 4, 128), Vf=v.view(nq, 32, 4, 128), cache=cache, max_blocks=nblocks + 2 * nq, nblocks=nblocks,
                        blocks_per_chunk=bpc, nchunks=nch, scale=api.SCALE, Opart=torch.zeros((nq, 4, nch, 128, 128), device="cuda"),
                        Mpart=torch.zeros((nq, 4, nch, 128), device="cuda"), Lpart=torch.zeros((nq, 4, nch, 128), device="cuda"))
        torch.cuda.synchronize()
        for _ in range(12):
            api.qk_norm_rope(qkv, pos, gain, gain, 1e-6, freq, q, k, v); between()
            api.kv_commit(k.view(nq, 32, 4, 128), v.view(nq, 32, 4, 128), cache, nblocks + 2 * nq, nblocks); between()
            api.attn_partial(args, nq); between()
            api.attn_combine(args.Opart, args.Mpart, args.Lpart, nch, nblocks, bpc, q8=q8, s8=s8, sum8=sum8, nb=nq); between()
            api.dense_w4a8(W, q8, s8, sum8, Y); between()
            qkv[:, :2048] = 0.5 * qkv[:, :2048] + Y; between()
        torch.cuda.synchronize()
        return qkv, cache, q, Y, q8

    want = chain(torch.cuda.synchronize)
    with torch.cuda.stream(torch.cuda.Stream() if own_stream else torch.cuda.current_stream()):
        got = chain(lambda: None)
    for a, b in zip(want, got):
        assert torch.equal(a, b) and bool(torch.isfinite(a.float()).all())
