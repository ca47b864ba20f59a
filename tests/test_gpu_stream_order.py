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


# The calls above reach the device about as fast as it runs them, so a launch seldom finds the kernel ahead of it still running. Here all of
# them are in the queue before the first starts: behind a delay on the stream, checked, or as a captured graph.
def _behind_a_delay(enqueue):
    torch.cuda.synchronize()
    torch.cuda._sleep(40_000_000)                  # 20 ms and more
    passed = torch.cuda.Event()
    passed.record()
    enqueue()
    assert not passed.query(), "the device was at work before the last call was in its queue"
    torch.cuda.synchronize()


def _captured(enqueue):
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        enqueue()
    graph.replay()
    torch.cuda.synchronize()


def _compare(state, run):
    """run(state, between) enqueues the calls and returns the tensors to compare; state() makes new buffers."""
    st = state()
    want = run(st, torch.cuda.synchronize)
    torch.cuda.synchronize()
    for how in (_behind_a_delay, _captured):
        st, got = state(), []
        how(lambda: got.extend(run(st, lambda: None)))
        for a, b in zip(want, got):
            assert torch.equal(a, b) and bool(torch.isfinite(a.float()).all())


# Layers of a batch: producer and commit in one, attention over what was just committed (a plan of whole tiles: an ordinary launch on the
# stream, a cooperative one in the graph), the projection on tcgen05 (one tile a CTA, and several) into the next layer's producer.
@pytest.mark.parametrize("nb,few", [(6, True), (40, False)])
def test_queued_layers(api, pkg, nb, few):
    wl, T, ctxb = pkg.workload, 32 * nb, 3
    kernel, tok = api.dense_preview(3072, 2048, T, torch.cuda.get_device_properties(0).multi_processor_count)
    assert kernel == api.DENSE_TCGEN05 and (24 * -(-T // tok) <= 148) == few
    g = torch.Generator(device="cuda"); g.manual_seed(21)
    W = torch.from_numpy(wl.dense_weights(3072, 2048, 22)[0]).cuda()
    pos, gain, freq = torch.arange(T, device="cuda", dtype=torch.int32), torch.ones(128, device="cuda"), torch.from_numpy(api.inv_freq()).cuda()
    qkv0 = torch.randn((T, 3072), generator=g, device="cuda")
    caches0 = torch.zeros((nb, 4, ctxb + 1, 4736), dtype=torch.uint8, device="cuda")
    for i in range(nb):
        api.kv_commit(torch.randn((ctxb, 32, 4, 128), generator=g, device="cuda").half(), torch.randn((ctxb, 32, 4, 128), generator=g, device="cuda").half(), caches0[i], ctxb + 1, 0)
    # block i of the batch becomes the last record of sequence i
    pages = ((torch.arange(nb, device="cuda")[:, None] * 4 + torch.arange(4, device="cuda")) * (ctxb + 1) + ctxb).to(torch.int32).contiguous()
    ctx = api.Context(0)
    plans = []

    def state():
        caches = caches0.clone()
        plans.append(ctx.plan([api.Seq(cache=caches[i], nblocks=ctxb + 1, nq=1, q_first=i) for i in range(nb)]))
        assert plans[-1].stats.nitems == 4 * nb
        return dict(qkv=qkv0.clone(), caches=caches, plan=plans[-1], q=torch.zeros((T, 16, 128), dtype=torch.half, device="cuda"),
                    k=torch.zeros((T, 4, 128), dtype=torch.half, device="cuda"), v=torch.zeros((T, 4, 128), dtype=torch.half, device="cuda"),
                    q8=torch.zeros((T, 2048), dtype=torch.int8, device="cuda"), s8=torch.zeros((T, 16), device="cuda"), sum8=torch.zeros((T, 16), dtype=torch.int32, device="cuda"))

    def run(st, between):
        q, k, v = st["q"].view(nb, 32, 16, 128), st["k"].view(nb, 32, 4, 128), st["v"].view(nb, 32, 4, 128)
        for _ in range(6):
            api.qkv_prepare_commit(st["qkv"], pos, gain, gain, 1e-6, freq, st["q"], st["k"], st["v"], st["caches"], pages=pages); between()
            ctx.attention(st["plan"], q, k, v, q8=st["q8"], s8=st["s8"], sum8=st["sum8"]); between()
            api.dense_w4a8(W, st["q8"], st["s8"], st["sum8"], st["qkv"]); between()
        return st["qkv"], st["caches"], st["q"], st["q8"]

    _compare(state, run)
    assert ctx.device_status() == 0 and api.dense_status() == 0
    for x in plans + [ctx]:
        x.close()


# The reference-grid attention lets its successor onto the chip early, whatever that is: another one of it, the commit over records that it
# reads, the folding launch, the producer over its query rows.
@pytest.mark.parametrize("nq,nblocks", [(1, 6), (2, 40), (3, 9)])
def test_queued_behind_the_reference_grid(api, nq, nblocks):
    T, maxb = 32 * nq, nblocks + nq
    g = torch.Generator(device="cuda"); g.manual_seed(31)
    rand = lambda *s: torch.randn(s, generator=g, device="cuda")
    zero = lambda *s: torch.zeros(s, dtype=torch.half, device="cuda")
    K, V, qkv0 = rand(nblocks, 32, 4, 128).half(), rand(nblocks, 32, 4, 128).half(), rand(T, 3072)
    pos, gain, freq = torch.arange(T, device="cuda", dtype=torch.int32), torch.ones(128, device="cuda"), torch.from_numpy(api.inv_freq()).cuda()
    bpc = api.pick_bpc(nblocks + nq - 1, nq)
    nch = api.chunks_for(nblocks + nq - 1, bpc)

    def state():
        cache = torch.zeros((4, maxb, 4736), dtype=torch.uint8, device="cuda")
        api.kv_commit(K, V, cache, maxb, 0)
        st = dict(qkv=qkv0.clone(), cache=cache, q=zero(nq, 32, 16, 128), k=zero(nq, 32, 4, 128), v=zero(nq, 32, 4, 128),
                  O=[zero(T, 16, 128) for _ in range(3)])
        st["args"] = [api.Args(Q=st["q"], Kf=st["k"], Vf=st["v"], cache=cache, max_blocks=maxb, nblocks=nblocks, blocks_per_chunk=bpc, nchunks=nch, scale=api.SCALE,
                               Opart=torch.zeros((nq, 4, nch, 128, 128), device="cuda"), Mpart=torch.zeros((nq, 4, nch, 128), device="cuda"),
                               Lpart=torch.zeros((nq, 4, nch, 128), device="cuda")) for _ in range(2)]
        return st

    def run(st, between):
        a, b = st["args"]
        fold = lambda x, o: api.attn_combine(x.Opart, x.Mpart, x.Lpart, nch, nblocks, bpc, O=o, nb=nq)
        for i in range(6):
            api.qk_norm_rope(st["qkv"], pos, gain, gain, 1e-6, freq, st["q"].view(T, 16, 128), st["k"].view(T, 4, 128), st["v"].view(T, 4, 128)); between()
            api.attn_partial(a, nq); between()
            api.kv_commit(V if i % 2 == 0 else K, K if i % 2 == 0 else V, st["cache"], maxb, 0); between()      # over the records just read
            api.attn_partial(b, nq); between()
            fold(a, st["O"][0]); between()
            api.attn_partial(a, nq); between()                                      # over the partial results just folded
            api.attn_partial(b, nq); between()
            fold(a, st["O"][1]); between()
            fold(b, st["O"][2]); between()
            st["qkv"][:, :2048] = 0.5 * st["qkv"][:, :2048] + (st["O"][0] + st["O"][1] - st["O"][2]).view(T, 2048); between()
        return [st["qkv"], st["cache"], *st["O"], b.Opart, b.Mpart, b.Lpart]

    _compare(state, run)
