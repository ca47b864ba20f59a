"""A plan of whole tiles is launched as an ordinary (dependent) kernel on a stream and cooperatively into a graph: the same bits either way,
also behind calls that are still running, and a graph captured then does for a plan that is cut later."""
import importlib

import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def api(pkg):
    return importlib.import_module(pkg.__name__ + ".api")


def _inputs(api, nseq, nblocks, room=0, seed=5):
    g = torch.Generator(device="cuda"); g.manual_seed(seed)
    r = lambda *s: torch.randn(s, generator=g, device="cuda").half()
    caches = torch.zeros((nseq, 4, nblocks + room + 1, 4736), dtype=torch.uint8, device="cuda")
    for i in range(nseq):
        api.kv_commit(r(nblocks + room, 32, 4, 128), r(nblocks + room, 32, 4, 128), caches[i], nblocks + room + 1, 0)
    return caches, r(nseq, 32, 16, 128), r(nseq, 32, 4, 128), r(nseq, 32, 4, 128)


@pytest.mark.parametrize("nseq,nblocks,precise", [(1, 0, False), (1, 4, False), (37, 9, False), (64, 12, True), (64, 12, False), (90, 1, True)])
def test_stream_and_graph_launch_agree(api, nseq, nblocks, precise):
    caches, Q, Kf, Vf = _inputs(api, nseq, nblocks, room=1)
    ctx = api.Context(0)
    plan = ctx.plan([api.Seq(cache=caches[i], nblocks=nblocks, nq=1, q_first=i) for i in range(nseq)])
    assert plan.stats.nitems == 4 * nseq                       # no tile is cut
    def outputs():
        return dict(O16=torch.zeros((32 * nseq, 16, 128), dtype=torch.half, device="cuda"), LSE=torch.zeros((32 * nseq, 16), device="cuda"),
                    q8=torch.zeros((32 * nseq, 2048), dtype=torch.int8, device="cuda"), s8=torch.zeros((32 * nseq, 16), device="cuda"),
                    sum8=torch.zeros((32 * nseq, 16), dtype=torch.int32, device="cuda"))
    a, b, c = outputs(), outputs(), outputs()
    ctx.attention(plan, Q, Kf, Vf, precise=precise, **a)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        ctx.attention(plan, Q, Kf, Vf, precise=precise, **b)
    graph.replay()
    # the query rows and the fresh keys arrive just before the call, and are overwritten just behind it
    Q2, K2, V2 = torch.zeros_like(Q), torch.zeros_like(Kf), torch.zeros_like(Vf)
    for _ in range(5):
        Q2.copy_(Q); K2.copy_(Kf); V2.copy_(Vf)
        ctx.attention(plan, Q2, K2, V2, precise=precise, **c)
        Q2.zero_(); K2.zero_(); V2.zero_()
    assert ctx.device_status() == 0
    for k in a:
        assert torch.equal(a[k], b[k]) and torch.equal(a[k], c[k]), k
    plan.close(); ctx.close()


def test_two_streams_with_whole_tiles(api):
    caches, Q, Kf, Vf = _inputs(api, 60, 20)
    ctxs = [api.Context(0) for _ in range(2)]
    plans = [c.plan([api.Seq(cache=caches[i], nblocks=20, nq=1, q_first=i) for i in range(60)]) for c in ctxs]
    outs = [torch.zeros((60 * 32, 16, 128), dtype=torch.half, device="cuda") for _ in range(2)]
    streams = [torch.cuda.Stream() for _ in range(2)]
    torch.cuda.synchronize()
    for _ in range(20):
        for c, p, o, s in zip(ctxs, plans, outs, streams):
            with torch.cuda.stream(s):
                c.attention(p, Q, Kf, Vf, O16=o)
    torch.cuda.synchronize()
    assert all(c.device_status() == 0 for c in ctxs) and torch.equal(*outs) and bool(torch.isfinite(outs[0].float()).all())
    for x in plans + ctxs:
        x.close()


def test_captured_whole_plan_updated_to_a_cut_one(api):
    caches, Q, Kf, Vf = _inputs(api, 1, 4, room=600)
    ctx = api.Context(0)
    seqs = lambda n: [api.Seq(cache=caches[0], nblocks=n, nq=1, q_first=0)]
    plan = ctx.plan(seqs(4))
    assert plan.stats.nitems == 4
    O = torch.zeros((32, 16, 128), dtype=torch.half, device="cuda")
    ctx.attention(plan, Q, Kf, Vf, O16=O)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        ctx.attention(plan, Q, Kf, Vf, O16=O)
    plan.update(seqs(600))
    assert plan.stats.nitems > 4
    for _ in range(3):
        graph.replay()
    assert ctx.device_status() == 0
    got = O.clone()
    other = ctx.plan(seqs(600))
    ctx.attention(other, Q, Kf, Vf, O16=O)
    assert ctx.device_status() == 0 and torch.equal(got, O)
    for x in (other, plan, ctx):
        x.close()
