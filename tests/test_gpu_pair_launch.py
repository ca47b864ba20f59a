"""The operator pair's folding launch is a programmatic dependent one: it may be on the chip before the launch ahead of it has
ended. Bit for bit the results of calls that are waited for one by one: back to back on the same partial buffers, inside a
captured graph, behind something that is no kernel, as the first node, and behind another stream's work."""
import importlib

import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def setup(pkg):
    api = importlib.import_module(pkg.__name__ + ".api")
    g = torch.Generator(device="cuda")
    g.manual_seed(5)
    half = lambda *s: torch.randn(s, generator=g, device="cuda").half()
    nblocks, nq, n = 41, 3, 6
    bpc = api.pick_bpc(nblocks, nq)
    nch = api.chunks_for(nblocks + nq - 1, bpc)
    cache = torch.zeros((4, nblocks + nq, 4736), dtype=torch.uint8, device="cuda")
    api.kv_commit(half(nblocks + nq, 32, 4, 128), half(nblocks + nq, 32, 4, 128), cache, nblocks + nq, 0)
    f32 = lambda *s: torch.zeros(s, device="cuda")
    calls = [api.Args(Q=half(nq, 32, 16, 128), Kf=half(nq, 32, 4, 128), Vf=half(nq, 32, 4, 128), cache=cache, max_blocks=nblocks + nq, nblocks=nblocks,
                      blocks_per_chunk=bpc, nchunks=nch, scale=api.SCALE, Opart=None, Mpart=None, Lpart=None) for _ in range(n)]
    part = f32(nq, 4, nch, 128, 128), f32(nq, 4, nch, 128), f32(nq, 4, nch, 128)
    for a in calls:
        a.Opart, a.Mpart, a.Lpart = part                     # all calls share the buffers
    outs = [torch.zeros((32 * nq, 16, 128), dtype=torch.half, device="cuda") for _ in range(n)]

    def partial(i):
        api.attn_partial(calls[i], nq)

    def combine(i):
        api.attn_combine(*part, nch, nblocks, bpc, O=outs[i], nb=nq)

    want = []
    for i in range(n):
        partial(i); torch.cuda.synchronize()
        combine(i); torch.cuda.synchronize()
        want.append(outs[i].clone())
        outs[i].zero_()
    torch.cuda.synchronize()
    assert all(float(w.float().abs().max()) > 0.01 for w in want) and not torch.equal(want[0], want[1])
    return api, n, partial, combine, outs, want, part


def _check(outs, want):
    torch.cuda.synchronize()
    for o, w in zip(outs, want):
        assert torch.equal(o, w)
        o.zero_()


def test_back_to_back_on_the_same_buffers(setup):
    api, n, partial, combine, outs, want, part = setup
    for _ in range(20):
        for i in range(n):
            partial(i); combine(i)
        _check(outs, want)


def test_captured_and_replayed(setup):
    api, n, partial, combine, outs, want, part = setup
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        for i in range(n):
            partial(i); combine(i)
    for _ in range(5):
        graph.replay()
        graph.replay()
        _check(outs, want)


def test_behind_copies_first_in_a_graph_and_behind_another_stream(setup):
    api, n, partial, combine, outs, want, part = setup
    saved = []
    for i in range(2):
        partial(i)
        saved.append([p.clone() for p in part])
    torch.cuda.synchronize()
    # nothing ahead of it; then a copy ahead of it
    graph = torch.cuda.CUDAGraph()
    for p, s in zip(part, saved[0]):
        p.copy_(s)
    torch.cuda.synchronize()
    with torch.cuda.graph(graph):
        combine(0)
        for p, s in zip(part, saved[1]):
            p.copy_(s)
        combine(1)
    graph.replay()
    _check(outs[:2], want[:2])
    # another stream's launch, joined by an event, directly and captured
    side = torch.cuda.Stream()

    def forked():
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            partial(2)
        torch.cuda.current_stream().wait_stream(side)
        combine(2)
        partial(3)
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            combine(3)
        torch.cuda.current_stream().wait_stream(side)

    for _ in range(10):
        forked()
        _check(outs[2:4], want[2:4])
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        forked()
    for _ in range(3):
        graph.replay()
        _check(outs[2:4], want[2:4])


@pytest.mark.parametrize("nchunks,nb,bpc", [(1, 3, 9), (4, 2, 3), (15, 2, 2), (16, 3, 1), (17, 3, 1), (18, 5, 2), (33, 2, 1), (64, 1, 1), (160, 1, 1)])
def test_folding_launch_against_fp64(pkg, orc, nchunks, nb, bpc):
    """Random partial results of 1 .. 160 chunks (up to 16 in the short form, more in the long one; the first query blocks may have
    a chunk less than the last): the fold in fp64. fp32 weights and sums: 2^-23 each for weight, product and sum and 2^-22 for
    exp2f, times the largest |term| sum over |result|, below 1e-5 of a row's RMS here; the fp16 form adds half an ulp."""
    api = importlib.import_module(pkg.__name__ + ".api")
    g = torch.Generator(device="cuda")
    g.manual_seed(nchunks)
    nblocks = bpc * nchunks - (nb - 1)                          # visible to block j: nblocks + j, the last has all chunks
    O = torch.randn((nb, 4, nchunks, 128, 128), generator=g, device="cuda")
    M = 6 * torch.randn((nb, 4, nchunks, 128), generator=g, device="cuda")
    L = torch.rand((nb, 4, nchunks, 128), generator=g, device="cuda") + 0.5
    live = [max(1, -(-(nblocks + j) // bpc)) for j in range(nb)]
    want = torch.empty((nb, 32, 16, 128), dtype=torch.float64, device="cuda")
    for j in range(nb):
        o, m, l = (x[j, :, :live[j]].double() for x in (O, M, L))
        w = torch.exp2(m - m.max(1, keepdim=True).values)
        r = (w[..., None] * o).sum(1) / (w * l).sum(1)[..., None]                   # [4][128 rows][128], row = 4 token + head
        want[j] = r.view(4, 32, 4, 128).permute(1, 0, 2, 3).reshape(32, 16, 128)
    for j in range(nb):
        O[j, :, live[j]:] = float("nan")                        # slots past a block's own are not read into anything
    got = torch.zeros((32 * nb, 16, 128), dtype=torch.half, device="cuda")
    api.attn_combine(O, M, L, nchunks, nblocks, bpc, O=got, nb=nb)
    rms = want.pow(2).mean(-1, keepdim=True).sqrt()
    err = (got.view(nb, 32, 16, 128).double() - want).abs()
    assert bool((err <= 1e-5 * rms + want.abs() * 2.0 ** -11 + 2.0 ** -25).all())
    q8 = torch.zeros((32 * nb, 2048), dtype=torch.int8, device="cuda")
    s8, sum8 = torch.zeros((32 * nb, 16), device="cuda"), torch.zeros((32 * nb, 16), dtype=torch.int32, device="cuda")
    api.attn_combine(O, M, L, nchunks, nblocks, bpc, q8=q8, s8=s8, sum8=sum8, nb=nb)
    wq, ws, wsum = (torch.from_numpy(x).cuda() for x in orc.act_q8(want.view(32 * nb, 16, 128).float().cpu().numpy()))
    assert bool(((s8 - ws.view_as(s8)).abs() <= 2e-5 * ws.view_as(s8)).all())
    assert int((q8.int() - wq.view_as(q8).int()).abs().max()) <= 1 and float((q8 != wq.view_as(q8)).float().mean()) < 1e-3
    assert torch.equal(sum8, q8.view(32 * nb, 16, 128).sum(2, dtype=torch.int32))
