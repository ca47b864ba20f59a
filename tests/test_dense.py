"""Dense W4.A8 projection that consumes the attention output (llattn_dense_w4a8): oracle on CPU, kernel on the GPU.

Integer group products are exact and every float operation is the reference's, in its order (one product of the two
scales, one fused multiply-add per 128-group, one add into Y): the GPU tests ask for identical bits against the CPU
oracle and against the reference's own moe8::gemm compiled for sm_100a (when it travelled)."""
import importlib

import numpy as np
import pytest


def test_oracle_against_float64_restatement(orc, pkg):
    """The C oracle (tile and fragment layouts of engine/moe_i8.cu:55-60,127-160) against a numpy restatement that
    takes the weights in logical order and the activations out of fragment order."""
    wl = pkg.workload
    rows, K, nt = 256, 384, 7
    strips, codes, scale, zero = wl.dense_weights(rows, K, 1)
    q, s, qsum = wl.int8_activations(nt, K, 2)
    Y0 = np.random.default_rng(3).normal(size=(nt, rows)).astype(np.float32)
    Y = Y0.copy()
    orc.dense_w4a8(strips, q, s, qsum, Y)
    fp = np.array([orc.frag_pos(c) for c in range(128)])
    ql = q.reshape(nt, K // 128, 128)[:, :, fp].astype(np.int64)
    P = np.einsum("rgk,ngk->nrg", codes.reshape(rows, K // 128, 128).astype(np.int64), ql)
    v = P - zero.astype(np.int64)[None] * qsum[:, None, :]
    ref = Y0 + (scale.astype(np.float64)[None] * s[:, None, :] * v).sum(axis=2)
    assert np.abs(Y - ref).max() <= 2e-6 * np.abs(ref).max()


def test_meta_layout(pkg):
    """Scale pairs (rows g | g + 8) at 4 g and zero pairs at 32 + 2 g of every 48-byte meta (engine/moe_i8.cu:38-40)."""
    strips, codes, scale, zero = pkg.workload.dense_weights(32, 256, 5)
    ktot = 2
    for sidx in range(2):
        for kt in range(ktot):
            meta = strips[sidx, ktot * 1024 + kt * 48: ktot * 1024 + (kt + 1) * 48]
            for g in range(8):
                pair = meta[4 * g:4 * g + 4].view(np.uint16)
                assert pair[0] == scale[16 * sidx + g, kt].view(np.uint16) and pair[1] == scale[16 * sidx + g + 8, kt].view(np.uint16)
                assert meta[32 + 2 * g] == zero[16 * sidx + g, kt] and meta[33 + 2 * g] == zero[16 * sidx + g + 8, kt]


torch = pytest.importorskip("torch")


@pytest.fixture(scope="module")
def api(pkg):
    m = importlib.import_module(pkg.__name__ + ".api")
    m.lib()
    return m


def _dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


@pytest.mark.gpu
@pytest.mark.parametrize("ntokens,rows,K", [(32, 2048, 2048), (64, 2048, 2048), (100, 256, 512), (1, 128, 128), (192, 2048, 2048)])
def test_dense_bit_exact_vs_oracle(api, orc, pkg, ntokens, rows, K):
    wl = pkg.workload
    strips, _, _, _ = wl.dense_weights(rows, K, 11)
    q, s, qsum = wl.int8_activations(ntokens, K, 12)
    Y0 = np.random.default_rng(13).normal(size=(ntokens, rows)).astype(np.float32)
    want = Y0.copy()
    orc.dense_w4a8(strips, q, s, qsum, want)
    Y = _dev(Y0)
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    api.dense_w4a8(_dev(strips), _dev(q), _dev(s), _dev(qsum), Y, err_word=err)
    torch.cuda.synchronize()
    assert int(err.item()) == 0
    got = Y.cpu().numpy()
    assert np.array_equal(got.view(np.uint32), want.view(np.uint32)), float(np.abs(got - want).max())


@pytest.mark.gpu
@pytest.mark.parametrize("ntokens,rows,K,odd", [
    (7, 128, 128, False), (8, 256, 2176, False), (31, 128, 2048, True), (33, 128, 4224, False), (63, 384, 256, False),   # a strip's tokens, one group, more groups than warps
    (65, 128, 128, False), (97, 128, 4224, True), (127, 256, 384, True), (129, 128, 2176, False), (257, 2048, 256, False),
    (1000, 384, 512, True), (2500, 1024, 128, False),
    (66, 2048, 512, True), (128, 2048, 128, False), (143, 2048, 2176, True), (144, 2048, 256, False), (145, 2048, 128, False), (288, 2048, 256, True), (290, 2048, 128, False)])     # where the tile size changes
def test_dense_tile_edges(api, orc, pkg, ntokens, rows, K, odd):
    """Token counts around the tile sizes of both kernels, one to more groups than pipeline stages or warps. `odd`: zero
    points over the whole byte and sums that are not the sums of the codes, which the formula allows."""
    wl = pkg.workload
    strips, _, _, zero = wl.dense_weights(rows, K, 41)
    q, s, qsum = wl.int8_activations(ntokens, K, 42)
    rng = np.random.default_rng(43)
    if odd:
        ktot = K // 128
        meta = strips.reshape(rows // 16, -1)[:, ktot * 1024:].reshape(rows // 16, ktot, 48)
        meta[..., 32:] = rng.integers(0, 256, meta[..., 32:].shape)
        qsum = qsum.copy()
        qsum[rng.random(qsum.shape) < 0.1] += 77
        q = q.copy()
        q[0, :5] = -128
    Y0 = rng.normal(size=(ntokens, rows)).astype(np.float32)
    want = Y0.copy()
    orc.dense_w4a8(strips, q, s, qsum, want)
    pad = torch.full((ntokens + 2, rows), 7.0, device="cuda")          # rows before and after Y must not change
    pad[1:-1] = _dev(Y0)
    api.dense_w4a8(_dev(strips), _dev(q), _dev(s), _dev(qsum), pad[1:-1])
    torch.cuda.synchronize()
    got = pad.cpu().numpy()
    assert (got[0] == 7).all() and (got[-1] == 7).all()
    assert np.array_equal(got[1:-1].view(np.uint32), want.view(np.uint32)), float(np.abs(got[1:-1] - want).max())


@pytest.mark.gpu
@pytest.mark.parametrize("ntokens,rows,K", [
    (1, 128, 128), (32, 128, 128), (64, 2048, 128), (1, 4096, 512), (32, 4096, 512), (33, 3072, 2048), (64, 3072, 2048), (24, 6144, 2048), (33, 8192, 256),
    (16, 12288, 256), (24, 12288, 256), (48, 12288, 256), (1, 16384, 512), (64, 16384, 512), (20, 32768, 256), (64, 32768, 256)])
def test_dense_few_tokens_many_rows(api, orc, pkg, ntokens, rows, K):
    """Few tokens on both sides of the line between the strip kernel and the tiles, and between the tile sizes: the same bits."""
    wl = pkg.workload
    strips, _, _, _ = wl.dense_weights(rows, K, 51)
    q, s, qsum = wl.int8_activations(ntokens, K, 52)
    want = np.random.default_rng(53).normal(size=(ntokens, rows)).astype(np.float32)
    Y = _dev(want.copy())
    orc.dense_w4a8(strips, q, s, qsum, want)
    api.dense_w4a8(_dev(strips), _dev(q), _dev(s), _dev(qsum), Y)
    assert np.array_equal(Y.cpu().numpy().view(np.uint32), want.view(np.uint32))


@pytest.mark.gpu
@pytest.mark.parametrize("rows,K", [(2048, 2048), (8192, 512), (16384, 512), (16384, 2048)])
def test_dense_few_tokens_cost_no_more_than_many(api, rows, K):
    """64 tokens take no longer than 96 of the same weights, whatever the rows, and 32 not longer than 64 (1.25 leaves room for
    timing; choosing the kernel by the tokens alone, 64 tokens took 1.8 .. 2.7 times as long as 96 at 8192 and 16,384 rows)."""
    ktot = K // 128
    W = torch.randint(0, 256, (rows // 16, ktot * 1072), device="cuda", dtype=torch.uint8)
    W[:, ktot * 1024:] = 0x11

    def us(n):
        q = torch.randint(-127, 128, (n, K), device="cuda", dtype=torch.int8)
        s, qsum = torch.rand((n, ktot), device="cuda"), q.view(n, ktot, 128).sum(2, dtype=torch.int32)
        Y = torch.zeros((n, rows), device="cuda")
        api.dense_w4a8(W, q, s, qsum, Y)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            for _ in range(20):
                api.dense_w4a8(W, q, s, qsum, Y)
        best = float("inf")
        for _ in range(6):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record(); graph.replay(); b.record(); b.synchronize()
            best = min(best, a.elapsed_time(b) * 1000 / 20)
        return best

    t32, t64, t96 = us(32), us(64), us(96)
    assert t64 <= 1.25 * t96 and t32 <= 1.25 * t64, (t32, t64, t96)


@pytest.mark.gpu
def test_dense_bit_exact_vs_reference_kernel(api, pkg):
    import refkernel
    if not refkernel.gemm_available():
        pytest.skip("reference GEMM library did not travel")
    wl = pkg.workload
    ntokens, rows, K = 96, 2048, 2048
    strips, _, _, _ = wl.dense_weights(rows, K, 21)
    q, s, qsum = wl.int8_activations(ntokens, K, 22)
    Y0 = np.random.default_rng(23).normal(size=(ntokens, rows)).astype(np.float32)
    dW, dq, ds, dsum = _dev(strips), _dev(q), _dev(s), _dev(qsum)
    Yr, Yn = _dev(Y0), _dev(Y0)
    refkernel.dense_w4a8(dW, dq, ds, dsum, Yr)
    api.dense_w4a8(dW, dq, ds, dsum, Yn)
    torch.cuda.synchronize()
    a, b = Yr.cpu().numpy(), Yn.cpu().numpy()
    assert np.array_equal(a.view(np.uint32), b.view(np.uint32)), float(np.abs(a - b).max())


@pytest.mark.gpu
def test_dense_consumes_the_attention_epilogue(api, orc, pkg):
    """Attention -> int8 Act (merge kernel) -> projection, against the oracle chain on the kernel's own fp32 output."""
    wl = pkg.workload
    Kc, Vc = wl.context_blocks(6, seq=400)
    Q, Kf, Vf = wl.query_blocks(1, seq=400)
    cache = np.zeros((4, 7, orc.REC_BYTES), np.uint8)
    orc.kv_commit(Kc, Vc, cache, 7, 0)
    ctx = api.Context(0)
    dc = _dev(cache)
    plan = ctx.plan([api.Seq(cache=dc, nblocks=6, nq=1, q_first=0)])
    q8 = torch.zeros((32, 2048), dtype=torch.int8, device="cuda")
    s8 = torch.zeros((32, 16), dtype=torch.float32, device="cuda")
    sum8 = torch.zeros((32, 16), dtype=torch.int32, device="cuda")
    ctx.attention(plan, _dev(Q), _dev(Kf), _dev(Vf), q8=q8, s8=s8, sum8=sum8)
    assert ctx.device_status() == 0
    strips, _, _, _ = wl.dense_weights(2048, 2048, 31)
    h0 = np.random.default_rng(32).normal(size=(32, 2048)).astype(np.float32)
    h = _dev(h0)
    api.dense_w4a8(_dev(strips), q8, s8, sum8, h)
    torch.cuda.synchronize()
    want = h0.copy()
    orc.dense_w4a8(strips, q8.cpu().numpy(), s8.cpu().numpy(), sum8.cpu().numpy(), want)
    assert np.array_equal(h.cpu().numpy().view(np.uint32), want.view(np.uint32))
    plan.close(); ctx.close()


@pytest.mark.gpu
def test_dense_argument_errors(api):
    t = torch.zeros(16, dtype=torch.uint8, device="cuda")
    with pytest.raises(api.LlattnError) as e:
        api.lib().llattn_dense_w4a8  # symbol exists
        api._check(api.lib().llattn_dense_w4a8(t.data_ptr(), t.data_ptr(), t.data_ptr(), t.data_ptr(), t.data_ptr(), 32, 100, 128, None, None))
    assert e.value.code == api.EINVAL


# A call without an error word of its own still has a place where an expired wait is read. (The codes come from the wait
# self-test, which no projection takes part in: nothing here fails.)
@pytest.mark.gpu
def test_dense_reports_without_an_error_word(api, orc, pkg):
    assert api.dense_status() == 0
    waited = torch.zeros(6, dtype=torch.int64, device="cuda")
    api._check(api.lib().llattn_wait_selftest(1_000_000, api.dense_error_word(), waited.data_ptr(), None))
    torch.cuda.synchronize()
    with pytest.raises(api.LlattnError) as e:
        api.dense_status()
    assert e.value.code == api.EDEVICE and "0x8f" in str(e.value)                    # every role's code
    assert api.dense_status() == 0                                                   # read once, cleared
    wl, n = pkg.workload, 300
    strips, _, _, _ = wl.dense_weights(2048, 2048, 61)
    q, s, qsum = wl.int8_activations(n, 2048, 62)
    want = np.zeros((n, 2048), np.float32)
    orc.dense_w4a8(strips, q, s, qsum, want)
    Y = torch.zeros((n, 2048), device="cuda")
    api.dense_w4a8(_dev(strips), _dev(q), _dev(s), _dev(qsum), Y)
    assert api.dense_status() == 0 and np.array_equal(Y.cpu().numpy().view(np.uint32), want.view(np.uint32))


def test_dense_status_argument_errors(api):
    assert api.lib().llattn_dense_status(None, None) == api.EINVAL
    assert api.lib().llattn_dense_error_word(None) == api.EINVAL


# Where the tcgen05 form takes over: 32, 64 and 128 tokens a CTA, each with a ragged last tile of few tokens and of all but one,
# one and several waves, the fewest groups it takes, an odd number of groups (a stage of one), and more groups than factors held at a time (16)
TCGEN05_CASES = [
    (149, 2048, 2048, 32), (160, 2048, 2176, 32), (289, 2048, 2048, 64), (321, 2048, 2176, 64), (577, 2048, 2048, 128), (641, 2048, 1152, 128),
    (1153, 2048, 2048, 128), (1217, 2048, 4096, 64), (2049, 1024, 4224, 128), (65, 8192, 2048, 64), (200, 8192, 4224, 128), (127, 4096, 2048, 32), (255, 4096, 2176, 64),
    (577, 2048, 768, 128), (511, 2048, 1280, 64), (1151, 2048, 768, 128)]


@pytest.mark.parametrize("ntokens,rows,K,tok", TCGEN05_CASES)
def test_dense_tcgen05_cases_take_that_form(api, ntokens, rows, K, tok):
    assert api.dense_preview(rows, K, ntokens, 148) == (api.DENSE_TCGEN05, tok)


def test_dense_preview(api):
    assert api.dense_preview(2048, 2048, 32, 148)[0] == api.DENSE_STRIPS
    assert api.dense_preview(2048, 128, 2560, 148) == (api.DENSE_TILES, 64)
    # many waves of six groups: the tiles (87.3 and 97.7 us; with a CTA per tile the tcgen05 form took 94.5 and 104.7, walking them it takes 74.6 and 86.5)
    assert api.dense_preview(16384, 768, 1184, 148) == api.dense_preview(12288, 768, 1800, 148) == (api.DENSE_TILES, 64)
    assert {t for *_, t in TCGEN05_CASES} == {32, 64, 128}
    for bad in ((100, 128, 1, 148), (128, 128, 0, 148), (128, 128, 1, 0)):
        with pytest.raises(api.LlattnError):
            api.dense_preview(*bad)


@pytest.mark.gpu
@pytest.mark.parametrize("ntokens,rows,K,tok", TCGEN05_CASES)
def test_dense_tcgen05_form(api, orc, pkg, ntokens, rows, K, tok):
    if torch.cuda.get_device_properties(0).multi_processor_count == 148:
        assert api.dense_preview(rows, K, ntokens, 148) == (api.DENSE_TCGEN05, tok)
    wl = pkg.workload
    strips, _, _, _ = wl.dense_weights(rows, K, 41)
    strips = strips.copy()
    strips[:, K // 128 * 1024:].reshape(-1, K // 128, 48)[:, ::3, 32:] = 255          # zero points up to the largest
    q, s, qsum = wl.int8_activations(ntokens, K, 42)
    q, qsum = q.copy(), qsum.copy()
    q.reshape(ntokens, -1, 128)[::5, ::2] = -127                                     # and sums down to the smallest
    qsum.reshape(ntokens, -1)[::5, ::2] = -127 * 128
    Y0 = np.random.default_rng(43).normal(size=(ntokens, rows)).astype(np.float32)
    want = Y0.copy()
    orc.dense_w4a8(strips, q, s, qsum, want)
    pad = torch.full((ntokens + 2 * tok, rows), 7.0, device="cuda")                  # a CTA's tokens before and after Y must not change
    pad[tok:-tok] = _dev(Y0)
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    api.dense_w4a8(_dev(strips), _dev(q), _dev(s), _dev(qsum), pad[tok:-tok], err_word=err)
    assert int(err.item()) == 0
    got = pad.cpu().numpy()
    assert (got[:tok] == 7).all() and (got[-tok:] == 7).all()
    assert np.array_equal(got[tok:-tok].view(np.uint32), want.view(np.uint32))


# A CTA of the tcgen05 form walks several tiles: two and three of them, an odd number of groups (the rings and accumulators are then out of
# step with the tile), more groups than factors held at a time, and a ragged last tile of tokens; with 32 tokens a CTA, few groups are what
# makes more tiles than SMs the choice.
@pytest.mark.gpu
@pytest.mark.parametrize("ntokens,rows,K,tok", [(1280, 4096, 1152, 128), (2050, 2048, 1152, 128), (300, 16384, 1152, 128), (1217, 2048, 4224, 64),
                                                   (657, 1792, 768, 32), (913, 1280, 640, 32), (81, 12544, 640, 32)])
def test_dense_tcgen05_several_tiles_per_cta(api, orc, pkg, ntokens, rows, K, tok):
    if torch.cuda.get_device_properties(0).multi_processor_count == 148:
        assert api.dense_preview(rows, K, ntokens, 148) == (api.DENSE_TCGEN05, tok) and rows // 128 * -(-ntokens // tok) > 148
    wl = pkg.workload
    strips, _, _, _ = wl.dense_weights(rows, K, 71)
    q, s, qsum = wl.int8_activations(ntokens, K, 72)
    want = np.random.default_rng(73).normal(size=(ntokens, rows)).astype(np.float32)
    Y, err = _dev(want), torch.zeros(1, dtype=torch.int32, device="cuda")
    orc.dense_w4a8(strips, q, s, qsum, want)
    api.dense_w4a8(_dev(strips), _dev(q), _dev(s), _dev(qsum), Y, err_word=err)
    assert int(err.item()) == 0 and np.array_equal(Y.cpu().numpy().view(np.uint32), want.view(np.uint32))
