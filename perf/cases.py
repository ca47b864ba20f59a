"""The work this framework is measured on: block attention over int4 "4c/4" KV and its neighbours on the layer path, through
the public Python binding of the C ABI.

A case is a dict of plain values; `kind` says which part of the path it is:

  step     a denoising step of one layer stack, captured once as a CUDA graph and replayed, as the engine runs it: per layer
           the producer (`qk_norm_rope`), the attention with the int8 activation form as its output, and the output
           projection added into the hidden state
  decode   one layer's attention of a batch of sequences, one 32-token query block each
  prefill  one layer of a prefill pass: producer fused with the block commit, then block-causal attention
  pair     the reference-shaped operator pair (`attn_partial` + `attn_combine`) on caller-owned buffers, split as the
           reference splits
  commit   the block quantiser alone
  produce  the producer alone (a decode step of a batch, where nothing is committed)
  dense    the W4.A8 output projection alone

Inputs follow the distributions that the framework's tests and benchmark use: Q, K, V ~ N(0,1) rounded to fp16 with four
outlier K channels; contexts are made by the commit kernel from a pool of seeded blocks and drawn from it, so every cache has
memory of its own; weights are random 4-bit codes.
"""
import importlib
import math
import random

import torch

api = importlib.import_module("llada2-orin-cuda_b200.api")
wl = importlib.import_module("llada2-orin-cuda_b200.workload")

REC, HID, QKV, GROUPS = 4736, 2048, 3072, 16
EPS = 1e-6
POOL_BLOCKS = 2048


# ---------------------------------------------------------------------------------------------------------------- cases

def listed():
    return [
        # the model's denoising step for one user at an ordinary context: 20 layers in one captured graph
        dict(name="step 1 x 8k", kind="step", nseq=1, blocks=256, layers=20),
        # the smallest call: one short conversation, one layer, called directly
        dict(name="decode 1 x 128", kind="decode", nseq=1, blocks=4, ragged=False, paged=False, out="o16", precise=False),
        # a full serving batch early in its conversations (nothing is long, every sequence is short)
        dict(name="decode 64 x 1k", kind="decode", nseq=64, blocks=32, ragged=False, paged=False, out="o16", precise=False),
        # the headline workload: a full batch at the longest context
        dict(name="decode 64 x 32k", kind="decode", nseq=64, blocks=1024, ragged=False, paged=False, out="o16", precise=False),
        # a large serving batch as it is in earnest: every length from 128 to 32 K tokens, pages anywhere in the pool
        dict(name="decode 256 ragged paged", kind="decode", nseq=256, blocks=1024, ragged=True, paged=True, out="o16", precise=False),
        # evaluation of a model: the precise option, fp32 outputs and log-sum-exps, an odd batch at an odd length
        dict(name="decode 9 x 201 precise", kind="decode", nseq=9, blocks=201, ragged=False, paged=False, out="o32", precise=True),
        # the last prefill pass of a 32 K prompt: 16 blocks behind 31,744 committed tokens
        dict(name="prefill 16 on 31744", kind="prefill", nseq=1, nq=16, blocks=992),
        # the first pass over four short prompts at once: no context yet, an odd number of blocks
        dict(name="prefill 4 x 13 on 0", kind="prefill", nseq=4, nq=13, blocks=0),
        # the engine's own call pair at an ordinary context, split as it asks for
        dict(name="pair 1 x 2k", kind="pair", nq=1, blocks=64),
        # a batch of blocks finished in the same step goes into the page pool
        dict(name="commit 64 paged", kind="commit", nb=64, paged=True),
        # the projection of one query block (the reference's decode shape), and of a full batch's
        dict(name="dense 32", kind="dense", tokens=32),
        dict(name="dense 2048", kind="dense", tokens=2048),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 0.49)))))


def draw(rng: random.Random):
    kind = rng.choice(["step", "decode", "decode", "decode", "prefill", "prefill", "pair", "commit", "produce", "dense"])
    if kind == "step":
        return dict(kind=kind, nseq=_log_int(rng, 1, 4), blocks=_log_int(rng, 4, 1024), layers=20)
    if kind == "decode":
        nseq = _log_int(rng, 1, 256)
        blocks = _log_int(rng, 1, min(1024, 65536 // nseq))
        return dict(kind=kind, nseq=nseq, blocks=blocks, ragged=rng.random() < 0.5, paged=rng.random() < 0.5,
                    out=rng.choice(["o16", "o16", "o32"]), precise=rng.random() < 0.2)
    if kind == "prefill":
        return dict(kind=kind, nseq=_log_int(rng, 1, 4), nq=rng.randint(1, 16), blocks=rng.choice([0, _log_int(rng, 1, 992), _log_int(rng, 1, 992)]))
    if kind == "pair":
        return dict(kind=kind, nq=_log_int(rng, 1, 16), blocks=_log_int(rng, 1, 512))
    if kind == "commit":
        return dict(kind=kind, nb=_log_int(rng, 1, 2048), paged=rng.random() < 0.5)
    if kind == "produce":
        return dict(kind=kind, tokens=_log_int(rng, 32, 8192))
    return dict(kind=kind, tokens=_log_int(rng, 1, 4096))


# --------------------------------------------------------------------------------------------------------------- inputs

def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _keys(g, shape):
    K = torch.randn(shape, generator=g, device="cuda")
    K[..., list(wl.OUTLIER_CHANNELS)] *= wl.OUTLIER_GAIN
    return K.half()


def _values(g, shape):
    return torch.randn(shape, generator=g, device="cuda").half()


def _record_pool(g, blocks):
    """Records of seeded blocks, [4][n][4736]."""
    n = max(1, min(POOL_BLOCKS, blocks))
    pool = torch.zeros((4, n, REC), dtype=torch.uint8, device="cuda")
    api.kv_commit(_keys(g, (n, 32, 4, 128)), _values(g, (n, 32, 4, 128)), pool, n, 0)
    return pool


def _contexts(g, lengths, room, layers=1):
    """Caches [layer][sequence][4][max + room][4736] of committed blocks drawn from a pool, one tensor."""
    longest = max(lengths) + room
    pool = _record_pool(g, max(lengths) * len(lengths))
    caches = torch.zeros((layers, len(lengths), 4, max(longest, 1), REC), dtype=torch.uint8, device="cuda")
    for layer in range(layers):
        for i, n in enumerate(lengths):
            if n:
                idx = torch.randint(0, pool.shape[1], (n,), generator=g, device="cuda")
                for h in range(4):
                    torch.index_select(pool[h], 0, idx, out=caches[layer, i, h, :n])
    return caches


def _lengths(case, seed):
    if not case.get("ragged"):
        return [case["blocks"]] * case["nseq"]
    rng = random.Random(seed)
    return [rng.randint(min(4, case["blocks"]), case["blocks"]) for _ in range(case["nseq"])]


def _producer_inputs(g, tokens, first_pos, layers=1):
    return dict(
        qkv=torch.randn((layers, tokens, QKV), generator=g, device="cuda"),
        pos=(torch.arange(tokens, device="cuda", dtype=torch.int32) + first_pos).contiguous(),
        gq=1.0 + 0.1 * torch.randn((128,), generator=g, device="cuda"),
        gk=1.0 + 0.1 * torch.randn((128,), generator=g, device="cuda"),
        freq=torch.from_numpy(api.inv_freq()).cuda(),
        q=torch.zeros((tokens, 16, 128), dtype=torch.half, device="cuda"),
        k=torch.zeros((tokens, 4, 128), dtype=torch.half, device="cuda"),
        v=torch.zeros((tokens, 4, 128), dtype=torch.half, device="cuda"))


def _weight_strips(g, layers=1):
    """[layers][128 strips][16 code tiles of 1024 bytes, then 16 metas of 48]: random codes, scales around 0.01, zero points 5..10."""
    strips = torch.randint(0, 256, (layers, HID // 16, GROUPS * 1072), generator=g, device="cuda", dtype=torch.uint8)
    meta = strips[:, :, GROUPS * 1024:].view(layers, HID // 16, GROUPS, 48)
    scale = (0.01 * torch.exp(0.5 * torch.randn((layers, HID // 16, GROUPS, 16), generator=g, device="cuda"))).half()
    meta[..., :32] = scale.view(torch.uint8)
    meta[..., 32:] = torch.randint(5, 11, meta[..., 32:].shape, generator=g, device="cuda", dtype=torch.uint8)
    return strips


def _activations(g, tokens):
    q = torch.randint(-127, 128, (tokens, HID), generator=g, device="cuda", dtype=torch.int8)
    s = 0.02 * torch.exp(0.5 * torch.randn((tokens, GROUPS), generator=g, device="cuda"))
    return q, s, q.view(tokens, GROUPS, 128).sum(2, dtype=torch.int32)


def prepare(case, seed):
    g = _gen(seed)
    st = dict(case=dict(case))
    kind = case["kind"]
    if kind == "step":
        nseq, n, layers = case["nseq"], case["blocks"], case["layers"]
        caches = _contexts(g, [n] * nseq, 1, layers)
        st.update(_producer_inputs(g, 32 * nseq, 0, layers))
        st["pos"] = (torch.arange(32 * nseq, device="cuda", dtype=torch.int32) % 32 + 32 * n).contiguous()
        st.update(caches=caches, W=_weight_strips(g, layers), Y=torch.randn((32 * nseq, HID), generator=g, device="cuda"),
                  q8=torch.zeros((32 * nseq, HID), dtype=torch.int8, device="cuda"),
                  s8=torch.zeros((32 * nseq, GROUPS), device="cuda"),
                  sum8=torch.zeros((32 * nseq, GROUPS), dtype=torch.int32, device="cuda"))
        st["ctx"] = ctx = api.Context(torch.cuda.current_device())
        st["plan"] = plan = ctx.plan([api.Seq(cache=caches[0, i], nblocks=n, nq=1, q_first=i) for i in range(nseq)])
        layer_bytes = caches[0].numel()

        def layers_of_a_step():
            for i in range(layers):
                api.qk_norm_rope(st["qkv"][i], st["pos"], st["gq"], st["gk"], EPS, st["freq"], st["q"], st["k"], st["v"])
                ctx.attention(plan, st["q"], st["k"], st["v"], q8=st["q8"], s8=st["s8"], sum8=st["sum8"], cache_offset=i * layer_bytes)
                api.dense_w4a8(st["W"][i], st["q8"], st["s8"], st["sum8"], st["Y"])

        y0 = st["Y"].clone()
        side = torch.cuda.Stream()
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            layers_of_a_step()
        torch.cuda.current_stream().wait_stream(side)
        st["graph"] = torch.cuda.CUDAGraph()
        with torch.cuda.graph(st["graph"]):
            layers_of_a_step()
        st["Y"].copy_(y0)
    elif kind == "decode":
        lengths = _lengths(case, seed)
        nseq = len(lengths)
        if case["paged"]:
            total = sum(lengths)
            src = _record_pool(g, total).view(-1, REC)
            pool = torch.empty((total * 4, REC), dtype=torch.uint8, device="cuda")
            torch.index_select(src, 0, torch.randint(0, src.shape[0], (total * 4,), generator=g, device="cuda"), out=pool)
            pages = torch.randperm(total, generator=g, device="cuda").to(torch.int32)
            seqs, tables, at = [], [], 0
            for i, n in enumerate(lengths):
                p = pages[at:at + n]
                tables.append((p[None, :] * 4 + torch.arange(4, device="cuda", dtype=torch.int32)[:, None]).contiguous())
                seqs.append(api.Seq(cache=pool, nblocks=n, nq=1, q_first=i, pages=tables[-1]))
                at += n
            st.update(pool=pool, tables=tables)
        else:
            caches = _contexts(g, lengths, 1)[0]
            seqs = [api.Seq(cache=caches[i], nblocks=n, nq=1, q_first=i) for i, n in enumerate(lengths)]
            st["caches"] = caches
        st.update(Q=_values(g, (nseq, 32, 16, 128)), Kf=_keys(g, (nseq, 32, 4, 128)), Vf=_values(g, (nseq, 32, 4, 128)))
        st["out"] = {"O16": torch.zeros((nseq * 32, 16, 128), dtype=torch.half, device="cuda")} if case["out"] == "o16" else \
                    {"O32": torch.zeros((nseq * 32, 16, 128), device="cuda"), "LSE": torch.zeros((nseq * 32, 16), device="cuda")}
        st["ctx"] = api.Context(torch.cuda.current_device())
        st["plan"] = st["ctx"].plan(seqs)
    elif kind == "prefill":
        nseq, nq, n = case["nseq"], case["nq"], case["blocks"]
        st["caches"] = caches = _contexts(g, [n] * nseq, nq)[0]
        st.update(_producer_inputs(g, 32 * nq * nseq, 0))
        st["pos"] = (torch.arange(32 * nq * nseq, device="cuda", dtype=torch.int32) % (32 * nq) + 32 * n).contiguous()
        # block j of the pass, head h -> record of its sequence's cache: the sequences' caches are one pool
        maxb = n + nq
        rec = (torch.arange(nseq, device="cuda")[:, None, None] * 4 + torch.arange(4, device="cuda")[None, None, :]) * maxb \
            + n + torch.arange(nq, device="cuda")[None, :, None]
        st["new_pages"] = rec.to(torch.int32).reshape(nseq * nq, 4).contiguous()
        st["O16"] = torch.zeros((32 * nq * nseq, 16, 128), dtype=torch.half, device="cuda")
        st["ctx"] = api.Context(torch.cuda.current_device())
        st["plan"] = st["ctx"].plan([api.Seq(cache=caches[i], nblocks=n, nq=nq, q_first=i * nq) for i in range(nseq)])
    elif kind == "pair":
        nq, n = case["nq"], case["blocks"]
        st["cache"] = _contexts(g, [n + nq - 1], 1)[0, 0]
        bpc = api.pick_bpc(n, nq)
        nch = api.chunks_for(n + nq - 1, bpc)
        st.update(bpc=bpc, nch=nch, O16=torch.zeros((32 * nq, 16, 128), dtype=torch.half, device="cuda"))
        st["args"] = api.Args(
            Q=_values(g, (nq, 32, 16, 128)), Kf=_keys(g, (nq, 32, 4, 128)), Vf=_values(g, (nq, 32, 4, 128)), cache=st["cache"],
            max_blocks=n + nq, nblocks=n, blocks_per_chunk=bpc, nchunks=nch, scale=api.SCALE,
            Opart=torch.zeros((nq, 4, nch, 128, 128), device="cuda"), Mpart=torch.zeros((nq, 4, nch, 128), device="cuda"),
            Lpart=torch.zeros((nq, 4, nch, 128), device="cuda"))
    elif kind == "commit":
        nb = case["nb"]
        st.update(K=_keys(g, (nb, 32, 4, 128)), V=_values(g, (nb, 32, 4, 128)), cache=torch.zeros((4, nb, REC), dtype=torch.uint8, device="cuda"))
        if case["paged"]:
            st["pages"] = torch.randperm(4 * nb, generator=g, device="cuda").to(torch.int32).reshape(nb, 4)
    elif kind == "produce":
        st.update(_producer_inputs(g, case["tokens"], 0))
        st["pos"] = torch.randint(0, 32768, (case["tokens"],), generator=g, device="cuda", dtype=torch.int32)
    else:
        q, s, qsum = _activations(g, case["tokens"])
        st.update(W=_weight_strips(g)[0], q=q, s=s, qsum=qsum, Y=torch.randn((case["tokens"], HID), generator=g, device="cuda"))
    torch.cuda.synchronize()
    return st


# ----------------------------------------------------------------------------------------------------------------- pass

def run(st):
    kind = st["case"]["kind"]
    if kind == "step":
        st["graph"].replay()
        return {"hidden": st["Y"], "k": st["k"], "v": st["v"]}
    if kind == "decode":
        st["ctx"].attention(st["plan"], st["Q"], st["Kf"], st["Vf"], precise=st["case"]["precise"], **st["out"])
        return st["out"]
    if kind == "prefill":
        api.qkv_prepare_commit(st["qkv"][0], st["pos"], st["gq"], st["gk"], EPS, st["freq"], st["q"], st["k"], st["v"], st["caches"],
                               pages=st["new_pages"])
        st["ctx"].attention(st["plan"], st["q"], st["k"], st["v"], O16=st["O16"])
        return {"q": st["q"], "k": st["k"], "v": st["v"], "cache": st["caches"], "o": st["O16"]}
    if kind == "pair":
        a = st["args"]
        nq = st["case"]["nq"]
        api.attn_partial(a, nq)
        api.attn_combine(a.Opart, a.Mpart, a.Lpart, st["nch"], a.nblocks, st["bpc"], O=st["O16"], nb=nq)
        return st["O16"]
    if kind == "commit":
        if st["case"]["paged"]:
            api.kv_commit_paged(st["K"], st["V"], st["cache"], st["pages"])
        else:
            api.kv_commit(st["K"], st["V"], st["cache"], st["cache"].shape[1], 0)
        return st["cache"]
    if kind == "produce":
        api.qk_norm_rope(st["qkv"][0], st["pos"], st["gq"], st["gk"], EPS, st["freq"], st["q"], st["k"], st["v"])
        return {"q": st["q"], "k": st["k"], "v": st["v"]}
    api.dense_w4a8(st["W"], st["q"], st["s"], st["qsum"], st["Y"])
    return st["Y"]


# ----------------------------------------------------------------------------------------------------- work and tolerance

def _attention_work(blocks, nq, records_once, out_bytes_per_token):
    """One sequence's attention: every record read once, Q and the fresh K/V read, the output written."""
    tokens = 32 * nq
    flops = sum(4 * 32 * 2048 * 32 * (blocks + j + 1) for j in range(nq))
    return records_once * 4 * REC + tokens * (4096 + 2048 + out_bytes_per_token), flops


def work(case):
    kind = case["kind"]
    dense_bytes = lambda tokens: HID // 16 * GROUPS * 1072 + tokens * (HID + 8 * GROUPS + 8 * HID)
    producer_bytes = lambda tokens: tokens * (4 * QKV + 2 * QKV)
    if kind == "step":
        n, nseq, layers = case["blocks"], case["nseq"], case["layers"]
        b, f = _attention_work(n, 1, n, 2048 + 128)
        tokens = 32 * nseq
        # the hidden state is read and written once in the step, the projections' weights once per layer
        return {"bytes": layers * (nseq * b + producer_bytes(tokens) + HID // 16 * GROUPS * 1072 + tokens * (HID + 8 * GROUPS)) + 8 * HID * tokens,
                "flops": layers * (nseq * f + 2 * tokens * HID * HID)}
    if kind == "decode":
        lengths = [case["blocks"]] * case["nseq"]
        if case["ragged"]:                      # lengths are uniform between the shortest and the longest
            lengths = [(min(4, case["blocks"]) + case["blocks"]) / 2] * case["nseq"]
        parts = [_attention_work(n, 1, n, 4096 if case["out"] == "o16" else 8192 + 64) for n in lengths]
        return {"bytes": sum(p[0] for p in parts), "flops": sum(p[1] for p in parts)}
    if kind == "prefill":
        n, nq, nseq = case["blocks"], case["nq"], case["nseq"]
        b, f = _attention_work(n, nq, n, 4096)      # the new blocks' records are written by the pass (below); what it re-reads is its own
        return {"bytes": nseq * (b + producer_bytes(32 * nq) + nq * 4 * REC), "flops": nseq * f}
    if kind == "pair":
        b, f = _attention_work(case["blocks"], case["nq"], case["blocks"] + case["nq"] - 1, 4096)
        return {"bytes": b, "flops": f}
    if kind == "commit":
        return {"bytes": case["nb"] * 4 * (16384 + REC), "flops": 0}
    if kind == "produce":
        return {"bytes": producer_bytes(case["tokens"]), "flops": 0}
    return {"bytes": dense_bytes(case["tokens"]), "flops": 2 * case["tokens"] * HID * HID}


def tolerance(case):
    kind = case["kind"]
    if kind in ("commit", "produce", "dense"):
        return "exact"                       # the framework's contract: the reference's bytes and bits
    if kind == "step":
        # an attention difference moves about one int8 code in a hundred by one step; the projections carry it into the hidden
        # state: rel 1.0e-3, worst element 4.6e-3 between two cuts of the same contexts
        return {"rel": 5e-3, "max": 4e-2}
    if kind == "decode" and case["precise"]:
        # value + remainder probabilities: rel 1e-6 .. 3.4e-5, worst element 1.6e-3 (the tensor core's fp32 sums over long runs)
        return {"rel": 1.4e-4, "max": 5e-3}
    # fp16 probabilities and outputs: rel 3.2e-4, worst element 5.0e-3 between two cuts of the same contexts
    return {"rel": 1.2e-3, "max": 2e-2}
