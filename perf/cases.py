"""Performance cases: what a serving host has this library do, over the range of sizes it meets.

Families (``kind`` of a case):

* ``step``      one decode layer-step of one layer (append -> select -> attend) through ``DsaDecodeLayer.step``
* ``stack``     one token through a stack of full and shared layers that share a page table (``DsaDecodeStack``)
* ``prompt``    a prompt's tokens quantised into the paged pools (``DsaDecodeLayer.append``)
* ``proj``      the projections around the cache path of one layer (``IndexerFrontEnd``, ``KvbProjection``)
* ``operators`` one token of one sequence through the single-sequence f32 operators a host binds one by one
* ``v4``        one decode token of the block-compressed variant (``V4TokenStep``)
* ``v4_prompt`` a prompt through that variant's two KV compressors

Everything is made on the GPU from the seed. Sequence lengths of a batch are spread evenly over [lo, hi] and
dealt to the sequences in an order that the seed decides, so that the work of a case does not depend on the seed.
"""
from __future__ import annotations

import math
import random

import torch

from rivoli_b200 import backend as be
from rivoli_b200.engine import DsaDecodeStack, indexer_layout
from rivoli_b200.layer import DsaDecodeLayer, IndexerFrontEnd, KvbProjection
from rivoli_b200.v4 import V4Compressor, V4DecodeLayer, V4TokenStep

DEV = "cuda:0"
KV_LORA, ROPE = 512, 64
WIDTH = KV_LORA + ROPE
NOPE, V_HEAD, HIDDEN, Q_LORA, BLOCK = 192, 256, 6144, 2048, 128      # the projections of the 64-head model
THETA, EPS = 10000.0, 1e-6
LAYOUT = ("full", "shared", "shared", "full")
CHUNK = 1 << 16                                                      # tokens appended per call while a cache is filled

MODEL = dict(heads=64, index_heads=32, index_dim=128, page=64)
SMALL = dict(heads=16, index_heads=8, index_dim=64, page=16)


def step(batch, lo, hi, top_k=2048, geom=MODEL):
    return dict(kind="step", batch=batch, lo=lo, hi=hi, top_k=top_k, **geom)


def stack(batch, lo, hi, top_k=2048):
    return dict(kind="stack", batch=batch, lo=lo, hi=hi, top_k=top_k, **MODEL)


def listed():
    return [
        # the smallest call: one short sequence of a 16-head layer with 16-token pages
        dict(step(1, 257, 257, 64, SMALL), name="step-1x257-small"),
        # one interactive user of the 64-head model
        dict(step(1, 4099, 4099), name="step-1x4099"),
        # short contexts: every token is attended (top-k = context)
        dict(step(32, 2048, 2048), name="step-32x2048"),
        # one GPU's slice of a continuously batched server: ragged contexts, four layers of which two own an indexer
        dict(stack(32, 512, 32768), name="stack-32xragged"),
        # a full batch of long contexts, the configuration the decode step is quoted on
        dict(step(128, 16384, 16384), name="step-128x16384"),
        # a few very long contexts
        dict(step(4, 131072, 131072), name="step-4x131072"),
        # prompts written to the cache
        dict(kind="prompt", batch=5, tokens=65537, name="prompt-65537"),
        # what runs before and after the cache path in every layer, at the full batch
        dict(kind="proj", batch=128, name="proj-128"),
        # one sequence through the operators that take one token each
        dict(kind="operators", tokens=8193, top_k=2048, name="operators-8193"),
        # the block-compressed variant, a full batch
        dict(kind="v4", batch=128, ctx=8192, name="v4-128x8192"),
        # and a nearly idle server
        dict(kind="v4", batch=3, ctx=3001, name="v4-3x3001"),
        # its prompts
        dict(kind="v4_prompt", tokens=16381, name="v4-prompt-16381"),
    ]


def _log(rng: random.Random, lo: int, hi: int) -> int:
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng: random.Random) -> dict:
    kind = rng.choice(("step", "step", "step", "step", "small", "stack", "prompt", "proj", "operators", "v4", "v4", "v4_prompt"))
    if kind == "step":
        batch = _log(rng, 1, 128)
        hi = _log(rng, 64, min(131072, 128 * 16384 // batch))
        lo = hi if rng.random() < 0.5 else _log(rng, max(1, hi // 16), hi)
        return step(batch, lo, hi, rng.choice((2048, 2048, 512, 256)))
    if kind == "small":
        hi = _log(rng, 32, 4096)
        return step(rng.randint(1, 8), _log(rng, max(1, hi // 4), hi), hi, rng.choice((64, 128, 256)), SMALL)
    if kind == "stack":
        hi = _log(rng, 1024, 32768)
        return stack(_log(rng, 2, 32), rng.randint(min(512, hi // 4), hi // 2), hi)
    if kind == "prompt":
        return dict(kind="prompt", batch=rng.randint(1, 8), tokens=_log(rng, 16, 65536))
    if kind == "proj":
        return dict(kind="proj", batch=_log(rng, 1, 128))
    if kind == "operators":
        return dict(kind="operators", tokens=_log(rng, 64, 8192), top_k=rng.choice((2048, 512)))
    if kind == "v4":
        return dict(kind="v4", batch=_log(rng, 1, 128), ctx=_log(rng, 256, 8192))
    return dict(kind="v4_prompt", tokens=_log(rng, 64, 16380))


# --- inputs -----------------------------------------------------------------------------------------------------
class _Rand:
    def __init__(self, seed):
        self.host = random.Random(seed)
        self.gen = torch.Generator(device=DEV)
        self.gen.manual_seed(seed)

    def f32(self, *shape, scale=1.0, shift=0.0):
        t = torch.randn(shape, generator=self.gen, device=DEV)
        return t.mul_(scale).add_(shift) if scale != 1.0 or shift != 0.0 else t

    def bf16(self, *shape):
        return torch.randn(shape, generator=self.gen, device=DEV, dtype=torch.bfloat16)

    def weights(self, rows, cols):
        """A block-scaled fp8 matrix: e4m3 codes and one positive scale per 128 x 128 block."""
        codes = self.f32(rows, cols, scale=0.7).to(torch.float8_e4m3fn).view(torch.uint8)
        scale = self.f32(-(-rows // BLOCK) * -(-cols // BLOCK)).abs_().mul_(0.01).add_(0.002)
        return codes, scale


def lengths(case, rnd=None):
    b, lo, hi = case["batch"], case["lo"], case["hi"]
    n = [lo + (hi - lo) * i // max(1, b - 1) for i in range(b)] if b > 1 else [hi]
    if rnd is not None:
        rnd.host.shuffle(n)
    return n


def _i32(v):
    return torch.tensor(v, dtype=torch.int32, device=DEV)


def _geom(case, lens):
    page = case["page"]
    pages = [-(-n // page) for n in lens]
    return be.DsaGeom.make(n_heads=case["heads"], kv_lora=KV_LORA, rope_dim=ROPE, index_heads=case["index_heads"],
                           index_dim=case["index_dim"], page_tokens=page, top_k=case["top_k"],
                           max_pages_per_seq=max(pages), n_pool_pages=max(sum(pages), math.ceil(1.25 * sum(pages))))


def _fill(layers, rnd, lens):
    """All tokens but each sequence's last, through the append operator, the same positions in every layer."""
    n = torch.tensor([k - 1 for k in lens], device=DEV)
    total = int(n.sum())
    if not total:
        return
    seq = torch.repeat_interleave(torch.arange(len(lens), device=DEV), n)
    pos = torch.arange(total, device=DEV) - (torch.cumsum(n, 0) - n)[seq]
    seq, pos = seq.to(torch.int32), pos.to(torch.int32)
    for layer in layers:
        for at in range(0, total, CHUNK):
            k = min(CHUNK, total - at)
            layer.append(rnd.bf16(k, WIDTH), rnd.bf16(k, layer.g.index_dim), pos[at:at + k], seq[at:at + k])


def _step_inputs(case, rnd):
    b = case["batch"]
    return (rnd.bf16(b, WIDTH), rnd.bf16(b, case["index_dim"]), rnd.bf16(b, case["index_heads"], case["index_dim"]),
            rnd.bf16(b, case["index_heads"]).float(), rnd.bf16(b, case["heads"], WIDTH))


def _prepare_step(case, rnd):
    lens = lengths(case, rnd)
    layer = DsaDecodeLayer(_geom(case, lens), case["batch"], device=DEV, max_ctx=max(lens), shuffle_seed=rnd.host.getrandbits(31))
    for b, n in enumerate(lens):
        layer.reserve(b, n)
    layer.upload_block_table()
    _fill([layer], rnd, lens)
    return dict(layer=layer, x=_step_inputs(case, rnd), pos=_i32([n - 1 for n in lens]), len=_i32(lens),
                hint=min(min(lens), case["top_k"]))       # what the scheduler knows about the batch


def _run_step(s):
    L = s["layer"]
    out = L.step(*s["x"], s["pos"], s["len"], min_rows_hint=s["hint"])
    return dict(out=out, lse=L.out_lse, rows=L.rows, n_sel=L.n_sel, latent=L.latent_pool, latent_scale=L.latent_scale,
                key=L.index_pool, key_scale=L.index_scale)


def _prepare_stack(case, rnd):
    lens = lengths(case, rnd)
    full = indexer_layout(LAYOUT, len(LAYOUT), case["index_heads"], case["index_dim"], case["top_k"])
    st = DsaDecodeStack(_geom(case, lens), case["batch"], full, device=DEV, max_ctx=max(lens), shuffle_seed=rnd.host.getrandbits(31))
    for b, n in enumerate(lens):
        st.pool.reserve(b, n)
    st.upload_block_table()
    _fill(st.layers, rnd, lens)
    return dict(stack=st, x=[_step_inputs(case, rnd) for _ in full], pos=_i32([n - 1 for n in lens]), len=_i32(lens),
                hint=min(min(lens), case["top_k"]))


def _run_stack(s):
    st, res = s["stack"], []
    for i, x in enumerate(s["x"]):
        L = st.layers[i]
        out = st.step_layer(i, *x, s["pos"], s["len"], min_rows_hint=s["hint"])
        res.append(dict(out=out, lse=L.out_lse, latent=L.latent_pool, latent_scale=L.latent_scale))
        if st.full[i]:
            res[-1].update(rows=L.rows, n_sel=L.n_sel, key=L.index_pool, key_scale=L.index_scale)
    return res


def _prompt_lengths(case):
    b, t = case["batch"], case["tokens"]
    return [t * (i + 1) // b - t * i // b for i in range(b)]


def _prepare_prompt(case, rnd):
    lens = [max(1, n) for n in _prompt_lengths(case)]
    layer = DsaDecodeLayer(_geom(dict(MODEL, top_k=2048), lens), len(lens), device=DEV, max_ctx=max(lens),
                           shuffle_seed=rnd.host.getrandbits(31))
    for b, n in enumerate(lens):
        layer.reserve(b, n)
    layer.upload_block_table()
    n = torch.tensor(_prompt_lengths(case), device=DEV)
    seq = torch.repeat_interleave(torch.arange(len(lens), device=DEV), n)
    pos = torch.arange(case["tokens"], device=DEV) - (torch.cumsum(n, 0) - n)[seq]
    return dict(layer=layer, latent=rnd.bf16(case["tokens"], WIDTH), key=rnd.bf16(case["tokens"], MODEL["index_dim"]),
                seq=seq.to(torch.int32), pos=pos.to(torch.int32))


def _run_prompt(s):
    L = s["layer"]
    L.append(s["latent"], s["key"], s["pos"], s["seq"])
    return dict(latent=L.latent_pool, latent_scale=L.latent_scale, key=L.index_pool, key_scale=L.index_scale)


def _front_weights(rnd):
    nh, hd = MODEL["index_heads"], MODEL["index_dim"]
    w = {}
    for name, rows, cols in (("wk", hd, HIDDEN), ("wq_b", nh * hd, Q_LORA), ("wproj", nh, HIDDEN)):
        w[name], w[name + "_scale"] = rnd.weights(rows, cols)
    w["knorm_w"], w["knorm_b"] = rnd.f32(hd, scale=0.1, shift=1.0), rnd.f32(hd, scale=0.05)
    return w


def _prepare_proj(case, rnd):
    b, H = case["batch"], MODEL["heads"]
    fg = be.IndexFrontGeom(HIDDEN, Q_LORA, MODEL["index_heads"], MODEL["index_dim"], 0, ROPE, BLOCK, EPS, THETA)
    g = be.DsaGeom.make(max_pages_per_seq=1, n_pool_pages=1)
    kvb, scale = rnd.weights(H * (NOPE + V_HEAD), KV_LORA)
    return dict(front=IndexerFrontEnd(fg, b, _front_weights(rnd), device=DEV), kvb=KvbProjection(g, b, kvb, scale, NOPE, V_HEAD, BLOCK),
                x=rnd.bf16(b, HIDDEN), q_resid=rnd.bf16(b, Q_LORA), pos=_i32([rnd.host.randrange(100000) for _ in range(b)]),
                q=rnd.bf16(b, H, NOPE + ROPE), latent=rnd.bf16(b, H, KV_LORA))


def _run_proj(s):
    key, iq, iw = s["front"].run(s["x"], s["q_resid"], s["pos"])
    return dict(key=key, index_q=iq, index_w=iw, q_abs=s["kvb"].absorb(s["q"]), ctx=s["kvb"].value(s["latent"]))


def _prepare_operators(case, rnd):
    nt, H, nh, hd = case["tokens"], MODEL["heads"], MODEL["index_heads"], MODEL["index_dim"]
    kvb, kvb_scale = rnd.weights(H * (NOPE + V_HEAD), KV_LORA)
    f = lambda n: torch.zeros(n, device=DEV)
    return dict(
        nt=nt, k=case["top_k"], w=_front_weights(rnd), kvb=kvb, kvb_scale=kvb_scale,
        x=rnd.f32(HIDDEN), q_resid=rnd.f32(Q_LORA), q=rnd.f32(H * (NOPE + ROPE)), latent=rnd.f32(KV_LORA), rope=rnd.f32(ROPE),
        lc8=rnd.f32(nt, KV_LORA).to(torch.float8_e4m3fn).view(torch.uint8),
        lscale=rnd.f32(nt, KV_LORA // BLOCK, scale=0.1).abs_().add_(0.01), rc=rnd.bf16(nt, ROPE), keys=rnd.bf16(nt, hd),
        key=f(hd), key_n=f(hd), iq=f(nh * hd), iw=f(nh), qabs=f(H * KV_LORA), qrope=f(H * ROPE), scores=f(nt),
        rows=torch.zeros(min(case["top_k"], nt), dtype=torch.int32, device=DEV), clat=f(H * KV_LORA), ctx=f(H * V_HEAD),
        partial=f(be.attend_scratch_floats(H, KV_LORA)))


def _run_operators(s):
    nt, k, w, H = s["nt"], s["k"], s["w"], MODEL["heads"]
    nh, hd, nb, pos = MODEL["index_heads"], MODEL["index_dim"], KV_LORA // BLOCK, s["nt"] - 1
    # indexer key, queries and head weights
    be.launch_gemv_fp8(s["x"], w["wk"], w["wk_scale"], hd, HIDDEN, BLOCK, 1, s["key"])
    be.launch_layernorm(s["key"], w["knorm_w"], w["knorm_b"], hd, EPS, s["key_n"])
    be.launch_rope_interleave(s["key_n"], 1, hd, ROPE, pos, THETA)
    be.launch_gemv_fp8(s["q_resid"], w["wq_b"], w["wq_b_scale"], nh * hd, Q_LORA, BLOCK, 1, s["iq"])
    be.launch_rope_interleave(s["iq"], nh, hd, ROPE, pos, THETA)
    be.launch_gemv_fp8(s["x"], w["wproj"], w["wproj_scale"], nh, HIDDEN, BLOCK, 1, s["iw"])
    # cache the token, absorb the query
    be.launch_append_kv(s["latent"], s["rope"], s["lc8"], s["lscale"], s["rc"], pos, KV_LORA, ROPE, nb)
    be.launch_index_append(s["key_n"], s["keys"], pos, hd)
    be.launch_mla_absorb(s["q"], s["kvb"], s["kvb_scale"], H, NOPE + ROPE, NOPE, V_HEAD, KV_LORA, BLOCK, 1, s["qabs"])
    be.launch_gather_rope(s["q"], s["qrope"], H, NOPE + ROPE, NOPE, ROPE)
    # rows to attend: the whole prefix up to top_k tokens, the indexer's choice beyond
    rows, n = None, nt
    if nt > k:
        be.launch_index_score(s["iq"], s["iw"], s["keys"], None, nt, nh, nh, hd, nh ** -0.5, hd ** -0.5, s["scores"])
        be.launch_index_topk(s["scores"], nt, k, s["rows"])
        rows, n = s["rows"], k
    be.launch_attend(s["qabs"], s["qrope"], s["lc8"], s["lscale"], s["rc"], rows, H, n, KV_LORA, ROPE, nb, WIDTH ** -0.5,
                     s["clat"], s["partial"])
    be.launch_mla_value(s["clat"], s["kvb"], s["kvb_scale"], H, NOPE, V_HEAD, KV_LORA, BLOCK, 1, s["ctx"])
    return {n: s[n] for n in ("key_n", "iq", "iw", "qabs", "qrope", "scores", "rows", "clat", "ctx", "lc8", "lscale", "rc", "keys")}


def _comp(rnd, d, n_pos, rotate, n_seqs=0):
    """Parameters of one compressor and, with ``n_seqs``, its pooling state in the middle of a text."""
    p = be.CompGeom.make(ratio=4, d=d, rd=ROPE)
    ang = torch.rand((n_pos, ROPE // 2), generator=rnd.gen, device=DEV) * (2 * math.pi)
    freqs = torch.stack([ang.cos(), ang.sin()], dim=-1).reshape(n_pos, ROPE).contiguous()
    norm = rnd.f32(d, scale=0.1, shift=1.0).to(torch.bfloat16).float()
    ape = rnd.f32(p.ratio, p.cd, scale=0.5)
    if not n_seqs:
        return p, ape, norm, freqs
    c = V4Compressor(p, n_seqs, ape, norm, freqs, rotate, device=DEV)
    c.kv_state.copy_(rnd.f32(n_seqs, p.ents, p.cd))
    c.score_state.copy_(rnd.f32(n_seqs, p.ents, p.cd))
    return c


def _v4_geom(case):
    return be.V4Geom.make(max_comp=-(-case["ctx"] // 4))


def _v4_positions(case):
    """Query positions: the last sixteenth of the context, so that a block closes for about every fourth sequence."""
    b, ctx = case["batch"], case["ctx"]
    return [ctx - 1 - (ctx // 16) * i // b for i in range(b)]


def _spread(rnd, *shape):
    """Indexer rows as the cache holds them: rotated, quantised to fp4 and back, bf16."""
    d = shape[-1]
    rows = rnd.bf16(math.prod(shape[:-1]), d).float()
    be.launch_act_quant_f4_rotated(rows, rows.shape[0], d)
    return rows.to(torch.bfloat16).view(torch.uint16).view(*shape)


def _prepare_v4(case, rnd):
    g, b, ctx = _v4_geom(case), case["batch"], case["ctx"]
    pos = _v4_positions(case)
    rnd.host.shuffle(pos)
    L = V4DecodeLayer(g, b, device=DEV)
    L.kv_cache.copy_(rnd.bf16(*L.kv_cache.shape).view(torch.uint16))
    L.index_kv.copy_(_spread(rnd, *L.index_kv.shape))
    L.sink.copy_(rnd.f32(g.n_heads))
    attn, index = _comp(rnd, g.head_dim, ctx, False, b), _comp(rnd, g.index_dim, ctx, True, b)
    token = V4TokenStep(L, attn, index)
    pos = _i32(pos)
    L.pack_index_rows(None, (pos // 4).to(torch.int32), g.max_comp)
    return dict(token=token, args=(pos, rnd.bf16(b, g.head_dim).view(torch.uint16), (rnd.f32(b, attn.p.cd), rnd.f32(b, attn.p.cd)),
                                   (rnd.f32(b, index.p.cd), rnd.f32(b, index.p.cd)),
                                   rnd.bf16(b, g.n_heads, g.head_dim).view(torch.uint16), _spread(rnd, b, g.index_heads, g.index_dim),
                                   (rnd.f32(b, g.index_heads) * g.index_heads ** -0.5).to(torch.bfloat16).float()))


def _run_v4(s):
    t = s["token"]
    L, bf = t.layer, torch.bfloat16
    out = t(*s["args"])
    return dict(out=out.view(bf), sel=L.sel, kv_cache=L.kv_cache.view(bf), index_kv=L.index_kv.view(bf), packed=L.packed,
                packed_exp=L.packed_exp, kv_state=t.attn_comp.kv_state, score_state=t.attn_comp.score_state,
                index_kv_state=t.index_comp.kv_state, index_score_state=t.index_comp.score_state)


def _prepare_v4_prompt(case, rnd):
    n, arms = case["tokens"], []
    for d in (512, 128):
        p, ape, norm, freqs = _comp(rnd, d, n, d == 128)
        arms.append(dict(p=p, ape=ape, norm=norm, freqs=freqs, kv=rnd.f32(n, p.cd), score=rnd.f32(n, p.cd),
                         out=torch.zeros((n // p.ratio, d), device=DEV), kv_state=torch.zeros((p.ents, p.cd), device=DEV),
                         score_state=torch.full((p.ents, p.cd), float("-inf"), device=DEV)))
    return dict(n=n, arms=arms)


def _run_v4_prompt(s):
    n = s["n"]
    for a in s["arms"]:
        p, blocks = a["p"], n // a["p"].ratio
        be.launch_kv_compress_prefill(a["kv"], a["score"], a["ape"], a["norm"], a["freqs"], a["out"], p, blocks)
        if p.d == 512:
            be.launch_act_quant_f8_prefix(a["out"], a["out"], blocks, p.d, p.d - p.rd, 64)
        else:
            be.launch_act_quant_f4_rotated(a["out"], blocks, p.d)
        be.launch_kv_compress_deposit(a["kv"], a["score"], a["ape"], a["kv_state"], a["score_state"], p, n, 0)
    return [dict(out=a["out"], kv_state=a["kv_state"], score_state=a["score_state"]) for a in s["arms"]]


_PREPARE = dict(step=_prepare_step, stack=_prepare_stack, prompt=_prepare_prompt, proj=_prepare_proj, operators=_prepare_operators,
                v4=_prepare_v4, v4_prompt=_prepare_v4_prompt)
_RUN = dict(step=_run_step, stack=_run_stack, prompt=_run_prompt, proj=_run_proj, operators=_run_operators, v4=_run_v4,
            v4_prompt=_run_v4_prompt)


def prepare(case: dict, seed: int):
    state = _PREPARE[case["kind"]](case, _Rand(seed))
    state["kind"] = case["kind"]
    return state


def run(state):
    return _RUN[state["kind"]](state)


# --- what a pass cannot do without --------------------------------------------------------------------------------
def _append_bytes(hd):
    return WIDTH * 2 + hd * 2 + 4 + WIDTH + 4 + hd + 4


def _attend_work(case, n_sel):
    H = case["heads"]
    return n_sel * (WIDTH + 4) + H * WIDTH * 2 + H * KV_LORA * 2 + H * 4, 2 * H * n_sel * (WIDTH + KV_LORA)


def _full_layer_work(case):
    nh, hd, k = case["index_heads"], case["index_dim"], case["top_k"]
    nbytes = flops = 0
    for nt in lengths(case):
        n_sel = min(k, nt)
        b, f = _attend_work(case, n_sel)
        nbytes += _append_bytes(hd) + nt * (hd + 4) + nh * hd * 2 + nh * 4 + n_sel * 4 + b
        flops += 2 * nh * hd * nt + f
    return nbytes, flops


def _shared_layer_work(case):
    nbytes = flops = 0
    for nt in lengths(case):
        n_sel = min(case["top_k"], nt)
        b, f = _attend_work(case, n_sel)
        nbytes += WIDTH * 3 + 8 + n_sel * 4 + b
        flops += f
    return nbytes, flops


def work(case: dict) -> dict:
    kind, nh, hd, H = case["kind"], MODEL["index_heads"], MODEL["index_dim"], MODEL["heads"]
    front = hd * HIDDEN + nh * hd * Q_LORA + nh * HIDDEN            # weights of the indexer's three projections
    kvb = H * (NOPE + V_HEAD) * KV_LORA
    if kind == "step":
        nbytes, flops = _full_layer_work(case)
    elif kind == "stack":
        full, shared = _full_layer_work(case), _shared_layer_work(case)
        n = LAYOUT.count("full")
        nbytes, flops = (n * f + (len(LAYOUT) - n) * s for f, s in zip(full, shared))
    elif kind == "prompt":
        nbytes, flops = case["tokens"] * (_append_bytes(hd) + 8), 0
    elif kind == "proj":
        b = case["batch"]
        acts = (HIDDEN + Q_LORA + hd + nh * hd) * 2 + nh * 4 + 4 + H * ((NOPE + ROPE) + WIDTH + KV_LORA + V_HEAD) * 2
        nbytes, flops = front + kvb + b * acts, 2 * b * (front + kvb)
    elif kind == "operators":
        nt, k = case["tokens"], case["top_k"]
        n_sel = min(nt, k)
        scored = nt if nt > k else 0
        acts = (HIDDEN + Q_LORA + hd + nh * hd + nh + H * (NOPE + ROPE + WIDTH + KV_LORA + V_HEAD)) * 4
        nbytes = front + kvb + acts + scored * (hd * 2 + 4) + n_sel * (KV_LORA + 16 + ROPE * 2 + 4)
        flops = 2 * (front + kvb) + 2 * nh * hd * scored + 2 * H * n_sel * (WIDTH + KV_LORA)
    elif kind == "v4":
        g = _v4_geom(case)
        nbytes = flops = 0
        for pos in _v4_positions(case):
            comp = (pos + 1) // g.ratio
            scored = comp if comp > g.index_topk else 0
            live = min(pos + 1, g.window) + min(comp, g.index_topk)
            closes = (pos + 1) % g.ratio == 0
            states = 2 * 2 * (g.head_dim + g.index_dim) * 4         # one (values, scores) row of width 2 d each
            nbytes += scored * (g.index_dim + 4) + g.index_heads * (g.index_dim * 2 + 4) + live * g.head_dim * 2
            nbytes += g.n_heads * g.head_dim * 4 + g.head_dim * 4 + 4 * (g.window + g.index_topk)
            nbytes += states * 2 + (states * 2 * g.ratio + (g.head_dim + g.index_dim) * 2 if closes else 0)
            flops += 2 * g.index_heads * g.index_dim * scored + 4 * g.n_heads * live * g.head_dim
    else:
        n = case["tokens"]
        nbytes = sum(n * 2 * d * 4 * 2 + n // 4 * d * 4 for d in (512, 128))
        flops = 0
    return {"bytes": nbytes, "flops": flops}


def tolerance(case: dict):
    kind = case["kind"]
    if kind == "prompt":
        return "exact"                                              # codes and scales
    if kind in ("step", "stack", "proj"):
        return {"rel": 1e-2, "max": 5e-2, "differ": 0.0}             # bf16 results; codes and selected rows are exact
    if kind == "operators":
        return {"rel": 2e-5, "max": 1e-4, "differ": 0.0}             # f32 results; codes and selected rows are exact
    if kind == "v4":
        # bf16 results; a pooled value on the edge between two codes may go either way
        return {"rel": 1e-2, "max": 1e-1, "differ": 1e-3}
    return {"rel": 2e-3, "max": 6e-1, "differ": 0.0}                 # as above, after the 4- and 8-bit round trips
