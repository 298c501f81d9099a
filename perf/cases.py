"""What the speed of this framework is measured on: the work a decoding program hands to it.

A case is one pass of such a program through the package's public operators, over the attention layers of a
model: a decode step of one token per sequence, or the append of a prompt.  The kinds are the ways in which the
path is driven:

  step     utils.decode_step_dev per layer, one sequence, captured once as a CUDA graph and replayed per token
  batch    SequenceBatch.decode_step_dev per layer, several sequences in the same launches, as a graph
  eager    the controller protocol with utils.decode_step per layer, launched call by call
  ops      the controller protocol with the separate operators (rotation, transform, append, estimate, top-k,
           sparse attention), launched call by call: what a model written for the reference's operators does
  dense    the layers that attend to every token (decode_step_dev with dense=True, one or several sequences)
  prefill  rotation and code-generating append of a prompt, or of a chunk of it behind a cached prefix

Every pass works at a fixed position, so that it can be repeated: the newest token's slot is written again.
"""
import math
from types import SimpleNamespace

import torch

import adamas_b200.utils as U
from adamas_b200 import _kernels, hadamard_transform
from adamas_b200.rope import yarn_inv_freq

DEV = "cuda:0"
DIM = 128
DTYPES = {"f16": torch.float16, "bf16": torch.bfloat16}


def _case(kind, **kw):
    c = dict(kind=kind, layers=4, batch=1, q_heads=32, kv_heads=32, ctx=4096, room=256, page=16, budget=256, dtype="f16",
             rope="none", ragged=False, past=0)
    c.update(kw)
    return c


def listed():
    return [
        # one token of a small model at a short context, call by call: launches and host time count
        _case("eager", name="eager_4k", layers=4, ctx=4096, budget=256),
        # the reference's own protocol at its own page size, every operator a call of its own
        _case("ops", name="ops_8k_page1", layers=2, ctx=8191, page=1, budget=512, rope="linear"),
        # the headline: one token of a 32-layer, 32-head model at 32K, budget 1024
        _case("step", name="step_32k", layers=32, ctx=32768, budget=1024),
        # a long context with YaRN frequencies, one sequence, all heads on one GPU
        _case("step", name="step_128k_yarn", layers=4, ctx=131072, budget=2048, dtype="bf16", rope="yarn"),
        # grouped queries, an odd length in a cache with room to grow
        _case("step", name="step_gqa_30k", layers=8, q_heads=32, kv_heads=8, ctx=30001, room=2767, budget=1024, dtype="bf16", rope="linear"),
        # 40 heads, an odd length, a small budget
        _case("step", name="step_40heads_12k", layers=8, q_heads=40, kv_heads=40, ctx=12289, room=4095, budget=320, dtype="bf16", rope="linear"),
        # one GPU's share of a model whose heads are split over eight, four long sequences
        _case("batch", name="batch4_128k_4heads", layers=4, batch=4, q_heads=4, kv_heads=4, ctx=131072, budget=2048, dtype="bf16", rope="yarn"),
        # serving: eight long sequences
        _case("batch", name="batch8_32k", layers=4, batch=8, ctx=32768, budget=512),
        # serving: many short sequences of different lengths
        _case("batch", name="batch32_8k_ragged", layers=4, batch=32, ctx=8192, budget=128, ragged=True, rope="linear"),
        # the first layers of the model, which attend to everything
        _case("dense", name="dense_32k", layers=2, ctx=32768, rope="linear"),
        # the append of a whole prompt
        _case("prefill", name="prefill_32k", layers=2, ctx=32768, rope="linear"),
        # the append of a short chunk behind a cached prefix, grouped queries
        _case("prefill", name="prefill_chunk_777", layers=2, q_heads=32, kv_heads=8, ctx=777, past=3000, dtype="bf16", rope="linear"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step", "step", "step", "batch", "batch", "eager", "ops", "dense", "prefill", "prefill"])
    hq, hkv = rng.choice([(32, 32), (32, 32), (32, 8), (16, 16), (8, 8), (4, 4), (28, 4), (40, 40), (64, 8)])
    c = _case(kind, q_heads=hq, kv_heads=hkv, dtype=rng.choice(["f16", "bf16"]), page=rng.choice([1, 16, 16, 32]),
              rope=rng.choice(["none", "linear", "yarn"]))
    if kind == "ops":
        c.update(kv_heads=hq if hq <= 40 else 32, q_heads=hq if hq <= 40 else 32)   # (this protocol is multi-head)
        c["rope"] = rng.choice(["none", "linear"])
    if kind == "prefill":
        c["ctx"] = _log(rng, 2, 32768)
        c["past"] = rng.choice([0, _log(rng, 16, 32768)])
        c["rope"] = "linear"
        c["layers"] = rng.choice([1, 2])
        return _within(c)
    if kind == "batch" or (kind == "dense" and rng.random() < 0.5):
        c["batch"] = _log(rng, 2, 32)
        c["ragged"] = rng.random() < 0.5
    top = {"step": 131072, "batch": 131072, "eager": 32768, "ops": 32768, "dense": 65536}[kind]
    top = min(top, 8 * 32768 * 32 // (c["batch"] * c["kv_heads"] * (4 if kind == "dense" else 1)))
    c["ctx"] = _log(rng, 1500, max(3000, top))
    c["room"] = _log(rng, 32, c["ctx"])
    if c["ragged"] and c["batch"] > 1:
        shortest = c["ctx"] // 2
    else:
        shortest = c["ctx"]
    c["budget"] = max(c["page"], _log(rng, 64, min(4096, shortest // 2)) // c["page"] * c["page"])
    # enough layers that a pass does not live in the cache, no more than the listed cases hold
    held = c["batch"] * (c["ctx"] + c["room"]) * c["kv_heads"] * 544
    c["layers"] = max(1, min(8, int(12e9 // held)))
    if kind in ("eager", "ops", "dense"):
        c["layers"] = min(c["layers"], 2)
    return _within(c)


def _within(c):
    """The case with fewer layers, then a smaller budget or prompt, until it costs no more than the listed ones of its kind do."""
    most = 3.8e9 if c["kind"] == "prefill" else 1.2e9
    while work(c)["bytes"] > most:
        if c["layers"] > 1:
            c["layers"] -= 1
        elif c["kind"] == "prefill" or c["budget"] < 4 * c["page"]:
            c["ctx"] = c["ctx"] * 3 // 4
        else:
            c["budget"] = c["budget"] // 2 // c["page"] * c["page"]
    return c


# ---- inputs ---------------------------------------------------------------------------------------------------
def _values(gen, shape, dtype, std, offsets):
    """Normal values plus a per-(head, channel) offset: keys and queries of real models have a few large channels,
    constant over the tokens, which spread the codes over all four buckets."""
    x = torch.empty(shape, dtype=dtype, device=DEV).normal_(0.0, std, generator=gen)
    return x.add_(offsets) if offsets is not None else x


def _offsets(gen, heads, dtype, size):
    o = torch.zeros(heads, DIM, device=DEV)
    at = torch.randint(0, DIM, (heads, 4), generator=gen, device=DEV)
    sign = torch.randint(0, 2, (heads, 4), generator=gen, device=DEV).float() * 2 - 1
    return o.scatter_(1, at, sign * size).to(dtype)


def _controller(case, capacity):
    hkv = case["kv_heads"]
    return U.InferenceController(case["layers"], hkv, DIM, case["page"], case["budget"] // case["page"], capacity,
                                 DTYPES[case["dtype"]], DEV, num_q_heads=case["q_heads"])


def _fill(c, case, gen, tokens, k_off):
    dtype, hkv = DTYPES[case["dtype"]], case["kv_heads"]
    c.prepare_hadamard(tokens)
    c.begin_forward(tokens)
    for layer in range(case["layers"]):
        k = _values(gen, (tokens, hkv, DIM), dtype, 1.5, k_off[layer])
        v = _values(gen, (tokens, hkv, DIM), dtype, 1.0, None)
        if tokens > 1:
            U.append_kvh(k, v, None, c, layer)
        else:
            U.append_qkv_fused(k.repeat_interleave(case["q_heads"] // hkv, 1).contiguous(), k, v, c, layer)
    c.end_forward()


def _lengths(case):
    """Tokens of each sequence, the newest included."""
    b, n = case["batch"], case["ctx"]
    if not case["ragged"] or b == 1:
        return [n] * b
    return [n - (n // 2) * i // (b - 1) for i in range(b)]


def _rope(case):
    if case["rope"] == "linear":
        return (8.0, 1e4)
    if case["rope"] == "yarn":
        inv_freq, mscale = yarn_inv_freq(32.0, 4096)
        return {"inv_freq": inv_freq.to(DEV), "mscale": mscale}
    return None


def _newest(c):
    """The cache rows of the newest token, all layers: K and V, and the packed key code."""
    page, entry = c.kv_cache.indicies[-1], c.kv_cache.last_page_len - 1
    code_page = c.hadamard_cache.indicies[-1]
    return c.kv_cache.pool.buf[:, page, :, entry], c.hadamard_cache.pool.buf[:, code_page, 0, entry].view(torch.int16)


def prepare(case, seed):
    gen = torch.Generator(device=DEV).manual_seed(int(seed))
    dtype, layers, b = DTYPES[case["dtype"]], case["layers"], case["batch"]
    hq, hkv = case["q_heads"], case["kv_heads"]
    k_off = [_offsets(gen, hkv, dtype, 20.0) for _ in range(layers)]
    q_off = [_offsets(gen, hq, dtype, 6.0) for _ in range(layers)]
    s = SimpleNamespace(case=case, layers=layers, rope=_rope(case))

    if case["kind"] == "prefill":
        c = s.c = _controller(case, case["past"] + case["ctx"])
        c.kv_cache.pool.buf.zero_()
        c.hadamard_cache.pool.buf.zero_()
        if case["past"]:
            _fill(c, case, gen, case["past"], k_off)
        n = case["ctx"]
        s.q = [_values(gen, (n, hq, DIM), dtype, 1.5, q_off[l]) for l in range(layers)]
        s.k = [_values(gen, (n, hkv, DIM), dtype, 1.5, k_off[l]) for l in range(layers)]
        s.v = [_values(gen, (n, hkv, DIM), dtype, 1.0, None) for l in range(layers)]
        c.prepare_hadamard(n)
        s.out = s.q + s.k + [c.kv_cache.pool.buf, c.hadamard_cache.pool.buf.view(torch.int16)]
        return s

    # the newest token's projections, one row per (layer, sequence): `fresh` is what the model computes, `rows` the
    # buffers it writes them to (a step with a rotation rotates q and k in place)
    parts = [torch.cat([_values(gen, (b, hq, DIM), dtype, 1.5, q_off[l]), _values(gen, (b, hkv, DIM), dtype, 1.5, k_off[l]),
                        _values(gen, (b, hkv, DIM), dtype, 1.0, None)], 1).transpose(0, 1) for l in range(layers)]
    s.fresh = torch.stack(parts).contiguous()                       # [layers, Hq + 2 H, batch, D]
    s.fresh = torch.cat([s.fresh[:, :hq].transpose(1, 2).reshape(layers, -1), s.fresh[:, hq:hq + hkv].transpose(1, 2).reshape(layers, -1),
                         s.fresh[:, hq + hkv:].transpose(1, 2).reshape(layers, -1)], 1).contiguous()
    s.rows = s.fresh.clone()
    nq, nk = b * hq * DIM, b * hkv * DIM
    s.q = [s.rows[l, :nq].view(b, hq, DIM) for l in range(layers)]
    s.k = [s.rows[l, nq:nq + nk].view(b, hkv, DIM) for l in range(layers)]
    s.v = [s.rows[l, nq + nk:].view(b, hkv, DIM) for l in range(layers)]
    s.o = torch.zeros(layers, b, hq, DIM, dtype=dtype, device=DEV)

    controllers = []
    for n in _lengths(case):
        c = _controller(case, case["ctx"] + case["room"])
        _fill(c, case, gen, n - 1, k_off)
        if b == 1:
            c.prepare_hadamard(1)
            c.begin_forward(1)
        controllers.append(c)
    s.c = controllers[0]
    if b > 1:
        s.batch = U.SequenceBatch(controllers)
        s.batch.prepare(1)
        s.batch.sync_seq_lens()
    rows = [_newest(c) for c in controllers]
    s.out = [s.o, s.rows] + [r[0] for r in rows] + ([r[1] for r in rows] if b <= 24 else [])   # (64 outputs at most)
    if case["kind"] in ("eager", "ops"):
        return s

    # one token's work as a graph, as a decode loop keeps it
    dense = case["kind"] == "dense"
    if b == 1:
        s.c.sync_seq_len()

    def token():
        s.rows.copy_(s.fresh)
        for l in range(layers):
            if b > 1:
                s.batch.decode_step_dev(s.q[l], s.k[l], s.v[l], l, out=s.o[l], dense=dense, rope=s.rope)
            else:
                U.decode_step_dev(s.q[l], s.k[l], s.v[l], s.c, l, out=s.o[l], dense=dense, rope=s.rope)

    token()
    torch.cuda.synchronize()
    s.graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(s.graph):
        token()
    return s


# ---- one pass -------------------------------------------------------------------------------------------------
def _run_prefill(s):
    c, case = s.c, s.case
    c.begin_forward(case["ctx"])
    for l in range(s.layers):
        U.apply_rope_in_place(s.q[l], s.k[l], case["past"], rope_scale=s.rope[0], rope_theta=s.rope[1])
        U.append_kvh(s.k[l], s.v[l], None, c, l)
    c.end_forward()
    return s.out


def _run_eager(s):
    c = s.c
    if s.rope is not None:
        s.rows.copy_(s.fresh)
    c.begin_forward(1)
    for l in range(s.layers):
        U.decode_step(s.q[l], s.k[l], s.v[l], c, l, out=s.o[l], rope=s.rope)
    c.end_forward()
    return s.out + [c.topk_dindices_buffer]


def _run_ops(s):
    c = s.c
    if s.rope is not None:
        s.rows.copy_(s.fresh)
    c.begin_forward(1)
    for l in range(s.layers):
        q, k, v = s.q[l], s.k[l], s.v[l]
        if s.rope is not None:
            U.apply_rope_in_place(q, k, c.kv_cache.seqlen - 1, rope_scale=s.rope[0], rope_theta=s.rope[1])
        q_code = U.append_kvh(k, v, hadamard_transform(torch.cat((q, k), dim=0)), c, l)
        est = U.decode_estimate(q_code, c, l)
        U.decode_topk(est, c)
        U.decode_sparse_attn(q, c, l, c.topk_dindices_buffer, out=s.o[l])
    c.end_forward()
    return s.out + [est.view(torch.int16), c.topk_dindices_buffer]


def run(s):
    kind = s.case["kind"]
    if kind == "prefill":
        return _run_prefill(s)
    if kind == "eager":
        return _run_eager(s)
    if kind == "ops":
        return _run_ops(s)
    s.graph.replay()
    return s.out


# ---- what a pass cannot do without ----------------------------------------------------------------------------
def work(case):
    hq, hkv, layers = case["q_heads"], case["kv_heads"], case["layers"]
    row = DIM * 2
    if case["kind"] == "prefill":
        n = case["ctx"]
        # q and k read and rotated in place, v read, K and V rows and the codes written
        bytes_ = n * (hq * 2 * row + hkv * (2 * row + row + 2 * row + 32))
        return {"bytes": layers * bytes_, "flops": layers * n * (hq + hkv) * DIM * 3 + layers * n * hkv * DIM * 8}
    bytes_ = flops = 0
    for n in _lengths(case):
        io = 2 * hq * row + 2 * hkv * row + hkv * (2 * row + 32)      # q in, o out; k, v in; K, V rows and code written
        if case["kind"] == "dense":
            attended = n * hkv
            scanned = 0
            pairs = n * hq
        else:
            # each query head has its own selection (heads that share a cache head read no row twice at best)
            attended = min(case["budget"] * hq, n * hkv)
            scanned = (n - 1) * hkv * 32
            pairs = case["budget"] * hq
            if case["kind"] in ("eager", "ops"):
                io += hq * (case["budget"] - 1) * 4                     # the selected slots are an output
            if case["kind"] == "ops":
                io += hq * (n - 1) * 2 + hq * 2 * 16                    # so are the distances and the query code
        bytes_ += layers * (io + attended * 2 * row + scanned)
        flops += layers * pairs * 4 * DIM
    return {"bytes": bytes_, "flops": flops}


def tolerance(case):
    # 32-bit accumulation, results rounded to 16 bits: one unit in the last place apart here and there; whole values
    # (codes, distances, selected slots) are the same.  A prompt's rotation rounds before it is coded, so that a
    # value at a threshold may fall on either side.
    rel = 1e-3 if case["dtype"] == "f16" else 5e-3
    return {"rel": rel, "differ": 1e-3 if case["kind"] == "prefill" else 0.0}
