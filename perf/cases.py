"""Performance cases of the split12 library: what they hold, how to run one, and what its outputs must be.

Every case is one pass through the package's public entry points, on synthetic tensors of the shapes that
``bench.py`` and the tests use.  Kinds:

  gemv      single-sequence products with a few small tensors (escapes corrected in the launch)
  layer     the seven projections of one decoder layer for a batch of sequences: q/k/v, o, gate/up, down
  gemm      one tensor times many activation rows (a prompt chunk)
  step      a whole greedy decode step of a small stack of layers, every kernel of it, with the output projection
  attention decode attention over the INT8 cache, sequences at different positions
  moe       the top-2 mixture-of-experts block
  pack      bf16 -> split12, as a program that converts weights on the device does it
  decompress  split12 -> bf16

Cases with ``graph`` set keep a captured CUDA graph of their calls, as a serving loop does (positions, tokens and
activations live in device memory, so one graph serves every step); the others call the library eagerly.
"""
import math

import torch

from turbo_lossless_b200 import CompressedWeight, Decoder, DecoderConfig, Split12Engine
from turbo_lossless_b200.moe import MoEFeedForward


def listed():
    return [
        # the smallest calls: two 4096 x 4096 tensors with 0.05 % outliers, one product each
        dict(name="gemv_4096x4096", kind="gemv", count=2, M=4096, K=4096, outliers=5e-4, graph=True),
        # interactive generation: one sequence, 256 positions in the cache
        dict(name="step_b1_position255", kind="step", hidden=4096, heads=32, kv_heads=8, ffn=14336, vocab=32000, layers=2,
             batch=1, position=255, max_seq=384, graph=True),
        # a few users or speculative tokens: an odd small batch
        dict(name="layer_b11", kind="layer", hidden=4096, q=4096, kv=1024, ffn=14336, batch=11, graph=True),
        # a small server's batch, not a power of two
        dict(name="layer_b40", kind="layer", hidden=4096, q=4096, kv=1024, ffn=14336, batch=40, graph=False),
        # the largest dense layer at a medium batch
        dict(name="layer_wide_b64", kind="layer", hidden=8192, q=8192, kv=1024, ffn=28672, batch=64, graph=False),
        # throughput serving: projections alone, then the whole step with its large vocabulary
        dict(name="layer_b256", kind="layer", hidden=4096, q=4096, kv=1024, ffn=14336, batch=256, graph=False),
        dict(name="step_b256_position191", kind="step", hidden=4096, heads=32, kv_heads=8, ffn=14336, vocab=128256, layers=2,
             batch=256, position=191, max_seq=256, graph=True),
        # a prompt chunk through one projection
        dict(name="gemm_1000_rows", kind="gemm", M=14336, K=4096, batch=1000),
        # long contexts of a mid-size batch
        dict(name="attention_b24_4k", kind="attention", heads=32, kv_heads=8, head_dim=128, batch=24, longest=4096),
        # mixture of experts, 0.25 % outliers in the expert weights
        dict(name="moe_b64", kind="moe", hidden=4096, ffn=14336, experts=8, batch=64, outliers=2.5e-3),
        # load time: converting a weight, and getting it back
        dict(name="pack_14336x4096", kind="pack", M=14336, K=4096, outliers=5e-4),
        dict(name="decompress_14336x4096", kind="decompress", M=14336, K=4096, outliers=5e-4),
    ]


def _log(rng, lo, hi, step=1):
    """A multiple of ``step`` in [lo, hi], spread over its logarithm."""
    v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return int(min(hi, max(lo, round(v / step) * step)))


def draw(rng):
    kind = rng.choice(["gemv", "layer", "layer", "gemm", "step", "attention", "attention", "moe", "pack", "decompress"])
    if kind == "gemv":
        return dict(kind=kind, count=rng.randint(1, 4), M=_log(rng, 1024, 16384), K=_log(rng, 1024, 16384, 32),
                    outliers=rng.choice([0.0, 5e-4, 2.5e-3]), graph=True)
    if kind == "layer":
        hidden = _log(rng, 1024, 8192, 128)
        batch = _log(rng, 1, 300)
        return dict(kind=kind, hidden=hidden, q=hidden, kv=rng.choice([hidden, hidden // 4, hidden // 8]),
                    ffn=_log(rng, 2 * hidden, int(3.5 * hidden), 32), batch=batch, graph=batch <= 16)
    if kind == "gemm":
        return dict(kind=kind, M=_log(rng, 1000, 30000), K=_log(rng, 1024, 8192, 32), batch=_log(rng, 17, 1024))
    if kind == "step":
        head_dim = rng.choice([64, 128])
        kv_heads = rng.choice([2, 4, 8])
        heads = kv_heads * rng.choice([1, 2, 4])
        position = _log(rng, 1, 1000)
        return dict(kind=kind, hidden=heads * head_dim, heads=heads, kv_heads=kv_heads, ffn=_log(rng, 512, 8192, 32),
                    vocab=_log(rng, 1000, 64000), layers=rng.randint(1, 3), batch=_log(rng, 1, 256), position=position,
                    max_seq=position + rng.randint(1, 200), graph=True)
    if kind == "attention":
        kv_heads = rng.choice([1, 2, 8])
        batch = _log(rng, 1, 256)
        return dict(kind=kind, heads=kv_heads * rng.choice([1, 2, 4, 8]), kv_heads=kv_heads, head_dim=rng.choice([64, 96, 128]),
                    batch=batch, longest=_log(rng, 16, min(16000, 400000 // batch)))
    if kind == "moe":
        return dict(kind=kind, hidden=_log(rng, 1024, 4096, 32), ffn=_log(rng, 2048, 8192, 32), experts=rng.choice([4, 8, 16]),
                    batch=_log(rng, 1, 128), outliers=rng.choice([0.0, 2.5e-3]))
    return dict(kind=kind, M=_log(rng, 512, 30000), K=_log(rng, 512, 8192, 2), outliers=rng.choice([0.0, 5e-4, 2.5e-3]))


# ---- inputs, from the seed alone --------------------------------------------------------------------------------

def _gen(seed, i):
    return torch.Generator(device="cuda").manual_seed((seed * 1000003 + i) % (1 << 62))


def _weight(seed, i, M, K, outliers=0.0):
    """bf16 [M, K]: N(0, 0.02) with a share of entries a hundred times larger."""
    g = _gen(seed, i)
    w = torch.randn(M, K, generator=g, device="cuda") * 0.02
    if outliers:
        w = torch.where(torch.rand(M, K, generator=g, device="cuda") < outliers, w * 100.0, w)
    return w.to(torch.bfloat16)


def _weight_to_pack(seed, M, K, outliers):
    """bf16 [M, K] whose number of escapes follows from the sizes alone, so that every seed's packed form has the same
    shapes: magnitudes of N(0, 0.02) kept inside 14 octaves, and one entry of every 1 / outliers (at a random place
    among them) far above."""
    g = _gen(seed, 0)
    w = torch.randn(M * K, generator=g, device="cuda") * 0.02
    w = torch.copysign(w.abs().clamp(2.0 ** -17, 0.12), w)
    if outliers:
        every = round(1.0 / outliers)
        n = M * K // every
        at = torch.arange(n, device="cuda") * every + torch.randint(0, every, (n,), generator=g, device="cuda")
        w[at] = torch.copysign(1.0 + 3.0 * torch.rand(n, generator=g, device="cuda"), w[at])
    return w.to(torch.bfloat16).view(M, K)


def _acts(seed, i, B, K):
    return torch.randn(B, K, generator=_gen(seed, i), device="cuda").to(torch.bfloat16)


def _layer_shapes(c):
    H = c["hidden"]
    q = c.get("q", H)
    kv = c["kv"] if "kv" in c else H // c["heads"] * c["kv_heads"]
    return {"wq": (q, H), "wk": (kv, H), "wv": (kv, H), "wo": (H, q), "w_gate": (c["ffn"], H), "w_up": (c["ffn"], H),
            "w_down": (H, c["ffn"])}


def _layer_weights(c, seed, li):
    """(name, bf16 tensor) of one layer, one at a time."""
    for i, (name, (M, K)) in enumerate(_layer_shapes(c).items()):
        yield name, _weight(seed, 100 * (li + 1) + i, M, K)


def _step_inputs(c, seed):
    """What a decode step reads besides its projections: table, norms, tokens, positions, cache with earlier entries."""
    g = _gen(seed, 7)
    r = dict(generator=g, device="cuda")
    H, B, L, hd = c["hidden"], c["batch"], c["layers"], c["hidden"] // c["heads"]
    names = [f"{k}.{i}" for i in range(L) for k in ("attn_norm", "ffn_norm")] + ["output_norm"]
    cache = (L, B, c["max_seq"], c["kv_heads"])
    return dict(embd=torch.randn(c["vocab"], H, **r).to(torch.bfloat16),
                norms={n: 1.0 + 0.1 * torch.randn(H, **r) for n in names},
                tokens=torch.randint(0, c["vocab"], (B,), dtype=torch.int32, **r),
                positions=torch.randint(c["position"] // 2, c["position"] + 1, (B,), dtype=torch.int32, **r),
                kv_k=torch.randint(-127, 128, cache + (hd,), dtype=torch.int8, **r),
                kv_v=torch.randint(-127, 128, cache + (hd,), dtype=torch.int8, **r),
                sc_k=0.01 + 0.02 * torch.rand(cache, **r), sc_v=0.01 + 0.02 * torch.rand(cache, **r))


def _attention_inputs(c, seed):
    r = dict(generator=_gen(seed, 3), device="cuda")
    B, T, n, hd = c["batch"], c["longest"], c["kv_heads"], c["head_dim"]
    positions = torch.randint(T // 2, T, (B,), dtype=torch.int32, **r)
    positions[0] = T - 1
    return dict(q=torch.randn(B, c["heads"] * hd, **r), positions=positions,
                kv_k=torch.randint(-127, 128, (B, T, n, hd), dtype=torch.int8, **r),
                kv_v=torch.randint(-127, 128, (B, T, n, hd), dtype=torch.int8, **r),
                sc_k=0.01 + 0.02 * torch.rand(B, T, n, **r), sc_v=0.01 + 0.02 * torch.rand(B, T, n, **r))


# ---- what a program holds, and one pass ---------------------------------------------------------------------------

def _call(state):
    """The library calls of one pass."""
    e, kind = state["eng"], state["kind"]
    if kind == "gemv":
        for w, o in zip(state["ws"], state["outs"]):
            e.gemv([w], state["x"], [o])
    elif kind == "layer":
        B, L, o = state["batch"], state["layer"], state["outs"]
        for names, x in ((("wq", "wk", "wv"), state["x_in"]), (("wo",), state["x_attn"]), (("w_gate", "w_up"), state["x_in"]),
                         (("w_down",), state["x_ffn"])):
            if B == 1:
                e.gemv([L[n] for n in names], x, [o[n] for n in names])
            else:
                e.gemm_multi([L[n] for n in names], x, [o[n] for n in names], x.shape[1], B)
    elif kind == "gemm":
        e.gemm(state["w"], state["x"], state["outs"], state["w"].K, state["w"].M, state["batch"])
    elif kind == "step":
        state["decoder"].forward()
    elif kind == "attention":
        s = state["in"]
        e.attention_all_heads_batch(s["q"], s["kv_k"], s["kv_v"], s["sc_k"], s["sc_v"], state["outs"].view(torch.int16), s["positions"],
                                    state["heads"], state["kv_heads"], state["head_dim"], state["longest"],
                                    1.0 / math.sqrt(state["head_dim"]), state["batch"],
                                    state["longest"] * state["kv_heads"] * state["head_dim"])
    elif kind == "moe":
        state["block"].forward(state["x"].view(torch.int16), state["router"], state["outs"])
    elif kind == "decompress":
        e.decompress(state["w"], state["outs"])


def prepare(case, seed):
    c = case
    kind = c["kind"]
    eng = Split12Engine()
    eng.init()
    eng.set_dependent_launch(True)
    s = dict(c, eng=eng)
    f32 = dict(device="cuda", dtype=torch.float32)
    pack = CompressedWeight.pack_on_device
    if kind == "gemv":
        s["ws"] = [pack(_weight(seed, i, c["M"], c["K"], c["outliers"])) for i in range(c["count"])]
        s["x"] = _acts(seed, 90, 1, c["K"])
        s["outs"] = [torch.empty(c["M"], **f32) for _ in range(c["count"])]
    elif kind == "layer":
        s["layer"] = {n: pack(w) for n, w in _layer_weights(c, seed, 0)}
        s["x_in"], s["x_attn"], s["x_ffn"] = (_acts(seed, 90 + i, c["batch"], k) for i, k in enumerate((c["hidden"], c["q"], c["ffn"])))
        s["outs"] = {n: torch.empty(c["batch"], M, **f32) for n, (M, K) in _layer_shapes(c).items()}
    elif kind == "gemm":
        s["w"] = pack(_weight(seed, 0, c["M"], c["K"]))
        s["x"] = _acts(seed, 90, c["batch"], c["K"])
        s["outs"] = torch.empty(c["batch"], c["M"], **f32)
    elif kind == "step":
        i = _step_inputs(c, seed)
        cfg = DecoderConfig(n_embd=c["hidden"], n_head=c["heads"], n_head_kv=c["kv_heads"], n_ff=c["ffn"], n_vocab=c["vocab"],
                            n_layer=c["layers"], max_seq=c["max_seq"])
        layers = [{n: pack(w) for n, w in _layer_weights(c, seed, li)} for li in range(c["layers"])]
        d = Decoder(cfg, layers, pack(_weight(seed, 99, c["vocab"], c["hidden"])), i["embd"].view(torch.int16), i["norms"],
                    batch=c["batch"], eng=eng)
        d.tokens.copy_(i["tokens"]); d.positions.copy_(i["positions"])
        d.kv_k, d.kv_v, d.sc_k, d.sc_v = i["kv_k"], i["kv_v"], i["sc_k"], i["sc_v"]
        s["decoder"] = d
        s["outs"] = {"logits": d.logits, "kv_k": d.kv_k, "kv_v": d.kv_v, "sc_k": d.sc_k, "sc_v": d.sc_v}
    elif kind == "attention":
        s["in"] = _attention_inputs(c, seed)
        s["outs"] = torch.empty(c["batch"], c["heads"] * c["head_dim"], device="cuda", dtype=torch.bfloat16)
    elif kind == "moe":
        experts = [{n: pack(_weight(seed, 10 * e + j, *mk, c["outliers"])) for j, (n, mk) in enumerate(
            (("w_gate", (c["ffn"], c["hidden"])), ("w_up", (c["ffn"], c["hidden"])), ("w_down", (c["hidden"], c["ffn"]))))}
            for e in range(c["experts"])]
        s["block"] = MoEFeedForward(experts, c["batch"], eng=eng)
        s["x"] = _acts(seed, 990, c["batch"], c["hidden"])
        s["router"] = torch.rand(c["batch"], c["experts"], generator=_gen(seed, 991), device="cuda")
        s["outs"] = torch.empty(c["batch"], c["hidden"], **f32)
    elif kind == "pack":
        s["bf16"] = _weight_to_pack(seed, c["M"], c["K"], c["outliers"])
    elif kind == "decompress":
        s["w"] = pack(_weight(seed, 0, c["M"], c["K"], c["outliers"]))
        s["outs"] = torch.empty(c["M"], c["K"], device="cuda", dtype=torch.int16)
    if c.get("graph"):
        side = torch.cuda.Stream()
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            _call(s)
        torch.cuda.current_stream().wait_stream(side)
        s["captured"] = torch.cuda.CUDAGraph()
        with torch.cuda.graph(s["captured"]):
            _call(s)
    return s


def run(state):
    if state["kind"] == "pack":
        w = CompressedWeight.pack_on_device(state["bf16"])
        return [w.split_sm, w.split_gr, w.base_exp, w.row_offsets, w.patch_cols, w.patch_correct, w.patch_wrong]
    if state.get("graph"):
        state["captured"].replay()
    else:
        _call(state)
    return state["outs"]


# ---- what a pass cannot do without -------------------------------------------------------------------------------

def _product(M, K, B, outliers=0.0):
    """(bytes, flops) of one packed tensor times B rows: 1.5 bytes a weight, the escape list, activations, outputs."""
    return 1.5 * M * K + 8.0 * outliers * M * K + 4.0 * (M + 1) + 2.0 * B * K + 4.0 * B * M, 2.0 * M * K * B


def _attention_work(lengths, heads, kv_heads, hd, batch):
    return lengths * kv_heads * (2 * hd + 8) + batch * heads * hd * 6, 4.0 * lengths * heads * hd


def work(case):
    c, kind = case, case["kind"]
    if kind == "gemv":
        b, f = _product(c["M"], c["K"], 1, c["outliers"])
        return {"bytes": b * c["count"], "flops": f * c["count"]}
    if kind == "gemm":
        b, f = _product(c["M"], c["K"], c["batch"])
        return {"bytes": b, "flops": f}
    if kind in ("layer", "step"):
        parts = [_product(M, K, c["batch"]) for M, K in _layer_shapes(c).values()] * c.get("layers", 1)
        if kind == "step":
            parts.append(_product(c["vocab"], c["hidden"], c["batch"]))
            mean = 0.75 * c["position"] + 1.0
            parts += [_attention_work(mean * c["batch"], c["heads"], c["kv_heads"], c["hidden"] // c["heads"], c["batch"])] * c["layers"]
        return {"bytes": sum(p[0] for p in parts), "flops": sum(p[1] for p in parts)}
    if kind == "attention":
        b, f = _attention_work(0.75 * c["longest"] * c["batch"], c["heads"], c["kv_heads"], c["head_dim"], c["batch"])
        return {"bytes": b, "flops": f}
    if kind == "moe":
        used = min(c["experts"], 2 * c["batch"])              # experts that some token chose: their weights are read
        b, f = _product(c["ffn"], c["hidden"], 0, c["outliers"])
        rows = 2.0 * c["batch"]
        return {"bytes": 3.0 * b * used + c["batch"] * c["hidden"] * 6.0, "flops": 6.0 * c["ffn"] * c["hidden"] * rows}
    return {"bytes": 3.5 * c["M"] * c["K"] + 8.0 * c["outliers"] * c["M"] * c["K"], "flops": 0.0}


def tolerance(case):
    kind = case["kind"]
    if kind in ("pack", "decompress"):
        return "exact"
    # about four times the distance from the 64-bit results at the shapes above
    if kind == "attention":
        return {"rel": 3e-4, "max": 0.03}                     # bf16 outputs of 32-bit sums: single roundings differ
    if kind == "moe":
        return {"rel": 8e-4, "max": 0.05}                     # bf16 between the projections
    if kind == "step":
        return {"rel": 1.5e-2, "max": 0.5, "differ": 5e-3}    # bf16 and int8 roundings travel through the layers
    if kind == "gemv":
        return {"rel": 2e-6}                                  # 32-bit sums
    # from 17 rows on the tensor cores cut off, where they add, what does not fit 32 bits: the error grows with K
    return {"rel": 6e-6 if case["batch"] <= 16 else 6e-5}


# ---- the same in 64 bits, plain torch -----------------------------------------------------------------------------

def _mul(x, w):
    """x [B, K] times w [M, K] transposed, in 64 bits, in pieces of w."""
    return torch.cat([x @ p.double().t() for p in w.split(16384)], dim=1)


def _bf16(x):
    return x.float().to(torch.bfloat16).double()


def _silu_mul(g, u):
    return _bf16(g / (1.0 + torch.exp(-g)) * u)


def _attend(q, k, v, sk, sv, positions, heads, kv_heads, hd):
    """q [B, heads*hd] over the INT8 cache [B, T, kv_heads, hd], one sequence at a time; bf16 values."""
    rows = []
    for b in range(q.shape[0]):
        n = int(positions[b]) + 1
        kb = k[b, :n].double() * sk[b, :n].double()[..., None]
        vb = v[b, :n].double() * sv[b, :n].double()[..., None]
        p = torch.einsum("hgd,thd->hgt", q[b].view(kv_heads, heads // kv_heads, hd), kb) / math.sqrt(hd)
        rows.append(torch.einsum("hgt,thd->hgd", torch.softmax(p, dim=-1), vb).reshape(-1))
    return _bf16(torch.stack(rows))


def _exact_step(c, seed):
    i = _step_inputs(c, seed)
    B, H, heads, n, hd = c["batch"], c["hidden"], c["heads"], c["kv_heads"], c["hidden"] // c["heads"]
    pos = i["positions"].long()
    rows = torch.arange(B, device="cuda")

    def norm(x, w):
        return _bf16(x * torch.rsqrt(x.square().mean(dim=-1, keepdim=True) + 1e-5) * w.double())

    def rope(x):
        d = torch.arange(hd // 2, device="cuda", dtype=torch.float64)
        ang = pos.double()[:, None, None] * (10000.0 ** (-2.0 * d / hd))
        x0, x1 = x.view(B, -1, hd)[..., :hd // 2], x.view(B, -1, hd)[..., hd // 2:]
        return torch.cat([x0 * ang.cos() - x1 * ang.sin(), x0 * ang.sin() + x1 * ang.cos()], dim=-1)

    def store(cache, scales, li, x):
        top = x.abs().amax(dim=-1)
        cache[li, rows, pos] = torch.clamp(torch.round(x * (127.0 / top.clamp_min(1e-300))[..., None]), -127, 127).to(torch.int8)
        scales[li, rows, pos] = top / 127.0

    i["sc_k"], i["sc_v"] = i["sc_k"].double(), i["sc_v"].double()
    cur = i["embd"][i["tokens"].long()].double()
    a = norm(cur, i["norms"]["attn_norm.0"])
    for li in range(c["layers"]):
        y = {}
        for name, w in _layer_weights(c, seed, li):
            if name == "wo":
                store(i["kv_k"], i["sc_k"], li, rope(y["wk"]))
                store(i["kv_v"], i["sc_v"], li, y["wv"].view(B, n, hd))
                a = _attend(rope(y["wq"]).reshape(B, -1), i["kv_k"][li], i["kv_v"][li], i["sc_k"][li], i["sc_v"][li], pos, heads, n, hd)
                cur = cur + _mul(a, w)
                a = norm(cur, i["norms"][f"ffn_norm.{li}"])
            elif name == "w_down":
                cur = cur + _mul(_silu_mul(y["w_gate"], y["w_up"]), w)
                a = norm(cur, i["norms"][f"attn_norm.{li + 1}" if li + 1 < c["layers"] else "output_norm"])
            else:
                y[name] = _mul(a, w)
    logits = _mul(a, _weight(seed, 99, c["vocab"], H))
    return {"logits": logits, "kv_k": None, "kv_v": None, "sc_k": i["sc_k"], "sc_v": i["sc_v"]}


def exact(case, seed):
    c, kind = case, case["kind"]
    if kind == "gemv":
        x = _acts(seed, 90, 1, c["K"]).double()
        return [_mul(x, _weight(seed, i, c["M"], c["K"], c["outliers"]))[0] for i in range(c["count"])]
    if kind == "layer":
        x = _acts(seed, 90, c["batch"], c["hidden"]).double()
        own = {"wo": _acts(seed, 91, c["batch"], c["q"]).double(), "w_down": _acts(seed, 92, c["batch"], c["ffn"]).double()}
        return {n: _mul(own.get(n, x), w) for n, w in _layer_weights(c, seed, 0)}
    if kind == "gemm":
        return _mul(_acts(seed, 90, c["batch"], c["K"]).double(), _weight(seed, 0, c["M"], c["K"]))
    if kind == "step":
        return _exact_step(c, seed)
    if kind == "attention":
        i = _attention_inputs(c, seed)
        return _attend(i["q"].double(), i["kv_k"], i["kv_v"], i["sc_k"], i["sc_v"], i["positions"], c["heads"], c["kv_heads"], c["head_dim"])
    if kind == "moe":
        x = _acts(seed, 990, c["batch"], c["hidden"]).double()
        router = torch.rand(c["batch"], c["experts"], generator=_gen(seed, 991), device="cuda").double()
        top, sel = router.topk(2, dim=1)
        share = torch.softmax(top, dim=1)
        out = torch.zeros(c["batch"], c["hidden"], device="cuda", dtype=torch.float64)
        for e in range(c["experts"]):
            t, k = (sel == e).nonzero(as_tuple=True)
            if t.numel() == 0:
                continue
            g = _mul(x[t], _weight(seed, 10 * e, c["ffn"], c["hidden"], c["outliers"]))
            u = _mul(x[t], _weight(seed, 10 * e + 1, c["ffn"], c["hidden"], c["outliers"]))
            out.index_add_(0, t, share[t, k][:, None] * _mul(_silu_mul(g, u), _weight(seed, 10 * e + 2, c["hidden"], c["ffn"], c["outliers"])))
        return out
    return None
