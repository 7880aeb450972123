"""Work that a user of this framework has a GPU do, as timed cases: sparse attention decode, the low-latency MoE layer,
low-latency and normal-mode dispatch / combine, the grouped expert GEMMs, the tensor-parallel GEMMs and the small fused
kernels of a decoder layer. Every case goes through the public entry points, on one GPU (a group of one rank).

The sizes are those of the framework's serving configuration (hidden 7168, 256 experts of width 2048, top-8, 128
attention heads over 576-wide latent rows, 2048 selected keys) and of its Llama-style tensor-parallel MLP (hidden 8192,
7168 gate/up and 3584 down features per rank), and the ranges around them.
"""
import math
import weakref

import torch

from umdk_b200.buffer import Buffer
from umdk_b200.ops import glue, moe_gemm
from umdk_b200.ops.attention import DIM, DIM_V, HEADS, PAGE, sparse_mla_decode
from umdk_b200.ops.ep_ll import EpLowLatency, ExpertWeights
from umdk_b200.ops.tp import TpComm
from umdk_b200.parallel.symm import SymmetricHeap

BF16, F8 = torch.bfloat16, torch.float8_e4m3fn


def listed():
    return [
        # one sequence being decoded: latency of a single user's attention call
        {"name": "mla_single", "kind": "mla", "batch": 1, "ctx": 32768, "topk": 2048, "ragged": False},
        # the serving benchmark's attention call: 64 sequences, 2048 of 32768 keys each
        {"name": "mla_serving", "kind": "mla", "batch": 64, "ctx": 32768, "topk": 2048, "ragged": False},
        # a half-full batch with short, uneven histories: unused entries and positions past the sequence's end
        {"name": "mla_ragged", "kind": "mla", "batch": 23, "ctx": 4096, "topk": 1000, "ragged": True},
        # one rank's share (32 experts) of the serving benchmark's MoE layer, shared expert folded in
        {"name": "moe_serving", "kind": "moe", "tokens": 128, "experts": 32, "topk": 8, "hidden": 7168, "ffn": 2048,
         "fold": True},
        # the same layer for a handful of sequences: only some experts are hit, latency counts
        {"name": "moe_few_tokens", "kind": "moe", "tokens": 3, "experts": 32, "topk": 8, "hidden": 7168, "ffn": 2048,
         "fold": False},
        # decode exchange for callers with their own expert code: low-latency dispatch, then combine
        {"name": "ll_exchange", "kind": "ll", "tokens": 128, "experts": 256, "topk": 8, "hidden": 7168, "drop": 0.0},
        # prefill exchange of the normal-mode benchmark: fp8 rows out, bf16 rows back
        {"name": "ep_prefill_fp8", "kind": "ep", "tokens": 4096, "experts": 256, "topk": 8, "hidden": 7168,
         "fp8": True, "drop": 0.0},
        # a ragged prefill chunk without quantisation, some routing slots dropped
        {"name": "ep_chunk_bf16", "kind": "ep", "tokens": 1003, "experts": 64, "topk": 6, "hidden": 4096,
         "fp8": False, "drop": 0.1},
        # expert FFN of a prefill batch: 16384 rows spread unevenly over 32 experts
        {"name": "ffn_prefill", "kind": "ffn", "rows": 16384, "experts": 32, "hidden": 7168, "ffn": 2048},
        # expert FFN of a decode batch through the separate GEMM calls
        {"name": "ffn_decode", "kind": "ffn", "rows": 1024, "experts": 32, "hidden": 7168, "ffn": 2048},
        # tensor-parallel MLP: all-gather -> GEMM (gate/up) and GEMM -> reduce-scatter (down)
        {"name": "tp_mlp", "kind": "tp", "tokens": 8192, "hidden": 8192, "up": 7168, "down": 3584},
        # the small fused kernels of one decoder layer around the GEMMs, for 64 sequences
        {"name": "decoder_glue", "kind": "glue", "batch": 64, "hidden": 7168, "q_lora": 1536, "experts": 256,
         "topk": 8},
    ]


def _log(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(("mla", "mla", "moe", "ll", "ep", "ffn", "tp", "glue"))
    if kind == "mla":
        batch = _log(rng, 1, 128)
        topk = min(_log(rng, 64, 4096), 131072 // batch)
        ctx = PAGE * _log(rng, 16, min(512, 32768 // batch))
        return {"kind": kind, "batch": batch, "ctx": ctx, "topk": min(topk, ctx), "ragged": rng.random() < 0.5}
    hidden = 128 * _log(rng, 8, 56)
    if kind == "moe":
        return {"kind": kind, "tokens": _log(rng, 1, 128), "experts": rng.choice((8, 16, 24, 32)),
                "topk": rng.randint(1, 8), "hidden": hidden, "ffn": 128 * _log(rng, 2, 16),
                "fold": rng.random() < 0.5}
    if kind == "ll":
        return {"kind": kind, "tokens": _log(rng, 1, 256), "experts": rng.choice((16, 64, 160, 256)),
                "topk": rng.randint(1, 8), "hidden": hidden, "drop": rng.choice((0.0, 0.2))}
    if kind == "ep":
        return {"kind": kind, "tokens": _log(rng, 16, 4096), "experts": rng.choice((16, 64, 160, 256)),
                "topk": rng.randint(1, 8), "hidden": hidden, "fp8": rng.random() < 0.6,
                "drop": rng.choice((0.0, 0.2))}
    if kind == "ffn":
        return {"kind": kind, "rows": _log(rng, 64, 16384), "experts": rng.choice((4, 8, 16, 32)), "hidden": hidden,
                "ffn": 128 * _log(rng, 2, 16)}
    if kind == "tp":
        return {"kind": kind, "tokens": 128 * _log(rng, 2, 64), "hidden": 256 * _log(rng, 8, 32),
                "up": 256 * _log(rng, 4, 28), "down": 64 * _log(rng, 16, 56)}
    return {"kind": kind, "batch": _log(rng, 1, 256), "hidden": hidden, "q_lora": 128 * _log(rng, 2, 12),
            "experts": rng.choice((16, 64, 160, 256)), "topk": rng.randint(1, 8)}


# ---- inputs (the same for prepare and exact) ---------------------------------------------------------------------
class State(dict):
    """What a program keeps between calls. Communication heaps are given back when the state goes."""


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _randn(g, *shape, scale=1.0):
    return (torch.randn(*shape, device="cuda", generator=g) * scale).to(BF16)


def _routing(g, tokens, experts, topk, drop=0.0):
    """Top-k of the softmax of normal gate logits, weights renormalised; `drop` of the slots are unused (-1)."""
    p = torch.softmax(torch.randn(tokens, experts, device="cuda", generator=g), dim=-1)
    w, idx = torch.topk(p, topk, dim=-1)
    w = (w / w.sum(-1, keepdim=True)).float().contiguous()
    out = torch.randperm(tokens * topk, device="cuda", generator=g)[:int(drop * tokens * topk)]
    idx = idx.contiguous()
    idx.view(-1)[out] = -1
    return idx, w


def _quant_weights(g, n, rows, cols):
    """n matrices N(0, 0.02) in e4m3 with one fp32 scale per 128 x 128 block."""
    q = torch.empty(n, rows, cols, dtype=F8, device="cuda")
    s = torch.empty(n, rows // 128, cols // 128, device="cuda")
    for i in range(n):
        w = (torch.randn(rows, cols, device="cuda", generator=g) * 0.02).view(rows // 128, 128, cols // 128, 128)
        amax = w.abs().amax(dim=(1, 3)).clamp_min(1e-4)
        q[i] = (w * (448.0 / amax)[:, None, :, None]).view(rows, cols).to(F8)
        s[i] = amax / 448.0
    return q, s


def _quant_rows(x):
    """e4m3 codes and fp32 scales per 1 x 128 block, as the dispatch makes them."""
    b = x.float().view(x.shape[0], -1, 128)
    amax = b.abs().amax(-1).clamp_min(1e-4)
    return (b * (448.0 / amax)[..., None]).view(x.shape).to(F8), (amax / 448.0).contiguous()


def _experts(g, n, hidden, ffn):
    w1q, w1s = _quant_weights(g, n, 2 * ffn, hidden)
    w2q, w2s = _quant_weights(g, n, hidden, ffn)
    return ExpertWeights(w1q, w1s, w2q, w2s)


def _mla_inputs(c, seed):
    g = _gen(seed)
    b, pages = c["batch"], c["ctx"] // PAGE
    kv = torch.empty(b * pages, PAGE, DIM, dtype=BF16, device="cuda")
    for i in range(0, b * pages, 4096):
        kv[i:i + 4096] = torch.randn(kv[i:i + 4096].shape, device="cuda", generator=g) * 0.5
    table = torch.randperm(b * pages, device="cuda", generator=g).to(torch.int32).view(b, pages).contiguous()
    q = _randn(g, b, HEADS, DIM, scale=0.5)
    idx = torch.stack([torch.randperm(c["ctx"], device="cuda", generator=g)[:c["topk"]] for _ in range(b)])
    lens = None
    if c["ragged"]:
        idx = torch.where(torch.rand(idx.shape, device="cuda", generator=g) < 0.05, torch.full_like(idx, -1), idx)
        lens = torch.randint(c["ctx"] // 2, c["ctx"] + 1, (b,), device="cuda", generator=g).to(torch.int32)
    return {"q": q, "kv": kv, "table": table, "idx": idx.to(torch.int32).contiguous(), "lens": lens,
            "scale": DIM ** -0.5}


def _moe_inputs(c, seed):
    g = _gen(seed)
    x = _randn(g, c["tokens"], c["hidden"])
    idx, w = _routing(g, c["tokens"], c["experts"], min(c["topk"], c["experts"]))
    experts = _experts(g, c["experts"], c["hidden"], c["ffn"])
    shared = _experts(g, 1, c["hidden"], c["ffn"]) if c["fold"] else None
    return x, idx, w, experts, shared


def _exchange_inputs(c, seed):
    """Tokens, routing and expert outputs in the order in which the dispatch delivers the rows."""
    g = _gen(seed)
    x = _randn(g, c["tokens"], c["hidden"])
    idx, w = _routing(g, c["tokens"], c["experts"], c["topk"], c["drop"])
    rows = int((idx >= 0).sum())
    return x, idx, w, rows, _randn(g, rows, c["hidden"])


def _ffn_inputs(c, seed):
    g = _gen(seed)
    xq, xs = _quant_rows(_randn(g, c["rows"], c["hidden"]))
    w = _experts(g, c["experts"], c["hidden"], c["ffn"])
    share = torch.softmax(0.4 * torch.randn(c["experts"], device="cuda", generator=g), 0)
    pick = torch.multinomial(share, c["rows"], replacement=True, generator=g)
    off = torch.zeros(c["experts"] + 1, dtype=torch.int32, device="cuda")
    off[1:] = torch.bincount(pick, minlength=c["experts"]).cumsum(0)
    return xq, xs, off, w


def _tp_inputs(c, seed):
    g = _gen(seed)
    t, h = c["tokens"], c["hidden"]
    return (_randn(g, t, h), _randn(g, c["up"], h, scale=0.02), _randn(g, t, c["down"]),
            _randn(g, h, c["down"], scale=0.02))


def _glue_inputs(c, seed):
    g = _gen(seed)
    b, h = c["batch"], c["hidden"]
    freq = 1.0 / (10000.0 ** (torch.arange(0, 64, 2, device="cuda").float() / 64))
    pos = torch.randint(1, 32768, (1,), device="cuda", generator=g).float()
    return {"x": _randn(g, b, h), "a": _randn(g, b, h), "b": _randn(g, b, h), "norm": _randn(g, h) * 0.1 + 1,
            "qkv": _randn(g, b, c["q_lora"] + DIM), "q_norm": _randn(g, c["q_lora"]) * 0.1 + 1,
            "kv_norm": _randn(g, DIM_V) * 0.1 + 1, "cos": torch.cos(pos * freq), "sin": torch.sin(pos * freq),
            "pool": _randn(g, b, PAGE, DIM), "row": torch.arange(b, device="cuda") * PAGE + 5,
            "q": _randn(g, b, HEADS, 192), "q_full": _randn(g, b, HEADS, DIM),
            "logits": _randn(g, b, c["experts"])}


# ---- the cases ---------------------------------------------------------------------------------------------------
def prepare(case, seed):
    c, s = case, State(kind=case["kind"], case=case)
    if c["kind"] == "mla":
        s.update(_mla_inputs(c, seed))
        s["status"] = torch.zeros(4, dtype=torch.int32, device="cuda")
    elif c["kind"] == "moe":
        s["x"], s["idx"], s["w"], experts, shared = _moe_inputs(c, seed)
        k = s["idx"].shape[1]
        if c["fold"]:
            need = EpLowLatency.heap_bytes(1, c["experts"], k, c["hidden"], c["tokens"], fold_shared=True)
            heap = SymmetricHeap(need)
            s["ep"] = EpLowLatency(heap, c["experts"], k, c["hidden"], c["ffn"], c["tokens"], fold_shared=True)
            s["experts"] = ExpertWeights.with_shared(experts, shared).to_tiled()
            s["idx"], s["w"] = s["ep"].fold_routing(s["idx"], s["w"])
            weakref.finalize(s, heap.close)
        else:
            s["buf"], s["experts"] = Buffer(max_tokens_per_rank=c["tokens"]), experts
            weakref.finalize(s, s["buf"].destroy)
        run(s)   # a program runs the layer once before it serves: buffers, kernel attributes
    elif c["kind"] in ("ll", "ep"):
        s["x"], s["idx"], s["w"], s["rows"], y = _exchange_inputs(c, seed)
        s["buf"] = Buffer(num_experts=c["experts"], max_tokens_per_rank=c["tokens"])
        s["y"] = y
        weakref.finalize(s, s["buf"].destroy)
    elif c["kind"] == "ffn":
        s["xq"], s["xs"], s["off"], s["w"] = _ffn_inputs(c, seed)
        n = c["rows"]
        s["hq"] = torch.empty(n, c["ffn"], dtype=F8, device="cuda")
        s["hs"] = torch.empty(n, c["ffn"] // 128, device="cuda")
        s["y"] = torch.empty(n, c["hidden"], dtype=BF16, device="cuda")
        s["status"] = torch.zeros(4, dtype=torch.int32, device="cuda")
    elif c["kind"] == "tp":
        s["x"], s["w_up"], s["h"], s["w_down"] = _tp_inputs(c, seed)
        heap = SymmetricHeap(TpComm.heap_bytes(1, c["tokens"], c["hidden"], c["hidden"]))
        s["tp"] = TpComm(heap, c["tokens"], c["hidden"], c["hidden"])
        weakref.finalize(s, heap.close)
    else:
        s.update(_glue_inputs(c, seed))
        s["status"] = torch.zeros(4, dtype=torch.int32, device="cuda")
    return s


def run(s):
    c = s["case"]
    if s["kind"] == "mla":
        return sparse_mla_decode(s["q"], s["kv"], s["table"], s["idx"], s["scale"], seq_lens=s["lens"],
                                 status=s["status"])
    if s["kind"] == "moe":
        if c["fold"]:
            return s["ep"].moe(s["x"], s["idx"], s["w"], s["experts"], prefolded=True)
        return s["buf"].fused_moe(s["x"], s["idx"], s["w"], s["experts"])
    if s["kind"] == "ll":
        (rx, rs), counts, h, _, _ = s["buf"].low_latency_dispatch(s["x"], s["idx"], c["tokens"], c["experts"])
        out, _, _ = s["buf"].low_latency_combine(s["y"], s["idx"], s["w"], h)
        rx, rs = rx[:s["rows"]], rs[:s["rows"]]
        rx.owner = rs.owner = s   # views of the heap: it stays as long as they do
        return rx, rs, counts, out
    if s["kind"] == "ep":
        rx, experts, weights, _, h, _ = s["buf"].dispatch(s["x"], topk_idx=s["idx"], topk_weights=s["w"],
                                                          use_fp8=c["fp8"])
        out, _, _ = s["buf"].combine(s["y"], h)
        return rx, experts, weights, out
    if s["kind"] == "ffn":
        w = s["w"]
        hq, hs = moe_gemm.gemm1_swiglu_quant(s["xq"], s["xs"], s["off"], w.w1q, w.w1s, s["status"], s["hq"], s["hs"])
        return hq, hs, moe_gemm.gemm2(hq, hs, s["off"], w.w2q, w.w2s, s["status"], s["y"])
    if s["kind"] == "tp":
        return s["tp"].ag_gemm(s["x"], s["w_up"]), s["tp"].gemm_rs(s["h"], s["w_down"])
    x, h = glue.add_rmsnorm(s["x"], s["norm"], s["a"], s["b"])
    qa = glue.qkv_post(s["qkv"], c["q_lora"], s["q_norm"], s["kv_norm"], s["cos"], s["sin"], s["pool"], s["row"],
                       s["status"])
    glue.q_rope(s["q"], 128, s["cos"], s["sin"], s["q_full"])
    idx, w = glue.router_topk(s["logits"], c["topk"])
    return x, h, qa, s["pool"], s["q_full"], idx, w


def work(case):
    c = case
    if c["kind"] == "mla":
        n = c["batch"] * c["topk"] * (0.7 if c["ragged"] else 1.0)
        return {"bytes": n * DIM * 2 + c["batch"] * HEADS * (DIM + DIM_V) * 2, "flops": 2.0 * n * HEADS * (DIM + DIM_V)}
    if c["kind"] == "glue":
        b = c["batch"]
        return {"bytes": b * 2.0 * (5 * c["hidden"] + 2 * (c["q_lora"] + DIM) + 2 * HEADS * 64 + c["experts"])
                + b * c["topk"] * 12.0, "flops": 0}
    if c["kind"] == "tp":
        t, h = c["tokens"], c["hidden"]
        return {"bytes": 2.0 * (t * h + c["up"] * h + t * c["up"] + t * c["down"] + h * c["down"] + t * h),
                "flops": 2.0 * t * h * (c["up"] + c["down"])}
    h = c["hidden"]
    if c["kind"] == "ffn":
        r, f, e = c["rows"], c["ffn"], c["experts"]
        return {"bytes": e * 3.0 * f * h + r * (h * 1.03 + f * 1.03 + 2.0 * h), "flops": 2.0 * r * 3 * f * h}
    t = c["tokens"]
    if c["kind"] == "moe":
        k, e, f = min(c["topk"], c["experts"]), c["experts"], c["ffn"]
        hit = e * (1 - (1 - k / e) ** t) + (1 if c["fold"] else 0)
        rows = t * (k + (1 if c["fold"] else 0))
        return {"bytes": hit * 3.0 * f * h + 4.0 * t * h, "flops": 2.0 * rows * 3 * f * h}
    rows = t * c["topk"] - int(c["drop"] * t * c["topk"])
    row = h * 1.03 if c.get("fp8", True) else 2.0 * h
    return {"bytes": t * h * 2.0 + rows * row + rows * h * 2.0 + t * h * 2.0, "flops": 0}


def tolerance(case):
    # Measured against `exact` (64-bit sums): the rounding of bf16 results alone is 1.7e-3. Where fp8 codes are made
    # from 32-bit sums, a sum in another order moves some codes to their neighbours.
    return {"rel": {"mla": 8e-3, "moe": 1.5e-2, "ll": 5e-3, "ep": 5e-3, "ffn": 1.5e-2, "tp": 5e-3, "glue": 8e-3}[
        case["kind"]]}


# ---- the same results in 64 bits ---------------------------------------------------------------------------------
def _f64_weight(q, s):
    return (q.double().view(q.shape[0] // 128, 128, -1, 128) * s.double()[:, None, :, None]).view(q.shape)


def _f64_quant(x):
    """(codes rounded to e4m3, scales) of 64-bit rows."""
    b = x.view(x.shape[0], -1, 128)
    amax = b.abs().amax(-1).clamp_min(1e-4)
    return (b * (448.0 / amax)[..., None]).float().to(F8).double().view(x.shape), amax / 448.0


def _f64_rows(q, s):
    return (q.view(q.shape[0], -1, 128) * s[..., None]).view(q.shape)


def _f64_ffn(x, w, e):
    y = x @ _f64_weight(w.w1q[e], w.w1s[e]).t()
    f = y.shape[1] // 2
    hq, hs = _f64_quant(torch.nn.functional.silu(y[:, :f]) * y[:, f:])
    return hq, hs, _f64_rows(hq, hs) @ _f64_weight(w.w2q[e], w.w2s[e]).t()


def _f64_rms(x, w):
    return x * torch.rsqrt((x * x).mean(-1, keepdim=True) + glue.RMS_EPS) * w.double()


def _f64_rope(x, cos, sin):
    a, b = x[..., 0::2], x[..., 1::2]
    return torch.stack((a * cos.double() - b * sin.double(), a * sin.double() + b * cos.double()), -1).flatten(-2)


def _row_order(idx, experts):
    """(token, slot) of every delivered row: by expert, then by token."""
    t, k = torch.nonzero(idx >= 0, as_tuple=True)
    order = torch.argsort(idx[t, k], stable=True)
    return t[order], k[order]


def exact(case, seed):
    c = case
    if c["kind"] == "mla":
        s = _mla_inputs(c, seed)
        outs, lses = [], []
        for b in range(c["batch"]):
            pos = s["idx"][b].long()
            pos = pos[(pos >= 0) & (pos < int(s["lens"][b]))] if s["lens"] is not None else pos[pos >= 0]
            k = s["kv"].view(-1, DIM)[s["table"][b].long()[pos // PAGE] * PAGE + pos % PAGE].double()
            sc = s["q"][b].double() @ k.t() * s["scale"]
            lses.append(torch.logsumexp(sc, -1))
            outs.append(torch.softmax(sc, -1) @ k[:, :DIM_V])
        return torch.stack(outs), torch.stack(lses)
    if c["kind"] == "moe":
        x, idx, w, experts, shared = _moe_inputs(c, seed)
        xd = _f64_rows(*_f64_quant(x.double()))
        out = torch.zeros(x.shape, dtype=torch.float64, device="cuda")
        for e in range(c["experts"]):
            t, k = torch.nonzero(idx == e, as_tuple=True)
            if t.numel():
                out.index_add_(0, t, _f64_ffn(xd[t], experts, e)[2] * w[t, k].double()[:, None])
        return out, (_f64_ffn(xd, shared, 0)[2] if c["fold"] else None), None
    if c["kind"] in ("ll", "ep"):
        x, idx, w, rows, y = _exchange_inputs(c, seed)
        t, k = _row_order(idx, c["experts"])
        out = torch.zeros(x.shape, dtype=torch.float64, device="cuda")
        out.index_add_(0, t, y[:rows].double() * w[t, k].double()[:, None])
        if c["kind"] == "ll" or c["fp8"]:
            q, sc = _f64_quant(x.double())
            rx = (q[t], sc[t])
        else:
            rx = x.double()[t]
        return (rx[0], rx[1], None, out) if c["kind"] == "ll" else (rx, None, w[t, k].double(), out)
    if c["kind"] == "ffn":
        xq, xs, off, w = _ffn_inputs(c, seed)
        xd, off = _f64_rows(xq.double(), xs.double()), off.tolist()
        parts = [_f64_ffn(xd[a:b], w, e) for e, (a, b) in enumerate(zip(off, off[1:])) if b > a]
        return tuple(torch.cat(p) for p in zip(*parts))
    if c["kind"] == "tp":
        x, wu, h, wd = _tp_inputs(c, seed)
        return tuple(torch.cat([p.double() @ w.double().t() for p in a.split(2048)]) for a, w in ((x, wu), (h, wd)))
    s = _glue_inputs(c, seed)
    x = s["x"].double() + s["a"].double() + s["b"].double()
    ql = c["q_lora"]
    qkv, pool, q_full = s["qkv"].double(), s["pool"].double().view(-1, DIM), s["q_full"].double()
    pool[s["row"]] = torch.cat((_f64_rms(qkv[:, ql:ql + DIM_V], s["kv_norm"]),
                                _f64_rope(qkv[:, ql + DIM_V:], s["cos"], s["sin"])), -1)
    q_full[..., DIM_V:] = _f64_rope(s["q"].double()[..., 128:], s["cos"], s["sin"])
    w = torch.topk(torch.softmax(s["logits"].double(), -1), c["topk"], dim=-1).values
    return (x, _f64_rms(x, s["norm"]), _f64_rms(qkv[:, :ql], s["q_norm"]), pool.view(s["pool"].shape), q_full, None,
            w / w.sum(-1, keepdim=True))
