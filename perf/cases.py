"""Workloads of the packed-weight path as a user's program runs them, with their inputs, their least work and the
precision that a correct implementation keeps.  Weights are Laplace codes (mean absolute code about 4.4, clipped to
+-127), made on the GPU from the seed.

kind "linear"   one packed linear layer called on `rows` activation rows: the unit that a deployed model calls
kind "deploy"   a bf16 weight quantised, packed and made resident, and its first row computed
kind "decode"   the packed streams back to a bf16 weight
kind "step"     one token of a Llama-style decoder (one CUDA graph)
kind "batch"    one token of each of `rows` sequences in lock-step (one CUDA graph)
kind "verify"   `rows` tokens of one sequence in one pass (one CUDA graph): verification of a speculative draft
kind "prefill"  a prompt of `rows` tokens
kind "hybrid"   one token of the hybrid decoder: gated-delta-rule and gated-attention layers (one CUDA graph)
"""
import torch

from ixrun_b200.engine import StreamingLinear
from ixrun_b200.gpu_pack import int8x_quantize_gpu, quantize_pack_gpu
from ixrun_b200.hybrid27b import Hybrid27B, HybridConfig
from ixrun_b200.kernels import decode_weight
from ixrun_b200.llama_runner import BatchedGreedyDecoder, LlamaConfig, PackedLlama, Verifier
from ixrun_b200.p6 import set_pdl

BITS = 5.4428          # bits per weight of the packed format on this code distribution


def listed():
    return [
        # the smallest call: a projection of the 1B-class decoder for one token; launch and host time count
        {"name": "linear small", "kind": "linear", "out_f": 2048, "in_f": 2048, "rows": 1, "bias": False},
        # down_proj of the 27B-class decoder for one token: the headline layer, bound by memory
        {"name": "linear down_proj", "kind": "linear", "out_f": 5120, "in_f": 17408, "rows": 1, "bias": False},
        # gate/up of the same decoder for eight rows: a small serving batch, or a draft under verification
        {"name": "linear gate 8 rows", "kind": "linear", "out_f": 17408, "in_f": 5120, "rows": 8, "bias": False},
        # row counts and sizes that fill no tile, with a bias: a middling batch on a layer of another model
        {"name": "linear ragged 23 rows", "kind": "linear", "out_f": 5000, "in_f": 2176, "rows": 23, "bias": True},
        # the largest batch of lock-step serving on the widest layer
        {"name": "linear gate 64 rows", "kind": "linear", "out_f": 17408, "in_f": 5120, "rows": 64, "bias": False},
        # deploying one square attention projection of the 27B-class decoder
        {"name": "deploy 5120", "kind": "deploy", "out_f": 5120, "in_f": 5120, "bias": True},
        # cached mode: the single-layer codec case, streams to bf16
        {"name": "decode 4096", "kind": "decode", "out_f": 4096, "in_f": 4096},
        # the 1B-class decoder generating behind a 1024-token prompt
        _llama("1B step", "step", rows=1, context=1024),
        # the same decoder serving forty sequences
        _llama("1B batch 40", "batch", rows=40, context=300),
        # the same decoder verifying a draft of four tokens behind the last confirmed one
        _llama("1B verify 5", "verify", rows=5, context=700),
        # the same decoder reading a prompt
        _llama("1B prefill 1000", "prefill", rows=1000, context=0),
        # hybrid decoder, three recurrent layers to one attention layer, at the 4096-token context
        {"name": "hybrid step", "kind": "hybrid", "layers": 16, "hidden": 1024, "ffn": 3072, "k_heads": 4, "v_heads": 12,
         "q_heads": 6, "kv_heads": 2, "vocab": 16384, "context": 4096},
    ]


def _llama(name, kind, rows, context, layers=24, hidden=2048, ffn=6144, vocab=73448):
    c = {"kind": kind, "layers": layers, "hidden": hidden, "ffn": ffn, "vocab": vocab, "rows": rows, "context": context}
    return {"name": name, **c} if name else c


def _log(rng, lo, hi):
    """a whole number spread evenly over the logarithm of [lo, hi]"""
    return max(lo, min(hi, int(round(lo * (hi / lo) ** rng.random()))))


def draw(rng):
    kind = rng.choice(["linear"] * 6 + ["deploy", "decode", "step", "step", "batch", "batch", "verify", "prefill", "hybrid"])
    if kind in ("linear", "deploy", "decode"):
        c = {"kind": kind, "out_f": _log(rng, 300, 17408), "in_f": 32 * _log(rng, 16, 544)}
        if kind != "decode":
            c["bias"] = rng.random() < 0.3
        if kind == "linear":
            if rng.random() < 0.5:                        # half of the layers have a whole number of tiles
                c["out_f"] = (c["out_f"] + 127) // 128 * 128
                c["in_f"] = (c["in_f"] + 63) // 64 * 64
            c["rows"] = rng.choice([1, rng.randint(2, 8), rng.randint(9, 64), _log(rng, 65, 1024)])
        return c
    if kind == "hybrid":
        kv = rng.choice([1, 2])
        return {"kind": kind, "layers": 4 * rng.randint(1, 4), "hidden": 64 * rng.randint(6, 16), "ffn": 64 * rng.randint(16, 48),
                "k_heads": 4, "v_heads": rng.choice([4, 8, 12]), "q_heads": kv * rng.choice([2, 3, 4]), "kv_heads": kv,
                "vocab": rng.randint(4000, 16384), "context": _log(rng, 100, 8192)}
    hidden = 256 * rng.randint(4, 8)
    rows = {"step": 1, "batch": rng.randint(2, 64), "verify": rng.randint(2, 16), "prefill": _log(rng, 65, 1000)}[kind]
    context = {"step": _log(rng, 64, 4096), "batch": _log(rng, 64, 512), "verify": _log(rng, 64, 2048), "prefill": 0}[kind]
    return _llama(None, kind, rows, context, layers=rng.randint(4, 24), hidden=hidden,
                  ffn=min(6144, 64 * int(hidden * rng.uniform(2, 3.5) / 64)), vocab=rng.randint(8000, 73448))


# ------------------------------------------------------------------------------------------------ inputs
def _weight(gen, out_f, in_f):
    """bf16 weight whose codes are round(Laplace(0, 4.4)), the largest of them 127, scale 2^-9: the quantiles of the
    distribution in an order from the seed, so that the packed streams of a shape have the same lengths for every seed"""
    n = out_f * in_f
    u = (torch.randperm(n, generator=gen, device="cuda") + 0.5).mul_(1.0 / n).sub_(0.5)
    c = u.sign() * torch.log1p(-2.0 * u.abs()).mul_(-4.4)
    c = c.round_().clamp_(-127, 127)
    c[c.argmax()] = 127
    return (c * 2.0 ** -9).bfloat16().view(out_f, in_f)


def _llama_parameters(case, gen):
    """the parameters as a checkpoint holds them: weight of every linear (all layers alike), embedding, head, norms"""
    h, heads, ffn = case["hidden"], case["hidden"] // 128, case["ffn"]
    w = {n: _weight(gen, *s) for n, s in
         {"q_proj": (h, h), "k_proj": (heads // 2 * 128, h), "v_proj": (heads // 2 * 128, h), "o_proj": (h, h),
          "gate_proj": (ffn, h), "up_proj": (ffn, h), "down_proj": (h, ffn)}.items()}
    # a residual stream that the layers add to, as in a trained model: bf16 rounding does not pile up to the stream's own size
    embed = torch.randn(case["vocab"], h, generator=gen, device="cuda").bfloat16()
    head = (torch.randn(case["vocab"], h, generator=gen, device="cuda") * 0.02).bfloat16()
    norm = [[(1 + 0.1 * torch.randn(h, generator=gen, device="cuda")).bfloat16() for _ in range(2)]
            for _ in range(case["layers"])]
    return w, embed, head, norm


def _max_seq(case):
    return case["context"] + (case["rows"] if case["kind"] != "batch" else 0) + 256


def _batch_positions(case, gen):
    """sequences of different lengths, from half of the context to all of it"""
    return (case["context"] * (0.5 + 0.5 * torch.rand(case["rows"], generator=gen, device="cuda"))).to(torch.int32)


def _llama_model(case, gen):
    heads = case["hidden"] // 128
    cfg = LlamaConfig(n_layers=case["layers"], hidden=case["hidden"], intermediate=case["ffn"], n_heads=heads,
                      n_kv_heads=heads // 2, vocab=case["vocab"], max_seq=_max_seq(case))
    w, embed, head, norm = _llama_parameters(case, gen)
    one = {n: int8x_quantize_gpu(t) for n, t in w.items()}         # every layer gets its own device copy
    return cfg, PackedLlama(cfg, [one] * cfg.n_layers, embed, head, norms=norm)


def _fill(gen, *caches):
    for t in caches:
        t.normal_(generator=gen)


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    kind = case["kind"]
    s = {"case": case}
    if kind in ("linear", "deploy", "decode"):
        out_f, in_f = case["out_f"], case["in_f"]
        w = _weight(gen, out_f, in_f)
        bias = (torch.randn(out_f, generator=gen, device="cuda") * 0.1).bfloat16() if case.get("bias") else None
        if kind == "decode":
            s["packed"] = quantize_pack_gpu(w)
            s["out"] = torch.empty(out_f * in_f, dtype=torch.bfloat16, device="cuda")
            return s
        s["x"] = torch.randn(case.get("rows", 1), in_f, generator=gen, device="cuda").bfloat16()
        if kind == "deploy":
            s.update(w=w, bias=bias)
            return s
        s["lin"] = StreamingLinear.from_weight(w, bias=bias)
        s["lin"]._set_shared_buf(torch.empty(out_f * in_f, dtype=torch.bfloat16, device="cuda"))
        return s
    if kind == "hybrid":
        cfg = HybridConfig(n_layers=case["layers"], hidden=case["hidden"], ffn=case["ffn"], vocab=case["vocab"],
                           gdn_k_heads=case["k_heads"], gdn_v_heads=case["v_heads"], attn_heads=case["q_heads"],
                           attn_kv_heads=case["kv_heads"])
        m = Hybrid27B(cfg, 1, 0, "cuda", context=case["context"], max_new=16, seed=seed)
        m.embed.mul_(50)                                  # standard deviation 1, as above
        m.gdn_state.normal_(generator=gen).mul_(0.1)
        m.conv_state.normal_(generator=gen)
        s["model"], s["token"] = m, int(seed) % cfg.vocab
        return _captured(s, m)
    cfg, m = _llama_model(case, gen)
    ids = torch.randint(0, cfg.vocab, (case["rows"],), generator=gen, device="cuda")
    s.update(model=m, ids=ids)
    if kind == "prefill":
        s["ids"] = ids.cpu()                              # a prompt comes from the tokenizer on the host
        return s
    if kind == "batch":
        d = s["dec"] = BatchedGreedyDecoder(m, case["rows"])
        _fill(gen, d.k_cache, d.v_cache)
        s["pos"] = _batch_positions(case, gen)
        d.pos32.copy_(s["pos"])
        return _captured(s, d)
    _fill(gen, m.k_cache, m.v_cache)
    s["ver"] = Verifier(m, case["rows"]) if kind == "verify" else None
    return _captured(s, s["ver"] or m)


def _captured(s, what):
    """the decode loops capture their step once, with dependent launches, when everything is deployed"""
    torch.cuda.synchronize()
    before = set_pdl(True)
    what.capture()
    set_pdl(before)
    return s


# ------------------------------------------------------------------------------------------------ one pass
@torch.no_grad()
def run(s):
    case, kind = s["case"], s["case"]["kind"]
    if kind == "linear":
        return s["lin"](s["x"])
    if kind == "decode":
        return decode_weight(s["packed"], out=s["out"])
    if kind == "deploy":
        dp, codes = quantize_pack_gpu(s["w"], return_codes=True)
        lin = StreamingLinear(dp, bias=s["bias"])
        return [lin(s["x"]), codes, dp.scale, dp.b1, dp.b2, dp.l1, dp.l2, dp.l3]
    m = s["model"]
    if kind == "step":
        logits = m.step(s["ids"], case["context"])
        return [logits, m.k_cache[:, case["context"]], m.v_cache[:, case["context"]]]
    if kind == "verify":
        logits = s["ver"](s["ids"], case["context"])
        at = slice(case["context"], case["context"] + case["rows"])
        return [logits, m.k_cache[:, at], m.v_cache[:, at]]
    if kind == "prefill":
        logits = m.prefill(s["ids"])
        return [logits, m.k_cache[:, :case["rows"]], m.v_cache[:, :case["rows"]]]
    if kind == "batch":
        d = s["dec"]
        d.pos32.copy_(s["pos"])                           # the same positions on every pass
        return [d.step(s["ids"]), d.k_cache, d.v_cache]
    # the same token and position on every pass; the recurrent state moves on.  (The token that the model feeds back to
    # itself is not returned: it may change at a near-tie.)
    m.tok.fill_(s["token"])
    m.pos32.fill_(case["context"])
    m.n_done.zero_()
    m.step()
    return [m.h, m.xn, m.gdn_state, m.conv_state, m.k_cache[:, case["context"]], m.v_cache[:, case["context"]]]


# ------------------------------------------------------------------------------------------------ least work, precision
def work(case):
    kind = case["kind"]
    if kind in ("linear", "deploy", "decode"):
        n, rows = case["out_f"] * case["in_f"], case.get("rows", 1)
        if kind == "decode":
            return {"bytes": n * (BITS / 8 + 2), "flops": n}
        act = 2 * rows * (case["out_f"] + case["in_f"])
        if kind == "deploy":                              # weight in; codes, streams and the layer's own copy out
            return {"bytes": n * (2 + 1 + 2 * BITS / 8) + act, "flops": 4 * n}
        return {"bytes": n * BITS / 8 + act, "flops": 2 * rows * n}
    if kind == "hybrid":
        h, d, da = case["hidden"], 128, 256
        gdn = h * d * (2 * case["k_heads"] + 2 * case["v_heads"]) + 2 * case["v_heads"] * h + h * d * case["v_heads"]
        att = h * da * (3 * case["q_heads"] + 2 * case["kv_heads"])
        n_att = case["layers"] // 4
        n = case["layers"] * 3 * h * case["ffn"] + (case["layers"] - n_att) * gdn + n_att * att
        head = case["vocab"] * h
        state = (case["layers"] - n_att) * case["v_heads"] * d * d
        kv = n_att * 2 * case["kv_heads"] * da * case["context"]
        return {"bytes": n * BITS / 8 + 2 * head + 8 * state + 2 * kv,
                "flops": 2 * (n + head) + 8 * state + 2 * kv * case["q_heads"] // case["kv_heads"]}
    h, rows, heads = case["hidden"], case["rows"], case["hidden"] // 128
    kv_heads = heads // 2
    n = case["layers"] * (h * 128 * (2 * heads + 2 * kv_heads) + 3 * h * case["ffn"])
    head = case["vocab"] * h
    row_ctx = {"step": case["context"] + 1, "verify": case["context"] + rows, "batch": 0.75 * case["context"], "prefill": rows / 2}[kind]
    seqs = rows if kind == "batch" else 1                 # caches that are read
    kv = case["layers"] * 2 * kv_heads * 128 * (rows if kind == "prefill" else row_ctx * seqs)
    out_rows = 1 if kind == "prefill" else rows
    return {"bytes": n * BITS / 8 + 2 * head + 2 * kv + 4 * out_rows * case["vocab"],
            "flops": 2 * rows * n + 2 * out_rows * head + 4 * case["layers"] * heads * 128 * row_ctx * rows}


def tolerance(case):
    kind = case["kind"]
    if kind == "decode":
        return "exact"
    if kind in ("linear", "deploy"):
        # a bf16 number on either side of a rounding boundary: against 64-bit sums rel 4e-5 and max 0.0075 (one unit in the
        # last place) without a bias; a bias added before or after the rounding differs by rel 6e-4
        return {"rel": 2e-3, "max": 0.03, "differ": 0.0}
    # bf16 activations through all layers: against the same weights in dense matmuls with eager glue rel 0.0084 and max 0.039
    return {"rel": 0.03, "max": 0.15}


# ------------------------------------------------------------------------------------------------ the same in 64 bits
def _codes(w):
    """the quantiser's int8 codes and bf16 scale of a bf16 weight"""
    scale = (w.abs().max().clamp_min(1e-8) / 127.0).bfloat16()
    return (w.float() / scale.float()).round().clamp(-127, 127), scale


def _dequantised(w):
    codes, scale = _codes(w)
    return (codes * scale.float()).bfloat16().double()             # the bf16 weight that the format stands for


@torch.no_grad()
def exact(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    kind = case["kind"]
    if kind in ("linear", "deploy", "decode"):
        out_f, in_f = case["out_f"], case["in_f"]
        w = _weight(gen, out_f, in_f)
        bias = (torch.randn(out_f, generator=gen, device="cuda") * 0.1).bfloat16() if case.get("bias") else None
        if kind == "decode":
            return _dequantised(w)
        x = torch.randn(case.get("rows", 1), in_f, generator=gen, device="cuda").bfloat16()
        y = x.double() @ _dequantised(w).t()
        if bias is not None:
            y = y + bias.double()
        if kind == "linear":
            return y
        codes, scale = _codes(w)
        return [y, codes.to(torch.int8), scale] + [None] * 5
    if kind == "hybrid":
        return None                                                # its weights are drawn inside the model
    return _exact_llama(case, gen)


def _exact_llama(case, gen):
    """the decoder on the dequantised weights, every activation in 64 bits"""
    kind, rows, hidden, d = case["kind"], case["rows"], case["hidden"], 128
    heads, layers = hidden // d, case["layers"]
    kvh, max_seq = heads // 2, _max_seq(case)
    w, embed, head, norm = _llama_parameters(case, gen)
    w = {n: _dequantised(t) for n, t in w.items()}
    ids = torch.randint(0, case["vocab"], (rows,), generator=gen, device="cuda")
    seqs = rows if kind == "batch" else 1
    kc = torch.zeros(layers, seqs, max_seq, kvh, d, dtype=torch.bfloat16, device="cuda")
    vc = torch.zeros_like(kc)
    if kind != "prefill":
        _fill(gen, kc, vc)
    if kind == "batch":
        pos = _batch_positions(case, gen).long()
        seq = torch.arange(rows, device="cuda")
    else:
        pos = case["context"] + torch.arange(rows, device="cuda")
        seq = torch.zeros(rows, dtype=torch.long, device="cuda")
    half = d // 2
    ang = pos[:, None].double() / 10000.0 ** (torch.arange(half, device="cuda").double() / half)
    cos, sin = ang.cos()[:, None, :], ang.sin()[:, None, :]

    def rope(t):
        a, b = t[..., :half], t[..., half:]
        return torch.cat([a * cos - b * sin, b * cos + a * sin], dim=-1)

    def rms(t, g):
        return t * torch.rsqrt(t.pow(2).mean(-1, keepdim=True) + 1e-5) * g

    h = embed[ids].double()
    ks, vs = [], []
    n_ctx = int(pos.max().item()) + 1
    mask = torch.arange(n_ctx, device="cuda")[None, :] <= pos[:, None]             # [rows, n_ctx]
    for li in range(layers):
        x = rms(h, norm[li][0].double())
        q = rope((x @ w["q_proj"].t()).view(rows, heads, d))
        k = rope((x @ w["k_proj"].t()).view(rows, kvh, d))
        v = (x @ w["v_proj"].t()).view(rows, kvh, d)
        kk, vv = kc[li].double(), vc[li].double()
        kk[seq, pos], vv[seq, pos] = k, v
        ks.append(kk if kind == "batch" else k)
        vs.append(vv if kind == "batch" else v)
        qg = q.view(rows, kvh, 2, d)
        if kind == "batch":
            s = torch.einsum("rghd,rsgd->rghs", qg, kk[:, :n_ctx])
        else:
            s = torch.einsum("rghd,sgd->rghs", qg, kk[0, :n_ctx])
        p = (s * d ** -0.5).masked_fill(~mask[:, None, None, :], -torch.inf).softmax(-1)
        a = torch.einsum("rghs,rsgd->rghd", p, vv[:, :n_ctx]) if kind == "batch" else torch.einsum("rghs,sgd->rghd", p, vv[0, :n_ctx])
        h = h + a.reshape(rows, hidden) @ w["o_proj"].t()
        x = rms(h, norm[li][1].double())
        g = x @ w["gate_proj"].t()
        h = h + (g * torch.sigmoid(g) * (x @ w["up_proj"].t())) @ w["down_proj"].t()
    h = rms(h[-1:] if kind == "prefill" else h, 1.0)
    return [h @ head.double().t(), torch.stack(ks), torch.stack(vs)]
