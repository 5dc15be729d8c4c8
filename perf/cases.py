"""Performance cases of the EXL3 path: what a serving program has this library do, through the public
Python entry points (LinearEXL3, Sliced / Multi bundles, DecodeGraph, moe_coop, moe_prep + moe_fused).

Kinds of case:
  linear       one LinearEXL3.forward call, from one decode row to a prefill chunk
  layer        the seven linears of a decoder layer as a model issues them: q|k|v as one sliced bundle,
               o, gate|up as one stacked bundle, down
  step         a whole greedy decode step (residual norms, linears, gated activation, lm_head) replayed
               as one CUDA graph
  moe          one fused decode MoE layer (routing on the device)
  moe_prefill  the expert layer of a prefill chunk: routing dispatch (moe_prep), then moe_fused

Weights are uniform random trellis words (every bit pattern is a valid stream and packed weights look
like noise), sign vectors on the input side, sign vectors with a per-layer scale on the output side;
activations are N(0, 1); routing comes from the top-k of random router logits."""
import math

import torch

import ampstein_b200 as amp
from ampstein_b200.models import DecodeGraph, LinearEXL3, Multi, Sliced

DEV = "cuda:0"
EPS = 1e-5
CODEBOOKS = ("plain", "mcg", "mul1")


def listed():
    return [
        # the smallest everyday call: the k or v projection of one decoded token, called eagerly
        dict(name="linear_kv_m1", kind="linear", m=1, k=4096, n=1024, bits=5, cb="mcg", dtype="f16", out="f16"),
        # three rows of logits (two drafted tokens verified together), fp32 as a sampler takes them
        dict(name="linear_head_m3", kind="linear", m=3, k=4096, n=128256, bits=6, cb="mcg", dtype="f16", out="f32"),
        # one decoded token on a mul1 checkpoint (the int8-activation form by default)
        dict(name="linear_mul1_m1", kind="linear", m=1, k=14336, n=4096, bits=4, cb="mul1", dtype="f16", out="f16"),
        # one decoded token on a checkpoint with a half-integer bitrate
        dict(name="linear_half_m1", kind="linear", m=1, k=4096, n=14336, bits=3.5, cb="mul1", dtype="f16", out="f16"),
        # eight sequences decoded together on the wide stack
        dict(name="linear_up_m8", kind="linear", m=8, k=5120, n=25600, bits=5, cb="plain", dtype="f16", out="f16"),
        # a short prompt, ragged
        dict(name="linear_o_m77", kind="linear", m=77, k=4096, n=4096, bits=4, cb="mcg", dtype="f16", out="f16"),
        # a layer over a medium prompt with an odd number of tokens
        dict(name="layer_m333", kind="layer", m=333, hidden=4096, kv=1024, ffn=14336, bits_attn=4, bits_gu=4, bits_down=4,
             cb="plain", dtype="f16"),
        # a layer over a full prefill chunk, bf16 activations, mixed bit widths
        dict(name="layer_m2048_bf16", kind="layer", m=2048, hidden=4096, kv=1024, ffn=14336, bits_attn=5, bits_gu=3, bits_down=4,
             cb="plain", dtype="bf16"),
        # one decoded token through 128 experts
        dict(name="moe_t1", kind="moe", t=1, experts=128, topk=8, hidden=2048, inter=768, bits=3, cb="plain"),
        # a batch of thirteen sequences through the same experts
        dict(name="moe_t13", kind="moe", t=13, experts=128, topk=8, hidden=2048, inter=768, bits=3, cb="plain"),
        # the experts over a prefill chunk
        dict(name="moe_prefill_t1500", kind="moe_prefill", t=1500, experts=128, topk=8, hidden=2048, inter=768, bits=3, cb="mul1"),
        # the decode step of the 32-layer stack, one token
        dict(name="step_m1", kind="step", m=1, layers=32, hidden=4096, kv=1024, ffn=14336, vocab=128256, bits=4, bits_head=6, cb="plain"),
    ]


def _log(rng, lo, hi, unit=1):
    """Log-uniform multiple of `unit` in [lo, hi]."""
    v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return min(hi // unit * unit, max(-(-lo // unit) * unit, int(round(v / unit)) * unit))


def draw(rng):
    kind = rng.choice(("linear", "linear", "linear", "rows", "rows", "layer", "layer", "moe", "moe_prefill", "step"))
    cb = rng.choice(CODEBOOKS)
    bits = rng.choice((2, 3, 3, 4, 4, 4, 5, 6, 8))
    if kind in ("linear", "rows"):
        k = _log(rng, 1024, 25600, 128)
        n = _log(rng, 512, 28672, 128)
        if kind == "linear":
            m = rng.choice((1, 1, 1, rng.randint(2, 4), rng.randint(5, 16)))
            if rng.random() < 0.15:
                k, n = rng.choice((2048, 4096)), _log(rng, 32768, 128256, 128)
            elif cb == "mul1" and rng.random() < 0.4:
                bits = rng.choice((1.5, 2.5, 3.5))
            dtype = "f16"
        else:
            m = _log(rng, 17, max(17, min(2048, int(4e11 / (k * n)))))
            dtype = rng.choice(("f16", "f16", "bf16"))
        # exl3_gemm_recon returns fp16 only; an fp32 result is asked for at decode sizes
        out = rng.choice(("f16", "f16", "f32")) if m <= 16 else "f16"
        return dict(kind="linear", m=m, k=k, n=n, bits=bits, cb=cb, dtype=dtype, out=out)
    hidden = rng.choice((2048, 2560, 3072, 4096, 5120))
    if kind == "layer":
        return dict(kind="layer", m=_log(rng, 17, 1500), hidden=hidden, kv=rng.choice((512, 1024)), ffn=_log(rng, 2 * hidden, 3 * hidden, 256),
                    bits_attn=bits, bits_gu=rng.choice((2, 3, 4)), bits_down=rng.choice((3, 4, 5)), cb=cb, dtype=rng.choice(("f16", "bf16")))
    if kind == "step":
        return dict(kind="step", m=rng.choice((1, 1, 1, 2, 4, 8)), layers=rng.randint(4, 16), hidden=hidden, kv=1024,
                    ffn=_log(rng, 2 * hidden, 3 * hidden, 256), vocab=_log(rng, 32000, 128256, 128), bits=rng.choice((3, 4, 5)), bits_head=6, cb=cb)
    t = rng.choice((1, rng.randint(2, 16))) if kind == "moe" else _log(rng, 40, 2048)
    return dict(kind=kind, t=t, experts=rng.choice((32, 64, 128)), topk=rng.choice((4, 6, 8)), hidden=rng.choice((1024, 2048)),
                inter=rng.choice((512, 768, 1024)), bits=rng.choice((2, 3, 4)), cb=cb)


# ---- inputs ---------------------------------------------------------------------------------


class _Make:
    """Seeded tensors on the device."""

    def __init__(self, seed):
        self.g = torch.Generator(device=DEV)
        self.g.manual_seed(seed)

    def randn(self, *shape):
        return torch.randn(shape, device=DEV, generator=self.g)

    def signs(self, *shape):
        return torch.randint(0, 2, shape, device=DEV, generator=self.g).to(torch.float16) * 2 - 1

    def trellis(self, *shape):
        return torch.randint(-32768, 32768, shape, dtype=torch.int16, device=DEV, generator=self.g)

    def linear(self, k, n, bits, cb):
        # decoded weights have standard deviation 1.2437: the outputs of N(0, 1) inputs are N(0, 1)
        svh = (self.signs(n) * (1.0 / (1.2437 * math.sqrt(k)))).to(torch.float16)
        return LinearEXL3(self.trellis(k // 16, n // 16, int(16 * bits)), self.signs(k), svh, mul1=cb == "mul1", mcg=cb == "mcg")


def _dtype(name):
    return {"f16": torch.float16, "bf16": torch.bfloat16, "f32": torch.float32}[name]


def _empty(*shape, dtype=torch.float16):
    return torch.empty(shape, dtype=dtype, device=DEV)


def _prepare_linear(c, mk):
    lin = mk.linear(c["k"], c["n"], c["bits"], c["cb"])
    x = mk.randn(c["m"], c["k"]).to(_dtype(c["dtype"]))
    out = _empty(c["m"], c["n"], dtype=torch.float32) if c["out"] == "f32" else None
    return dict(lin=lin, x=x, out=out)


def _run_linear(s):
    return s["lin"].forward(s["x"], s["out"])


def _prepare_layer(c, mk):
    h, kv, f, m, cb = c["hidden"], c["kv"], c["ffn"], c["m"], c["cb"]
    a, g = c["bits_attn"], c["bits_gu"]
    q, k, v = (mk.linear(h, n, a, cb) for n in (h, kv, kv))
    outs = [_empty(1, m, n) for n in (h, kv, kv)]
    gu_out = _empty(2, m, f)
    dt = _dtype(c["dtype"])
    return dict(qkv=Sliced([q, k, v], outs), o=mk.linear(h, h, a, cb), gu=Multi([mk.linear(h, f, g, cb) for _ in range(2)], gu_out),
                down=mk.linear(f, h, c["bits_down"], cb), had=_empty(3, m, h),
                x=mk.randn(1, m, h).to(dt), a=mk.randn(m, h).to(dt), r=mk.randn(1, m, h).to(dt), act=mk.randn(m, f).to(dt))


def _run_layer(s):
    # attention, norms and the activation belong to the model: their results are inputs here
    q, k, v = s["qkv"].run(s["x"], s["had"])
    o = s["o"].forward(s["a"])
    gu = s["gu"].run(s["r"], s["had"])
    down = s["down"].forward(s["act"])
    return dict(q=q, k=k, v=v, o=o, gu=gu, down=down)


_stream = None


def _decode_stream():
    """The one stream of a decoder's graphs."""
    global _stream
    if _stream is None:
        _stream = torch.cuda.Stream()
    return _stream


def _prepare_step(c, mk):
    h, kv, f, m, cb, b = c["hidden"], c["kv"], c["ffn"], c["m"], c["cb"], c["bits"]
    q, k, v = (_empty(1, m, n) for n in (h, kv, kv))
    gu_out, act = _empty(2, m, f), _empty(m, f)
    o_out, d_out, r = _empty(m, h), _empty(m, h), _empty(1, m, h)
    hid = _empty(1, m, h)
    logits = _empty(m, c["vocab"])
    zero = torch.zeros((1, m, h), dtype=torch.float16, device=DEV)
    layers = []
    for _ in range(c["layers"]):
        layers.append(dict(qkv=Sliced([mk.linear(h, n, b, cb) for n in (h, kv, kv)], [q, k, v]), o=mk.linear(h, h, b, cb),
                           gu=Multi([mk.linear(h, f, b, cb) for _ in range(2)], gu_out), down=mk.linear(f, h, b, cb),
                           norms=(1.0 + 0.05 * mk.randn(2, h)).to(torch.float16)))
    head = mk.linear(h, c["vocab"], c["bits_head"], cb)
    last_norm = (1.0 + 0.05 * mk.randn(h)).to(torch.float16)
    x = mk.randn(1, m, h).to(torch.float16)

    def step():
        prev, add = x, zero
        for L in layers:
            amp.rms_norm_res(prev, add, L["norms"][0], EPS, hid, r)
            L["qkv"].run(r)
            L["o"].forward(q[0], o_out)                      # attention itself is outside the library
            amp.rms_norm_res(hid, o_out.view(1, m, h), L["norms"][1], EPS, hid, r)
            L["gu"].run(r)
            amp.silu_mul(gu_out[0], gu_out[1], act)
            L["down"].forward(act, d_out)
            prev, add = hid, d_out.view(1, m, h)
        amp.rms_norm_res(prev, add, last_norm, EPS, hid, r)
        head.forward(r[0], logits)

    stream = _decode_stream()
    stream.wait_stream(torch.cuda.current_stream())
    graph = DecodeGraph(step, stream=stream)
    return dict(graph=graph, hidden=hid, logits=logits, keep=(layers, head, last_norm, x, zero, q, k, v, act, o_out, d_out, r))


def _run_step(s):
    s["graph"].replay()
    return dict(hidden=s["hidden"], logits=s["logits"])


def _experts(c, mk):
    """Pointer tables of the experts' gate, up and down projections and the tensors behind them."""
    e, h, i, w = c["experts"], c["hidden"], c["inter"], 16 * c["bits"]
    cfg, keep = {}, []
    for key, k, n in (("g", h, i), ("u", h, i), ("d", i, h)):
        tr, suh = mk.trellis(e, k // 16, n // 16, w), mk.signs(e, k)
        svh = (mk.signs(e, n) * (1.0 / (1.2437 * math.sqrt(k)))).to(torch.float16)
        keep += [tr, suh, svh]
        for name, t in (("trellis", tr), ("suh", suh), ("svh", svh)):
            cfg["%s_%s" % (key, name)] = amp.ptr_array([t.data_ptr() + j * t.stride(0) * 2 for j in range(e)], DEV)
    cfg.update(Kg=c["bits"], Ku=c["bits"], Kd=c["bits"], act=0, act_limit=0.0, mcg=c["cb"] == "mcg", mul1=c["cb"] == "mul1", I=i, Hi=h)
    return cfg, keep


def _prepare_moe(c, mk):
    cfg, keep = _experts(c, mk)
    t, h, i, slots = c["t"], c["hidden"], c["inter"], c["t"] * c["topk"]
    zeros = lambda *shape, dtype: torch.zeros(shape, dtype=dtype, device=DEV)
    w, sel = torch.topk(mk.randn(t, c["experts"]), c["topk"], dim=1)
    probs = torch.softmax(w, 1).contiguous()
    x = mk.randn(t, h).to(torch.float16)
    if c["kind"] == "moe_prefill":
        return dict(x=x, sel=sel.contiguous(), probs=probs, experts=c["experts"], cfg=cfg, keep=keep)
    cfg.update(gu_g=zeros(slots, i, dtype=torch.float16), gu_u=zeros(slots, i, dtype=torch.float16), d_out=zeros(slots, h, dtype=torch.float32),
               ctr=zeros(amp.moe_coop_ctr_len(slots, t, i, h), dtype=torch.int32), out=zeros(t, h, dtype=torch.float32))
    return dict(x=x, sel=sel.contiguous(), rw=probs.to(torch.float16), cfg=cfg, keep=keep)


def _run_moe(s):
    amp.moe_coop(s["x"], s["sel"], s["rw"], s["cfg"])
    return s["cfg"]["out"]


def _run_moe_prefill(s):
    fe, order, tok, wts, count, start, inv, kind = amp.moe_prep(s["sel"], s["probs"], s["experts"])
    out = torch.zeros(s["x"].shape, dtype=torch.float32, device=DEV)
    amp.moe_fused(s["x"], out, count, tok, wts, s["cfg"])
    return out


_PREPARE = {"linear": _prepare_linear, "layer": _prepare_layer, "step": _prepare_step, "moe": _prepare_moe, "moe_prefill": _prepare_moe}
_RUN = {"linear": _run_linear, "layer": _run_layer, "step": _run_step, "moe": _run_moe, "moe_prefill": _run_moe_prefill}


def prepare(case, seed):
    state = _PREPARE[case["kind"]](case, _Make(seed))
    state["run"] = _RUN[case["kind"]]
    return state


def run(state):
    return state["run"](state)


# ---- what a pass cannot do without --------------------------------------------------------------


def _linear_work(m, k, n, bits, out_bytes=2):
    """Packed weights, both scale vectors, activations in and out; multiply-adds."""
    return k * n * bits / 8 + 2 * (k + n) + m * (2 * k + out_bytes * n), 2.0 * m * k * n


def _add(*parts):
    return dict(bytes=float(sum(p[0] for p in parts)), flops=float(sum(p[1] for p in parts)))


def work(case):
    c = case
    if c["kind"] == "linear":
        return _add(_linear_work(c["m"], c["k"], c["n"], c["bits"], 4 if c["out"] == "f32" else 2))
    if c["kind"] in ("layer", "step"):
        h, kv, f, m = c["hidden"], c["kv"], c["ffn"], c["m"]
        a, g, d = (c["bits_attn"], c["bits_gu"], c["bits_down"]) if c["kind"] == "layer" else (c["bits"],) * 3
        parts = [_linear_work(m, h, n, a) for n in (h, kv, kv, h)] + [_linear_work(m, h, f, g)] * 2 + [_linear_work(m, f, h, d)]
        shared = -2 * m * h * 3                                  # q|k|v and gate|up read one input each
        one = (sum(p[0] for p in parts) + shared, sum(p[1] for p in parts))
        if c["kind"] == "layer":
            return _add(one)
        return _add(*[one] * c["layers"], _linear_work(m, h, c["vocab"], c["bits_head"]))
    e, h, i, t = c["experts"], c["hidden"], c["inter"], c["t"]
    slots = t * c["topk"]
    distinct = e * (1.0 - (1.0 - c["topk"] / e) ** t)            # experts that a random routing reaches
    return dict(bytes=distinct * 3 * h * i * c["bits"] / 8 + t * h * (2 + 4) + slots * 12, flops=6.0 * slots * h * i)


def tolerance(case):
    if case["kind"] == "step":
        # fp16 residual stream through every layer of the stack
        return {"rel": 1e-2}
    if case["cb"] == "mul1" and case["kind"] == "linear" and case["m"] == 1:
        # 8-bit activation codes by default; another grouping of the scales differs by this much
        return {"rel": 1e-2}
    # fp16 operands (the rotated input rounded once; for experts also the activation between the
    # two projections), fp32 accumulation, one fp16 rounding of the result
    return {"rel": 3e-3}
