"""Timed cases of the inference path, each through entry points of the C ABI (include/kf_device.h, include/kf_model.h) as a host program calls them.

Kinds
  mlp      one feed-forward block on M tokens: norm + gate / up + SwiGLU, then down + residual (two calls); with `half` only the first call
  attn     one attention block with a step of M tokens, one per sequence (decode): norm + Q / K / V, per-head norm + rotation + cache append +
           attention, then the output projection + residual
  prefill  the same block for a panel of M consecutive tokens of one sequence that already holds `past` positions
  sample   temperature / top-k / top-p over M rows of logits
  experts  a routed feed-forward on M tokens: router, routing tables, gate / up and down of the chosen experts, weighted sum
  model    whole forward calls of a small model with host tokens in and host logits out: a decode step of M sequences, or a prompt

Sizes are those of the Qwen3 0.6B / 8B / 32B blocks and of the size presets in koifish_b200/bench_arch.py; drawn cases take other widths and
token counts of the same ranges.  Weights are packed here in the documented storage form (128-bit words, one bf16 zero and step per 128 weights),
so the reference results need nothing of the library.
"""
import ctypes as C
import math

import numpy as np
import torch

import koifish_b200 as kf

VOCAB = 151936
EPS = 1e-6
THETA = 1e6
TYPES = {"q4": kf.KF_T_Q4, "q2": kf.KF_T_SIGN, "q1": kf.KF_T_BINARY, "f8": kf.KF_T_F8E5M2, "bf16": kf.KF_T_BF16}


def listed():
    q3 = dict(E=5120, heads=64, kv=8)
    return [
        # one token through the feed-forward of a 32B model in 4 bits: most of the bytes of single-user decoding
        dict(name="mlp_one", kind="mlp", type="q4", E=5120, F=25600, M=1),
        # the same in ternary weights on the 8B block, a few tokens: low-bit serving of a handful of users
        dict(name="mlp_lowbit", kind="mlp", type="q2", E=4096, F=12288, M=2),
        # batched decoding, an odd number of users: the wide half of the block
        dict(name="mlp_batch", kind="mlp", type="q4", E=5120, F=25600, M=45, half=True),
        # the same for a prompt panel: the largest matmuls
        dict(name="mlp_prompt", kind="mlp", type="q4", E=5120, F=25600, M=2048, half=True),
        # the smallest block in 8 bits, one token, short context: latency and launches
        dict(name="attn_small", kind="attn", type="f8", E=1024, heads=16, kv=8, M=1, ctx=200),
        # batched decoding over ragged contexts
        dict(name="attn_batch", kind="attn", type="q4", E=4096, heads=32, kv=8, M=64, ctx=2000),
        # one user deep into a long context
        dict(name="attn_long", kind="attn", type="q4", M=1, ctx=30000, **q3),
        # a ragged prompt panel behind 4096 earlier positions
        dict(name="prefill_panel", kind="prefill", type="q4", E=4096, heads=32, kv=8, M=1999, past=4096),
        # drawing the next tokens of eight users
        dict(name="sample", kind="sample", M=8, V=VOCAB, temperature=0.7, top_k=50, top_p=0.95),
        # a routed feed-forward on a prompt panel (bench_arch preset m)
        dict(name="experts_panel", kind="experts", E=2048, F=1408, experts=64, top=6, M=512),
        # whole calls on the 0.6B model in 4 bits: a decode step of eight users, and a prompt
        dict(name="model_step", kind="model", layers=28, E=1024, F=3072, heads=16, kv=8, M=8, ctx=24, prompt=0),
        dict(name="model_prompt", kind="model", layers=28, E=1024, F=3072, heads=16, kv=8, M=1, ctx=0, prompt=700),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["mlp", "mlp", "mlp", "attn", "attn", "prefill", "prefill", "sample", "experts"])
    typ = rng.choice(["q4", "q4", "q4", "q2", "q1", "f8", "bf16"])
    if kind == "mlp":
        e = 128 * rng.randint(8, 40)
        f = 128 * rng.choice([rng.randint(24, 48), rng.randint(24, 200)])
        m = _log(rng, 1, 2000)
        return dict(kind=kind, type=typ, E=e, F=f, M=m, half=m > 8 and f > 6144)
    if kind == "attn":
        kv = 8
        m = rng.choice([1, 1, _log(rng, 2, 64)])
        heads = kv * rng.choice([2, 4, 8] if m <= 8 else [2, 4])
        return dict(kind=kind, type=typ, E=128 * rng.randint(8, 40), heads=heads, kv=kv, M=m, ctx=_log(rng, 20, 40000 if m == 1 else 100000 // m))
    if kind == "prefill":
        kv = 8
        return dict(kind=kind, type=typ, E=128 * rng.randint(8, 40), heads=kv * rng.choice([2, 4]), kv=kv, M=_log(rng, 17, 2000),
                    past=rng.choice([0, _log(rng, 1, 4000)]))
    if kind == "sample":
        return dict(kind=kind, M=_log(rng, 1, 64), V=rng.choice([VOCAB, 32768, rng.randint(1000, 150000)]), temperature=round(rng.uniform(0.3, 1.2), 2),
                    top_k=rng.choice([20, 50, 200]), top_p=rng.choice([0.8, 0.95, 1.0]))
    x = rng.choice([16, 32, 64])
    return dict(kind=kind, E=128 * rng.randint(8, 24), F=128 * rng.randint(4, 14), experts=x, top=rng.choice([2, 4, 6]), M=_log(rng, 1, 700))


# ---------------------------------------------------------------------------------------------------------------- context, calls, weights
_CTX = []


def _ctx():
    if not _CTX:
        s = torch.cuda.Stream()
        _CTX.extend([kf.Context(0, s.cuda_stream), s])
    return _CTX[0]


def _stream():
    _ctx()
    return torch.cuda.stream(_CTX[1])


def _ok(st):
    if st:
        raise RuntimeError("status %d: %s" % (st, _ctx().lib.kf_last_error(_ctx().h).decode()))


def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(1000003 * int(seed) + 17)
    return g


def _normal(g, *shape, sigma=1.0, mean=0.0):
    return (torch.randn(*shape, generator=g, device="cuda") * sigma + mean).bfloat16()


def _pack(codes, bits):
    """[rows, cols] codes -> bytes of 128-bit words: the first code of a word in its most significant bits, bytes in little-endian order"""
    rows, cols = codes.shape
    per = 8 // bits
    c = codes.view(rows, cols // per, per).to(torch.uint8)
    b = torch.zeros(rows, cols // per, dtype=torch.uint8, device=codes.device)
    for j in range(per):
        b |= c[:, :, j] << (8 - bits * (j + 1))
    return b.view(rows, -1, 16).flip(2).contiguous().view(rows, -1)


class Weight:
    """One weight [rows, cols] in storage form, and its values in 64 bits."""

    def __init__(self, g, typ, rows, cols, sigma=0.02):
        self.typ, self.rows, self.cols, self.qbias, self.gama = typ, rows, cols, 0, None
        w = torch.randn(rows, cols, generator=g, device="cuda") * sigma
        if typ == "bf16":
            self.data = w.bfloat16()
            return
        if typ == "f8":  # the upper byte of the fp16 value
            self.data = (w.half().view(torch.int16).to(torch.int32) >> 8).to(torch.uint8)
            return
        grp = w.view(rows, cols // 128, 128)
        if typ == "q4":  # round to nearest over the group's range
            lo, hi = grp.amin(2), grp.amax(2)
            step, zero, bits, top = ((hi - lo) / 15).bfloat16(), (-lo).bfloat16(), 4, 15
            q = torch.round((grp + zero.float()[:, :, None]) / step.float()[:, :, None]).clamp_(0, top)
        elif typ == "q2":  # ternary: step * {-1, 0, 1}, stored with a bias of one
            step, bits, self.qbias = grp.abs().mean(2).bfloat16(), 2, 1
            zero = torch.zeros_like(step)
            q = torch.round(grp / step.float()[:, :, None]).clamp_(-1, 1) + 1
        else:  # binary: step * {0, 1}
            step, bits = grp.clamp(min=0).square().mean(2).sqrt().bfloat16(), 1
            zero = torch.zeros_like(step)
            q = torch.round(grp / step.float()[:, :, None]).clamp_(0, 1)
        self.bits, self.zero, self.step = bits, zero, step
        self.data = _pack(q.view(rows, cols), bits)
        one = torch.ones(rows + cols, device="cuda", dtype=torch.bfloat16)
        self.gama = torch.cat([one, zero.reshape(-1), step.reshape(-1)])

    def desc(self):
        return kf.TensorDesc(self.data.data_ptr(), None if self.gama is None else self.gama.data_ptr(), self.rows, self.cols, TYPES[self.typ], 128, self.qbias, None, None)

    def exact(self):
        if self.typ == "bf16":
            return self.data.double()
        if self.typ == "f8":
            return (self.data.to(torch.int32) << 8).to(torch.int16).view(torch.float16).double()
        b = self.data.view(self.rows, -1, 16).flip(2).reshape(self.rows, -1)
        per = 8 // self.bits
        q = torch.stack([(b >> (8 - self.bits * (j + 1))) & ((1 << self.bits) - 1) for j in range(per)], 2).view(self.rows, -1, 128)
        return (self.step.double()[:, :, None] * (q.double() - self.qbias) - self.zero.double()[:, :, None]).view(self.rows, self.cols)


def _bytes_of(typ, rows, cols):
    bits = {"q4": 4, "q2": 2, "q1": 1, "f8": 8, "bf16": 16}[typ]
    return rows * cols * bits / 8 + (rows * cols / 128 * 4 if bits in (1, 2, 4) else 0)


# ---------------------------------------------------------------------------------------------------------------- inputs of each kind
def _make(c, seed):
    g, k = _gen(seed), c["kind"]
    s = dict(c)
    if k == "mlp":
        s["x"] = _normal(g, c["M"], c["E"])
        s["norm"] = _normal(g, c["E"], sigma=0.1, mean=1.0)
        s["gate"], s["up"] = Weight(g, c["type"], c["F"], c["E"]), Weight(g, c["type"], c["F"], c["E"])
        s["down"] = None if c.get("half") else Weight(g, c["type"], c["E"], c["F"])
    elif k in ("attn", "prefill"):
        e, qd, kd, m = c["E"], c["heads"] * 128, c["kv"] * 128, c["M"]
        s["x"] = _normal(g, m, e)
        s["norm"] = _normal(g, e, sigma=0.1, mean=1.0)
        s["wq"], s["wk"], s["wv"], s["wo"] = (Weight(g, c["type"], r, n) for r, n in ((qd, e), (kd, e), (kd, e), (e, qd)))
        s["qnorm"], s["knorm"] = _normal(g, 128, sigma=0.1, mean=1.4), _normal(g, 128, sigma=0.1, mean=1.4)
        if k == "attn":
            s["max_seq"] = c["ctx"] + 1
            low = max(0, c["ctx"] // 4) if m > 1 else c["ctx"]
            s["pos"] = torch.randint(low, c["ctx"] + 1, (m,), generator=g, device="cuda", dtype=torch.int32)
            seqs = m
        else:
            s["max_seq"] = c["past"] + m
            s["pos"] = torch.arange(c["past"], c["past"] + m, device="cuda", dtype=torch.int32)
            seqs = 1
        s["kc"] = _normal(g, seqs, s["max_seq"], kd, sigma=1.4)
        s["vc"] = _normal(g, seqs, s["max_seq"], kd, sigma=0.6)
    elif k == "sample":
        s["logits"] = _normal(g, c["M"], c["V"], sigma=2.5)
        s["seeds"] = torch.randint(1, 2 ** 62, (c["M"],), generator=g, device="cuda", dtype=torch.int64)
    elif k == "experts":
        e, f, x, m = c["E"], c["F"], c["experts"], c["M"]
        s["x"] = _normal(g, m, e)
        s["router"] = _normal(g, x, e, sigma=e ** -0.5)
        s["wg"], s["wu"], s["wd"] = _normal(g, x, f, e, sigma=0.02), _normal(g, x, f, e, sigma=0.02), _normal(g, x, e, f, sigma=0.02)
    else:
        r = np.random.RandomState(seed % (2 ** 31))
        s["tokens"] = r.randint(0, VOCAB, size=(c["M"], max(c["ctx"] + 1, c["prompt"]))).astype(np.int32)
    return s


def prepare(case, seed):
    ctx = _ctx()
    with _stream():
        s = _make(case, seed)
        k, m = s["kind"], s["M"]
        buf = lambda *shape, dtype=torch.bfloat16: torch.zeros(*shape, dtype=dtype, device="cuda")  # noqa: E731
        if k == "mlp":
            s["h"], s["y"] = buf(m, s["F"]), buf(m, s["E"])
            s["gu"], s["dn"] = (kf.TensorDesc * 2)(s["gate"].desc(), s["up"].desc()), s["down"].desc() if s["down"] else None
            s["hs"] = (C.c_void_p * 2)(s["h"].data_ptr(), s["h"].data_ptr())
        elif k in ("attn", "prefill"):
            qd, kd = s["heads"] * 128, s["kv"] * 128
            s["q"], s["k"], s["v"], s["a"], s["y"] = buf(m, qd), buf(m, kd), buf(m, kd), buf(m, qd), buf(m, s["E"])
            s["qkv"], s["od"] = (kf.TensorDesc * 3)(s["wq"].desc(), s["wk"].desc(), s["wv"].desc()), s["wo"].desc()
            s["ys"] = (C.c_void_p * 3)(s["q"].data_ptr(), s["k"].data_ptr(), s["v"].data_ptr())
            s["table"] = buf(s["max_seq"] * 64 * 2, dtype=torch.float32)
            _ok(ctx.lib.kf_rope_table(ctx.h, s["table"].data_ptr(), s["max_seq"], 128, THETA))
        elif k == "sample":
            s["state"], s["out"] = buf(m, dtype=torch.int64), buf(m, dtype=torch.int32)
        elif k == "experts":
            x, n = s["experts"], m * s["top"]
            for name, t in (("tg", "wg"), ("tu", "wu"), ("td", "wd")):
                s[name] = torch.tensor([s[t][i].data_ptr() for i in range(x)], dtype=torch.int64, device="cuda")
            s["rd"] = kf.TensorDesc(s["router"].data_ptr(), None, x, s["E"], kf.KF_T_BF16, 128, 0, None, None)
            i32 = dict(dtype=torch.int32)
            s["logits"], s["wgt"] = buf(m, x, dtype=torch.float32), buf(n, dtype=torch.float32)
            s["idx"], s["offsets"], s["slot"], s["row"], s["group"], s["work"] = buf(n, **i32), buf(x + 1, **i32), buf(n, **i32), buf(n, **i32), buf(n, **i32), buf(2 * n + x, **i32)
            s["h"], s["ys"], s["y"] = buf(n, s["F"]), buf(n, s["E"], dtype=torch.float32), buf(m, s["E"], dtype=torch.float32)
        else:
            quant = {"group_size": 128, "self_attn": {"quant_method": "RTN", "bits": 4}, "mlp": {"quant_method": "RTN", "bits": 4}}
            cfg = kf.qwen3_config(s["layers"], s["E"], s["F"], s["heads"], s["kv"], 128, VOCAB, quant, True, 1024, s["M"], seed % 100003 + 1, THETA,
                                  max_prefill=1024 if s["prompt"] else None)
            s["model"] = kf.Model(ctx, cfg)
            s["model"].init_random()
            for t in range(s["ctx"]):  # the context of every sequence
                s["model"].forward(s["tokens"][:, t], np.full(m, t), seq_mode=1, want_logits=False)
    torch.cuda.synchronize()
    return s


def run(s):
    ctx = _CTX[0]
    lib, h, k, m = ctx.lib, ctx.h, s["kind"], s["M"]
    if k == "mlp":
        _ok(lib.kf_rmsnorm_linear(h, 2, s["hs"], s["gu"], s["x"].data_ptr(), s["norm"].data_ptr(), EPS, m, 2))
        if s["down"] is None:
            return [s["h"]]
        _ok(lib.kf_linear(h, s["y"].data_ptr(), C.byref(s["dn"]), s["h"].data_ptr(), m, kf.KF_EPI_RESIDUAL, s["x"].data_ptr()))
        return [s["h"], s["y"]]
    if k in ("attn", "prefill"):
        q, kk, v, a, kc, vc, pos = (s[n].data_ptr() for n in ("q", "k", "v", "a", "kc", "vc", "pos"))
        nh, kv, ms = s["heads"], s["kv"], s["max_seq"]
        stride = ms * kv * 128 if k == "attn" else 0
        _ok(lib.kf_rmsnorm_linear(h, 3, s["ys"], s["qkv"], s["x"].data_ptr(), s["norm"].data_ptr(), EPS, m, 0))
        if k == "attn" and m * nh <= 64 and s["ctx"] < 1024:  # the choice the model runtime makes: few heads over a short context in one launch
            _ok(lib.kf_qkv_attention(h, a, q, kk, v, s["qnorm"].data_ptr(), s["knorm"].data_ptr(), kc, vc, s["table"].data_ptr(), pos, m, nh, kv, 128, ms, EPS, stride, s["ctx"]))
        else:
            _ok(lib.kf_qknorm_rope_kvappend(h, q, kk, v, s["qnorm"].data_ptr(), s["knorm"].data_ptr(), kc, vc, s["table"].data_ptr(), pos, m, nh, kv, 128, ms, EPS, stride))
            if k == "attn":
                _ok(lib.kf_attn_decode_gqa(h, a, q, kc, vc, pos, m, nh, kv, 128, ms, s["ctx"], stride))
            else:
                _ok(lib.kf_attn_prefill(h, a, q, kc, vc, pos, m, nh, kv, 128, ms))
        _ok(lib.kf_linear(h, s["y"].data_ptr(), C.byref(s["od"]), a, m, kf.KF_EPI_RESIDUAL, s["x"].data_ptr()))
        return [s["a"], s["y"], s["kc"], s["vc"]]
    if k == "sample":
        _ok(lib.kf_d2d(h, s["state"].data_ptr(), s["seeds"].data_ptr(), 8 * m))  # every request starts from its own seed
        _ok(lib.kf_sample(h, s["out"].data_ptr(), s["logits"].data_ptr(), m, s["V"], s["temperature"], s["top_k"], s["top_p"], s["state"].data_ptr(), 0))
        return [s["out"], s["state"]]
    if k == "experts":
        e, f, x, top = s["E"], s["F"], s["experts"], s["top"]
        p = {n: s[n].data_ptr() for n in ("x", "logits", "wgt", "idx", "offsets", "slot", "row", "group", "work", "h", "ys", "y", "tg", "tu", "td")}
        _ok(lib.kf_linear_g(h, p["logits"], x, C.byref(s["rd"]), p["x"], 0, e, m))
        _ok(lib.kf_moe_route(h, p["idx"], p["wgt"], p["offsets"], p["slot"], p["row"], p["group"], p["work"], p["logits"], x, None, m, x, top))
        _ok(lib.kf_linear_grouped(h, p["h"], f, p["tg"], p["tu"], x, f, e, p["x"], 0, e, p["offsets"], p["group"], p["row"], m * top))
        _ok(lib.kf_linear_grouped(h, p["ys"], e, p["td"], None, x, e, f, p["h"], 0, f, p["offsets"], p["group"], None, m * top))
        _ok(lib.kf_moe_combine(h, p["y"], p["ys"], p["slot"], p["wgt"], None, None, 0, m, e, top))
        return [s["logits"], s["y"]]
    t = s["tokens"]
    if s["prompt"]:
        logits, _ = s["model"].prefill(t[0], want_logits=True)
    else:
        logits, _ = s["model"].forward(t[:, s["ctx"]], np.full(m, s["ctx"], dtype=np.int32), seq_mode=1, want_logits=True)
    return [torch.from_numpy(logits.view(np.int16)).view(torch.bfloat16)]


# ---------------------------------------------------------------------------------------------------------------- cost, tolerance, 64-bit results
def work(case):
    c, k, m = case, case["kind"], case["M"]
    if k == "mlp":
        n = 2 if c.get("half") else 3
        return dict(bytes=n * _bytes_of(c["type"], c["F"], c["E"]) + 2 * (n - 1) * m * c["E"] + 2 * m * c["F"], flops=2 * m * n * c["E"] * c["F"])
    if k in ("attn", "prefill"):
        e, qd, kd = c["E"], c["heads"] * 128, c["kv"] * 128
        keys = (c["ctx"] if m == 1 else 0.625 * c["ctx"]) * m if k == "attn" else m * (c["past"] + 0.5 * m)
        rows = keys if k == "attn" else c["past"] + m
        w = _bytes_of(c["type"], qd + 2 * kd, e) + _bytes_of(c["type"], e, qd)
        return dict(bytes=w + 4 * kd * rows + 4 * m * e + 2 * m * qd, flops=2 * m * e * (2 * qd + 2 * kd) + 4 * keys * qd)
    if k == "sample":
        return dict(bytes=2 * m * c["V"] + 20 * m, flops=0)
    if k == "experts":
        hit = c["experts"] * (1 - (1 - c["top"] / c["experts"]) ** m)
        return dict(bytes=hit * 6 * c["E"] * c["F"] + 2 * c["experts"] * c["E"] + 6 * m * c["E"] + 4 * m * c["experts"], flops=2 * m * (3 * c["top"] * c["E"] * c["F"] + c["experts"] * c["E"]))
    layer = c["E"] * (3 * c["F"] + (2 * c["heads"] + 2 * c["kv"]) * 128)
    rows = c["prompt"] or m
    head = VOCAB * c["E"]
    return dict(bytes=c["layers"] * _bytes_of("q4", 1, layer) + 2 * head + 2 * m * VOCAB, flops=2 * rows * c["layers"] * layer + 2 * (1 if c["prompt"] else m) * head)


def tolerance(case):
    # relative errors between two correct implementations, times about four: weights rounded to bf16 or not, sums in another order
    k = case["kind"]
    if k == "sample":
        return "exact"
    if k == "model":
        return dict(rel=0.03, max=0.5)
    return dict(rel=0.012, max=0.2)


def _rms(x, w):
    return x / torch.sqrt(x.square().mean(-1, keepdim=True) + EPS) * w


def _rotate(x, pos):
    """halves of every head of 128 rotated by pos * THETA^(-i / 64)"""
    inv = THETA ** (-torch.arange(64, device=x.device, dtype=torch.float64) / 64)
    ang = pos.double()[:, None, None] * inv
    a, b = x[..., :64], x[..., 64:]
    return torch.cat([a * ang.cos() - b * ang.sin(), b * ang.cos() + a * ang.sin()], -1)


def exact(case, seed):
    k, m = case["kind"], case["M"]
    if k in ("model", "sample"):
        return None
    s = _make(case, seed)
    x = s["x"].double()
    if k == "mlp":
        n = _rms(x, s["norm"].double())
        g = n @ s["gate"].exact().T
        h = g * torch.sigmoid(g) * (n @ s["up"].exact().T)
        return [h] if s["down"] is None else [h, x + h @ s["down"].exact().T]
    if k == "experts":
        lg = x @ s["router"].double().T
        val, idx = lg.topk(case["top"], dim=1)
        wgt, y = torch.softmax(val, 1), torch.zeros_like(x)
        for e in range(case["experts"]):
            t, j = (idx == e).nonzero(as_tuple=True)
            if len(t):
                g = x[t] @ s["wg"][e].double().T
                y.index_add_(0, t, wgt[t, j, None] * ((g * torch.sigmoid(g) * (x[t] @ s["wu"][e].double().T)) @ s["wd"][e].double().T))
        return [lg, y]
    nh, kv, pos = case["heads"], case["kv"], s["pos"]
    n = _rms(x, s["norm"].double())
    q = _rotate(_rms((n @ s["wq"].exact().T).view(m, nh, 128), s["qnorm"].double()), pos)
    kk = _rotate(_rms((n @ s["wk"].exact().T).view(m, kv, 128), s["knorm"].double()), pos)
    v = (n @ s["wv"].exact().T).view(m, kv, 128)
    seqs = s["kc"].shape[0]
    kc, vc = s["kc"].double().view(seqs, -1, kv, 128), s["vc"].double().view(seqs, -1, kv, 128)
    at = torch.arange(m, device="cuda") if k == "attn" else torch.zeros(m, device="cuda", dtype=torch.long)
    kc[at, pos.long()], vc[at, pos.long()] = kk, v
    a = torch.empty_like(q)
    for i in range(m) if k == "attn" else range(0):
        n_i = int(pos[i]) + 1
        sc = torch.einsum("gjd,tgd->gjt", q[i].view(kv, nh // kv, 128), kc[i, :n_i]) / 128 ** 0.5
        a[i] = torch.einsum("gjt,tgd->gjd", torch.softmax(sc, -1), vc[i, :n_i]).reshape(nh, 128)
    for hd in range(nh) if k == "prefill" else range(0):
        sc = q[:, hd] @ kc[0, :, hd // (nh // kv)].T / 128 ** 0.5
        sc.masked_fill_(torch.arange(sc.shape[1], device="cuda")[None, :] > pos[:, None], -math.inf)
        a[:, hd] = torch.softmax(sc, -1) @ vc[0, :, hd // (nh // kv)]
    a = a.reshape(m, -1)
    return [a, x + a @ s["wo"].exact().T, kc.view(seqs, -1, kv * 128), vc.view(seqs, -1, kv * 128)]
