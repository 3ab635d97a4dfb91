"""The measured cases: what programs have this framework do, through the calls they make.

Six paths, each over a range of sizes that `draw` spans:
  decode    one step of the Llama engine for a batch (Decoder.step / step_paged), hidden rows in and out, keys and values appended
  prefill   prompts through the Llama engine into the paged cache (Decoder.prefill_paged), with and without earlier context
  head      the tail of every generated token: final norm, LM head, top-k, sampling (Decoder.lm_head_topk_sample)
  vasolix   a whole Vasolix-shaped model on the layer-list decoder: prompts and the first token after them, or one decode step
  zefenex   one Zefenex-shaped layer (latent attention in a window, dense feed-forward): prompts and the first token after them
  fedovik   one Fedovik-shaped layer (windowed attention beside a gated delta rule, gated feed-forward): the same
Sizes are those of bench.py's configurations; weights are random, of each design's distributions."""
import importlib
import math

import numpy as np
import torch

F64 = torch.float64
PAGE = 64
DEV = "cuda"
TYPES = {"bf16": torch.bfloat16, "fp16": torch.float16, "fp32": torch.float32, "fp8": torch.bfloat16, "int4": torch.bfloat16}
GROUP = 128  # INT4: weights that share a scale

# hidden, query heads, kv heads, feed-forward, head size 128
LLAMA = {
    "7b": (4096, 32, 32, 11008),
    "70b": (8192, 64, 8, 28672),
    "70b-shard": (8192, 8, 1, 3584),   # one of eight tensor-parallel shards
    "small": (2048, 16, 4, 2688),
    "tiny": (1024, 8, 2, 1408),
}
VASOLIX = {
    "s": dict(width=1024, heads=8, kv_heads=2, chunk=512, g_heads=4, g_dim=64, g_vdim=256, rank=32, experts=16, top=2, ff=512, shared=1024),
    "m": dict(width=2048, heads=16, kv_heads=4, chunk=1024, g_heads=8, g_dim=128, g_vdim=256, rank=64, experts=32, top=4, ff=512, shared=2048),
}
ZEFENEX = {"s": dict(width=1024, heads=8, rank=192, window=512, ff=4096), "m": dict(width=2048, heads=16, rank=192, window=1024, ff=8192)}
FEDOVIK = {
    "s": dict(width=1024, ff=2816, heads=8, kv_heads=2, window=512, r_heads=4, r_dim=64, r_vdim=256, rank=32),
    "m": dict(width=2048, ff=5632, heads=16, kv_heads=4, window=1024, r_heads=8, r_dim=128, r_vdim=256, rank=64),
}
HEAD_DIM = 128
LAYER_VOCAB = 1024  # of the single-layer cases: the head is not what they are about


def _pkg(sub=""):
    return importlib.import_module("llm-inference-engine_b200" + sub)


def listed():
    return [
        # one user at a terminal: the step that bench.py times, four of its layers
        dict(name="decode 7b bf16 b1", path="decode", model="7b", fmt="bf16", layers=4, batch=1, ctx=1024, paged=False),
        # a busy server: requests of different ages over the paged cache
        dict(name="decode 7b bf16 b16 ragged", path="decode", model="7b", fmt="bf16", layers=4, batch=16, ctx=1024, paged=True),
        # weight-only quantisation where it is used: FP8 for throughput, INT4 for latency
        dict(name="decode 7b fp8 b16 ragged", path="decode", model="7b", fmt="fp8", layers=4, batch=16, ctx=1024, paged=True),
        dict(name="decode 7b int4 b1", path="decode", model="7b", fmt="int4", layers=4, batch=1, ctx=1024, paged=False),
        # the smallest calls: a small model in the reference's own type, a short context
        dict(name="decode tiny fp32 b1", path="decode", model="tiny", fmt="fp32", layers=4, batch=1, ctx=129, paged=False),
        # one long prompt
        dict(name="prefill 7b bf16 2048", path="prefill", model="7b", fmt="bf16", layers=2, lens="2048", hist="0"),
        # admitted together: prompts of any length, some continuing an earlier portion; grouped heads
        dict(name="prefill 70b fp16 ragged", path="prefill", model="70b", fmt="fp16", layers=1, lens="37,611,129,302,5", hist="0,512,0,77,1000"),
        # the tail of a decode step of eight requests
        dict(name="head 7b b8", path="head", hidden=4096, vocab=32000, fmt="bf16", batch=8, k=5),
        # a whole layer-list model: one long prompt and its first token; a decode step of sixteen requests
        dict(name="vasolix m prompt 4096", path="vasolix", size="m", dtype="bf16", lens="4096", decode=False),
        dict(name="vasolix m decode 16", path="vasolix", size="m", dtype="bf16", lens=",".join(["1536"] * 16), decode=True),
        # single layers of two other designs over prompts of uneven lengths
        dict(name="zefenex m layer", path="zefenex", size="m", dtype="bf16", lens="2048,1037"),
        dict(name="fedovik m layer", path="fedovik", size="m", dtype="bf16", lens="1500,511,900"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _lens(rng, total, most):
    n = min(rng.randint(1, most), total)
    cuts = sorted(rng.sample(range(1, total), n - 1)) if n > 1 else []
    return [b - a for a, b in zip([0] + cuts, cuts + [total])]


def draw(rng):
    path = rng.choice(("decode", "decode", "decode", "prefill", "prefill", "head", "vasolix", "vasolix", "zefenex", "fedovik"))
    if path == "decode":
        fmt = rng.choice(("bf16", "bf16", "fp16", "fp8", "int4", "fp32"))
        model = rng.choice(("tiny", "small")) if fmt == "fp32" else rng.choice(("7b", "7b", "70b-shard", "small"))
        batch = rng.randint(1, 4) if fmt == "fp32" else _log(rng, 1, 32)
        return dict(path="decode", model=model, fmt=fmt, layers=4, batch=batch, ctx=_log(rng, 16, 2048), paged=fmt != "fp32" and rng.random() < 0.7)
    if path == "prefill":
        model = rng.choice(("7b", "70b", "small"))
        lens = _lens(rng, _log(rng, 16, 1024 if model == "70b" else 2048), 6)
        hist = [rng.choice((0, 0, rng.randint(1, 1024))) for _ in lens]
        return dict(path="prefill", model=model, fmt=rng.choice(("bf16", "bf16", "fp16", "fp8", "int4")), layers={"7b": 2, "70b": 1, "small": 4}[model],
                    lens=",".join(map(str, lens)), hist=",".join(map(str, hist)))
    if path == "head":
        return dict(path="head", hidden=rng.choice((2048, 4096, 5120, 8192)), vocab=rng.choice((32000, 50257)), fmt=rng.choice(("bf16", "fp16")),
                    batch=_log(rng, 1, 32), k=rng.randint(1, 8))
    if path == "vasolix":
        if rng.random() < 0.5:
            lens, decode = [_log(rng, 16, 2000)] * _log(rng, 1, 32), True
        else:
            lens, decode = _lens(rng, _log(rng, 64, 4000), 4), False
        return dict(path="vasolix", size=rng.choice(("s", "m")), dtype=rng.choice(("bf16", "bf16", "fp16")), lens=",".join(map(str, lens)), decode=decode)
    return dict(path=path, size=rng.choice(("s", "m")), dtype=rng.choice(("bf16", "bf16", "fp16")), lens=",".join(map(str, _lens(rng, _log(rng, 64, 4000), 4))))


def _ints(text):
    return [int(v) for v in text.split(",")]


class _Random:
    """Random tensors on the device, of one seed."""

    def __init__(self, seed):
        self.gen = torch.Generator(device=DEV).manual_seed(seed)

    def normal(self, *shape, std=1.0, mean=0.0, dtype=torch.bfloat16):
        return (torch.randn(*shape, generator=self.gen, device=DEV) * std + mean).to(dtype)

    def uniform(self, *shape, lo=0.0, hi=1.0, dtype=torch.bfloat16):
        return (torch.rand(*shape, generator=self.gen, device=DEV) * (hi - lo) + lo).to(dtype)

    def ints(self, lo, hi, *shape, dtype=torch.int32):
        return torch.randint(lo, hi, shape, generator=self.gen, device=DEV, dtype=dtype)

    def perm(self, n):
        return torch.randperm(n, generator=self.gen, device=DEV).to(torch.int32)


# ------------------------------------------------------------------------------------------------ the Llama engine
def _linear_weight(r, n, k, fmt):
    """One linear's device tensors as the engine takes them: dense, or codes with their scales (and zero points)."""
    if fmt == "fp8":
        return r.normal(n, k).to(torch.float8_e4m3fn).view(torch.uint8), r.uniform(n, lo=0.8, hi=1.2, dtype=torch.float32) / math.sqrt(k), None
    if fmt == "int4":
        codes = r.ints(0, 256, n, k // 2, dtype=torch.uint8)
        return codes, r.uniform(n, k // GROUP, lo=0.17 / math.sqrt(k), hi=0.26 / math.sqrt(k)), r.ints(7, 9, n, k // GROUP, dtype=torch.uint8)
    return r.normal(n, k, std=1.0 / math.sqrt(k), dtype=TYPES[fmt])


def _dense64(w, fmt):
    if fmt == "fp8":
        return w[0].view(torch.float8_e4m3fn).to(torch.float32).to(F64) * w[1].to(F64)[:, None]
    if fmt == "int4":
        codes, scales, zeros = w
        q = torch.stack((codes & 15, codes >> 4), -1).reshape(codes.shape[0], -1, GROUP)
        return ((q.to(F64) - zeros.to(F64)[..., None]) * scales.to(F64)[..., None]).reshape(codes.shape[0], -1)
    return w.to(F64)


def _llama_layers(case, r):
    h, heads, kv, inter = LLAMA[case["model"]]
    dt, fmt, d = TYPES[case["fmt"]], case["fmt"], HEAD_DIM
    return [dict(g1=r.normal(h, std=0.1, mean=1.0, dtype=dt), g2=r.normal(h, std=0.1, mean=1.0, dtype=dt),
                 qkv=_linear_weight(r, (heads + 2 * kv) * d, h, fmt), o=_linear_weight(r, h, heads * d, fmt),
                 gate_up=_linear_weight(r, 2 * inter, h, fmt), down=_linear_weight(r, h, inter, fmt)) for _ in range(case["layers"])]


def _llama_engine(case, layers, max_seq, max_batch):
    m = _pkg()
    h, heads, kv, inter = LLAMA[case["model"]]
    code = {torch.bfloat16: m.BF16, torch.float16: m.F16, torch.float32: m.F32}[TYPES[case["fmt"]]]
    fmt = {"fp8": m.W_FP8, "int4": m.W_INT4}.get(case["fmt"], m.W_DENSE)
    dec = m.Decoder(m.DecoderConfig(h, heads, kv, HEAD_DIM, inter, case["layers"], max_seq, max_batch, code, fmt, GROUP, 1e-6, HEAD_DIM, 10000.0, 1, 0), DEV)
    for i, w in enumerate(layers):
        dec.set_layer(i, w)
    return dec


def _llama_inputs(case, seed):
    """(random source, layers, contexts per row, new tokens per row, ids, embedding table, pages, key and value caches)."""
    r = _Random(seed)
    h, heads, kv, _ = LLAMA[case["model"]]
    dt = TYPES[case["fmt"]]
    layers = _llama_layers(case, r)
    if case["path"] == "decode":
        b = case["batch"]
        # a ragged batch: ages spread between an eighth of the context and all of it
        hist = [case["ctx"] - 1] * b if not case["paged"] or b == 1 else [max(1, case["ctx"] * (8 * (b - 1) - 7 * i) // (8 * (b - 1))) - 1 for i in range(b)]
        new = [1] * b
    else:
        new, hist = _ints(case["lens"]), _ints(case["hist"])
    ids = r.ints(0, 4096, sum(new))
    table = r.normal(4096, h, dtype=dt)
    per = (max(a + b for a, b in zip(hist, new)) + PAGE - 1) // PAGE
    if case.get("paged", True):
        pages = r.perm(per * len(new)).reshape(len(new), per)
        shape = (case["layers"], per * len(new), kv, PAGE, HEAD_DIM)
    else:
        pages, shape = None, (case["layers"], len(new), kv, per * PAGE, HEAD_DIM)
    return r, layers, hist, new, ids, table, pages, r.normal(*shape, dtype=dt), r.normal(*shape, dtype=dt)


def _prepare_llama(case, seed):
    _, layers, hist, new, ids, table, pages, k, v = _llama_inputs(case, seed)
    total = [a + b for a, b in zip(hist, new)]
    per = (max(total) + PAGE - 1) // PAGE
    dev = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)  # noqa: E731
    return dict(case=case, engine=_llama_engine(case, layers, per * PAGE, len(new)), ids=ids, table=table, pages=pages, k=k, v=v, total=dev(total),
                hist=dev(hist), new=dev(new), longest=max(total), widest=max(new))


def _run_llama(s):
    hidden = _pkg().input_embedding(s["ids"], s["table"])
    e = s["engine"]
    if s["case"]["path"] == "prefill":
        e.prefill_paged(hidden, s["k"], s["v"], s["pages"], s["new"], s["hist"], s["total"], s["widest"])
    elif s["pages"] is not None:
        e.step_paged(hidden, s["k"], s["v"], s["pages"], s["total"], s["longest"])
    else:
        e.step(hidden, s["k"], s["v"], s["longest"])
    return hidden, s["k"], s["v"]


def _rope64(x, pos):
    """x [T, heads, d]: channel i turns with channel i + d/2."""
    half = x.shape[-1] // 2
    ang = pos.to(F64)[:, None] * 10000.0 ** (-torch.arange(half, device=x.device, dtype=F64) / half)
    c, s = torch.cos(ang)[:, None], torch.sin(ang)[:, None]
    a, b = x[..., :half], x[..., half:]
    return torch.cat((a * c - b * s, b * c + a * s), -1)


def _rms64(x, eps):
    return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + eps)


def _causal64(q, k, v, scale, start, see=None, sink=None, bias=None, tiny=0.0):
    """Softmax attention of q [T, heads, d] at positions start.. over k, v [S, kv heads, d]; see(i, j) narrows the mask, bias(head, i - j) joins the score."""
    T, H, _ = q.shape
    S, G = k.shape[0], k.shape[1]
    i, j = torch.arange(start, start + T, device=q.device)[:, None], torch.arange(S, device=q.device)[None, :]
    mask = j <= i if see is None else (j <= i) & see(i, j)
    out = torch.empty(T, H, v.shape[-1], dtype=F64, device=q.device)
    for h in range(H):
        g = h // (H // G)
        s = q[:, h] @ k[:, g].T * scale
        if bias is not None:
            s = s + bias(h, (i - j).clamp(min=0))
        s = s.masked_fill(~mask, -math.inf)
        top = s.amax(-1, keepdim=True)
        if sink is not None:
            top = torch.maximum(top, sink[h])
        e = torch.exp(s - top)
        total = e.sum(-1, keepdim=True) + tiny + (torch.exp(sink[h] - top) if sink is not None else 0.0)
        out[:, h] = (e / total) @ v[:, g]
    return out


def _exact_llama(case, seed):
    _, layers, hist, new, ids, table, pages, k_cache, v_cache = _llama_inputs(case, seed)
    _, heads, kv, inter = LLAMA[case["model"]]
    d, fmt = HEAD_DIM, case["fmt"]
    x = table[ids.long()].to(F64)
    k_out, v_out = k_cache.to(F64), v_cache.to(F64)
    pos = torch.cat([torch.arange(a, a + b, device=DEV) for a, b in zip(hist, new)])
    start = np.cumsum([0] + new).tolist()
    rows = []  # per sequence: where its positions lie in a layer of the cache
    for b, (a, n) in enumerate(zip(hist, new)):
        p = torch.arange(a + n, device=DEV)
        rows.append((pages[b].long()[p // PAGE], p % PAGE) if pages is not None else (torch.full_like(p, b), p))
    for li, w in enumerate(layers):
        qkv = ((_rms64(x, 1e-6) * w["g1"].to(F64)) @ _dense64(w["qkv"], fmt).T).reshape(-1, heads + 2 * kv, d)
        q, k, v = _rope64(qkv[:, :heads], pos), _rope64(qkv[:, heads:heads + kv], pos), qkv[:, heads + kv:]
        out = torch.empty(x.shape[0], heads, d, dtype=F64, device=DEV)
        for b, (page, row) in enumerate(rows):
            t = slice(start[b], start[b + 1])
            k_out[li, page[hist[b]:], :, row[hist[b]:]] = k[t]
            v_out[li, page[hist[b]:], :, row[hist[b]:]] = v[t]
            out[t] = _causal64(q[t], k_out[li, page, :, row], v_out[li, page, :, row], d ** -0.5, hist[b], tiny=1e-6)
        x = x + out.reshape(-1, heads * d) @ _dense64(w["o"], fmt).T
        gu = (_rms64(x, 1e-6) * w["g2"].to(F64)) @ _dense64(w["gate_up"], fmt).T
        x = x + (torch.nn.functional.silu(gu[:, :inter]) * gu[:, inter:]) @ _dense64(w["down"], fmt).T
    return x, k_out, v_out


def _work_llama(case):
    h, heads, kv, inter = LLAMA[case["model"]]
    params = case["layers"] * ((heads + 2 * kv) * HEAD_DIM * h + heads * HEAD_DIM * h + 3 * h * inter)
    size = 4 if case["fmt"] == "fp32" else 2
    per_weight = {"fp8": 1.0, "int4": 0.5 + 3.0 / GROUP}.get(case["fmt"], size)
    if case["path"] == "decode":
        b, c = case["batch"], case["ctx"]
        hist = [c] * b if not case["paged"] or b == 1 else [max(1, c * (8 * (b - 1) - 7 * i) // (8 * (b - 1))) for i in range(b)]
        new = [1] * b
    else:
        new = _ints(case["lens"])
        hist = [a + n for a, n in zip(_ints(case["hist"]), new)]
    pairs = sum(n * (t - n) + n * (n + 1) // 2 for n, t in zip(new, hist))
    tokens = sum(new)
    return dict(bytes=params * per_weight + size * (case["layers"] * 2 * kv * HEAD_DIM * (sum(hist) + tokens) + 2 * tokens * h),
                flops=2.0 * params * tokens + 4.0 * case["layers"] * heads * HEAD_DIM * pairs)


# ------------------------------------------------------------------------------------------------ the tail of a decode step
def _head_inputs(case, seed):
    r = _Random(seed)
    dt = TYPES[case["fmt"]]
    h = case["hidden"]
    return r.normal(case["batch"], h, std=2.0, dtype=dt), r.normal(h, std=0.1, mean=1.0, dtype=dt), r.normal(case["vocab"], h, std=2.0 / math.sqrt(h), dtype=dt)


def _prepare_head(case, seed):
    m = _pkg()
    hidden, gamma, head = _head_inputs(case, seed)
    b, k = case["batch"], case["k"]
    code = {torch.bfloat16: m.BF16, torch.float16: m.F16}[hidden.dtype]
    engine = m.Decoder(m.DecoderConfig(case["hidden"], case["hidden"] // HEAD_DIM, case["hidden"] // HEAD_DIM, HEAD_DIM, 2048, 1, 64, b, code, m.W_DENSE, GROUP, 1e-6,
                                       HEAD_DIM, 10000.0, 1, 0), DEV)
    z = lambda *s, dtype=torch.int32: torch.zeros(*s, dtype=dtype, device=DEV)  # noqa: E731
    bufs = dict(logits=z(b, case["vocab"], dtype=torch.float32), tmp_ids=z(b, m.TOPK_BLOCKS, k), tmp_vals=z(b, m.TOPK_BLOCKS, k, dtype=torch.float32), topk_ids=z(b, k),
                topk_vals=z(b, k, dtype=torch.float32), seq_len=z(b), finished=z(b, dtype=torch.uint8), output_id=z(b))
    return dict(case=case, engine=engine, hidden=hidden, gamma=gamma, head=head, bufs=bufs, step=17 + seed % 1000)


def _run_head(s):
    b = s["bufs"]
    s["engine"].lm_head_topk_sample(s["hidden"], s["gamma"], s["head"], b, s["case"]["k"], s["step"], 2)
    return b["logits"], b["topk_ids"], b["topk_vals"], b["output_id"], b["seq_len"], b["finished"]


def _exact_head(case, seed):
    hidden, gamma, head = _head_inputs(case, seed)
    logits = (_rms64(hidden.to(F64), 1e-6) * gamma.to(F64)) @ head.to(F64).T
    top = torch.topk(logits, case["k"], -1).values
    return logits, None, torch.exp(top - top[:, :1]), None, None, None  # the sampler leaves the weights in the place of the values


def _work_head(case):
    b, h, v = case["batch"], case["hidden"], case["vocab"]
    return dict(bytes=2.0 * v * h + 4.0 * b * v + 2.0 * b * h, flops=2.0 * b * v * h)


# ------------------------------------------------------------------------------------------------ layer-list models
def _matrix(r, out, inn, gain=1.0):
    return r.normal(out, inn, std=gain / math.sqrt(inn))


def _vasolix(case, seed):
    z = VASOLIX[case["size"]]
    w = z["width"]
    mlp = {"kind": "moe", "expert": {"ff": z["ff"]}, "router": {"experts": z["experts"], "top": z["top"]}, "shared": {"ff": z["shared"]}}
    gla = {"type": "gla", "mixer": {"heads": z["g_heads"], "dim": z["g_dim"], "vdim": z["g_vdim"], "tau": 16.0}, "mlp": mlp}
    att = {"type": "attention", "mixer": {"heads": z["heads"], "kv_heads": z["kv_heads"], "dim": HEAD_DIM, "vdim": HEAD_DIM, "scale": HEAD_DIM ** -0.5,
                                          "mask": {"size": z["chunk"]}}, "mlp": mlp}
    config = {"architecture": "Vasolix", "layers": [gla, att, gla, att], "norm": {"eps": 1e-6}, "vocab": 32000, "width": w}
    r = _Random(seed)
    t = {"embed": r.normal(32000, w, dtype=torch.float32), "head": _matrix(r, 32000, w), "final.norm": r.normal(w, std=0.1, mean=1.0)}
    for i, layer in enumerate(config["layers"]):
        p, mx = f"l{i}.", layer["mixer"]
        H, d, dv = mx["heads"], mx["dim"], mx["vdim"]
        t[p + "norm1"], t[p + "norm2"] = r.normal(w, std=0.1, mean=1.0), r.normal(w, std=0.1, mean=1.0)
        if layer["type"] == "attention":
            g = mx["kv_heads"]
            t.update({p + "mix.q": _matrix(r, H * d, w), p + "mix.k": _matrix(r, g * d, w), p + "mix.g": _matrix(r, H * d, w), p + "mix.o": _matrix(r, w, H * d),
                      p + "mix.q.norm": r.normal(H * d, std=0.1, mean=1.0), p + "mix.k.norm": r.normal(g * d, std=0.1, mean=1.0), p + "mix.sink": r.normal(H)})
        else:
            t.update({p + "mix.q": _matrix(r, H * d, w), p + "mix.k": _matrix(r, H * d, w), p + "mix.v": _matrix(r, H * dv, w), p + "mix.g": _matrix(r, H * dv, w),
                      p + "mix.o": _matrix(r, w, H * dv), p + "mix.a1": _matrix(r, z["rank"], w), p + "mix.a2": _matrix(r, H * d, z["rank"], 2.0),
                      p + "mix.a2.b": r.normal(H * d, std=1.5, mean=1.0), p + "mix.norm": r.normal(dv, std=0.1, mean=1.0)})
        router = t[p + "mlp.router"] = _matrix(r, z["experts"], w, 0.25)
        # a trained router is sure of most tokens: every token's embedding has a part along the rows of the experts that are meant for it
        meant = torch.zeros(32000, z["experts"], device=DEV).scatter_(1, torch.topk(r.uniform(32000, z["experts"], dtype=torch.float32), z["top"], -1).indices, 28.0)
        t["embed"] = t["embed"] + meant @ torch.nn.functional.normalize(router.float(), dim=-1)
        up, down = _stack(r, z["experts"], z["ff"], w), _stack(r, z["experts"], w, z["ff"])
        for e in range(z["experts"]):
            t[f"{p}mlp.e{e}.up"], t[f"{p}mlp.e{e}.down"] = up[e], down[e]
        t.update({p + "mlp.shared.up": _matrix(r, z["shared"], w), p + "mlp.shared.down": _matrix(r, w, z["shared"]), p + "mlp.shared.sg": _matrix(r, 1, w)})
    t["embed"] = t["embed"].to(torch.bfloat16)
    return config, t, r


def _stack(r, n, out, inn):
    return r.normal(n, out, inn, std=1.0 / math.sqrt(inn))


def _zefenex(case, seed):
    z = ZEFENEX[case["size"]]
    w, H, rank, d, dr, ff = z["width"], z["heads"], z["rank"], 128, 64, z["ff"]
    layer = {"type": "latent_attention", "mixer": {"heads": H, "dim": d, "rot_dim": dr, "vdim": d, "kv_rank": rank, "scale": (d + dr) ** -0.5, "mask": {"size": z["window"]},
                                                   "rot": {"base": 10000.0, "dims": dr}}, "mlp": {"kind": "dense", "ff": ff}}
    config = {"architecture": "Zefenex", "embedding": {"scale": 1.0}, "layers": [layer], "logit_softcap": 30.0, "norm": {"eps": 1e-6}, "vocab": LAYER_VOCAB, "width": w}
    r = _Random(seed)
    t = {"embed": r.normal(LAYER_VOCAB, w, std=0.4), "head": _matrix(r, LAYER_VOCAB, w, 3.0)}
    for name in ("l0.norm1", "l0.norm1b", "l0.norm2", "l0.norm2b", "final.norm"):
        t[name], t[name + ".b"], t[name + ".alpha"] = r.normal(w, std=0.2, mean=1.0), r.normal(w, std=0.1), r.uniform(1, lo=0.6, hi=0.9)[0]
    t.update({"l0.ls1": r.normal(w, std=0.2, mean=0.8), "l0.ls2": r.normal(w, std=0.2, mean=0.8), "l0.mix.q": _matrix(r, H * (d + dr), w, 2.0),
              "l0.mix.g": _matrix(r, H * d, w), "l0.mix.o": _matrix(r, w, H * d), "l0.mix.uk": _matrix(r, H * d, rank), "l0.mix.uv": _matrix(r, H * d, rank),
              "l0.mix.sink": r.normal(H, mean=0.5), "l0.mix.dkv": _matrix(r, rank + dr, w, 2.0), "l0.mix.dkv.norm": r.normal(rank, std=0.2, mean=1.0),
              "l0.mlp.up": _matrix(r, ff, w), "l0.mlp.up.b": r.normal(ff, std=0.3), "l0.mlp.down": _matrix(r, w, ff), "l0.mlp.down.b": r.normal(w, std=0.3)})
    return config, t, r


def _fedovik(case, seed):
    z = FEDOVIK[case["size"]]
    w, ff, H, g, d = z["width"], z["ff"], z["heads"], z["kv_heads"], HEAD_DIM
    rh, rd, rv, rank = z["r_heads"], z["r_dim"], z["r_vdim"], z["rank"]
    left = dict(heads=H, kv_heads=g, dim=d, vdim=d, scale=d ** -0.5, mask=dict(size=z["window"]))
    right = dict(heads=rh, kv_heads=rh, dim=rd, vdim=rv, conv=4)
    layer = {"type": "parallel", "mixer": dict(left=left, right=right, left_scale=0.8, right_scale=0.9), "mlp": {"kind": "dense", "ff": ff}}
    config = {"architecture": "Fedovik", "layers": [layer], "norm": {"eps": 1e-5}, "embedding": {"scale": 1.0}, "vocab": LAYER_VOCAB, "width": w}
    r = _Random(seed)
    t = {"embed": r.normal(LAYER_VOCAB, w), "final.norm": r.normal(w, std=0.1, mean=1.0), "final.norm.b": r.normal(w, std=0.1),
         "l0.norm1": r.normal(w, std=0.1, mean=1.0), "l0.norm1.b": r.normal(w, std=0.1), "l0.mlp.gate": _matrix(r, ff, w), "l0.mlp.up": _matrix(r, ff, w),
         "l0.mlp.down": _matrix(r, w, ff)}
    p = "l0.mix.left."
    t.update({p + "q": _matrix(r, H * d, w), p + "k": _matrix(r, g * d, w), p + "v": _matrix(r, g * d, w), p + "o": _matrix(r, w, H * d), p + "q.b": r.normal(H * d, std=0.3),
              p + "k.b": r.normal(g * d, std=0.3), p + "v.b": r.normal(g * d, std=0.1), p + "q.norm": r.normal(d, std=0.2, mean=1.0), p + "k.norm": r.normal(d, std=0.2, mean=1.0),
              p + "r1": r.uniform(H, lo=0.2, hi=1.2), p + "r2": r.uniform(H, lo=0.5, hi=1.5)})
    p = "l0.mix.right."
    t.update({p + "q": _matrix(r, rh * rd, w), p + "k": _matrix(r, rh * rd, w), p + "v": _matrix(r, rh * rv, w), p + "b": _matrix(r, rh, w), p + "o": _matrix(r, w, rh * rv),
              p + "q.conv": r.normal(rh * rd, 4, std=0.6), p + "k.conv": r.normal(rh * rd, 4, std=0.6), p + "v.conv": r.normal(rh * rv, 4, std=0.6),
              p + "a1": _matrix(r, rank, w), p + "a2": _matrix(r, rh * rd, rank, 2.0), p + "dt_bias": r.normal(rh * rd, mean=-1.0), p + "A_log": r.uniform(rh, lo=-1.5, hi=0.5),
              p + "g1": _matrix(r, rank, w), p + "g2": _matrix(r, rh * rv, rank, 2.0), p + "norm": r.normal(rv, std=0.2, mean=1.0)})
    return config, t, r


_MODELS = {"vasolix": (_vasolix, "VasolixModel"), "zefenex": (_zefenex, "ZefenexModel"), "fedovik": (_fedovik, "FedovikModel")}


def _list_inputs(case, seed):
    """(config, tensors, prompts, the token after each): host lists of ids, as a tokenizer gives them."""
    config, tensors, r = _MODELS[case["path"]][0](case, seed)
    lens = _ints(case["lens"])
    ids = r.ints(0, config["vocab"], sum(lens) + len(lens)).tolist()
    prompts, at = [], 0
    for n in lens:
        prompts.append(ids[at:at + n])
        at += n
    return config, tensors, prompts, ids[at:]


def _prepare_list(case, seed):
    config, tensors, prompts, after = _list_inputs(case, seed)
    lens, n = [len(p) for p in prompts], len(prompts)
    per = max(lens) // PAGE + 1
    decode = case.get("decode", False)
    model = getattr(_pkg(".models." + case["path"]), _MODELS[case["path"]][1])(
        config, tensors, dtype=TYPES[case["dtype"]], device=DEV, max_tokens=max(lens) if decode else sum(lens), max_seqs=n, max_pages_per_seq=per)
    eng = model.engine
    eng.set_pools(per * n, n)
    table = np.random.default_rng(seed).permutation(per * n).astype(np.int32).reshape(n, per)
    i32 = lambda v: np.asarray(v, dtype=np.int32)  # noqa: E731
    s = dict(case=case, model=model, engine=eng, trace=case["path"] != "vasolix", decode=decode)
    starts = np.cumsum([0] + lens)
    s["prompt"] = (i32(sum(prompts, [])), i32(starts), i32([0] * n), i32(range(n)), table.reshape(-1), i32(starts[1:] - 1))
    s["next"] = (i32(after), i32(range(n + 1)), i32(lens), i32(range(n)), table.reshape(-1), i32(range(n)))
    if decode:
        for b, p in enumerate(prompts):
            eng.forward(p, [0, len(p)], [0], [b], table[b], [])
    return s


def _run_list(s):
    e, trace = s["engine"], s["trace"]
    after = None
    if not s["decode"]:
        after = e.forward(*s["prompt"], trace=trace)
    return after, e.forward(*s["next"], trace=trace)


def _padded(prompts, after):
    n = max(len(p) for p in prompts) + 1
    ids = torch.tensor([p + [a] + [0] * (n - len(p) - 1) for p, a in zip(prompts, after)], device=DEV)
    return ids, [len(p) for p in prompts]


def _lin(x, w):
    return x @ w.to(F64).T


def _attend(rows, q, k, v, **kw):
    """Every sequence's causal attention; past a sequence's end its rows are padding that nothing reads."""
    out = torch.zeros(*q.shape[:-1], v.shape[-1], dtype=F64, device=q.device)
    for b, n in enumerate(rows):
        out[b, :n + 1] = _causal64(q[b, :n + 1], k[b, :n + 1], v[b, :n + 1], start=0, **kw)
    return out


def _vasolix64(config, t, ids, rows):
    eps = 1e-6
    B, T = ids.shape
    x = t["embed"][ids].to(F64)
    for i, layer in enumerate(config["layers"]):
        p, mx, ml = f"l{i}.mix.", layer["mixer"], layer["mlp"]
        H, d, dv = mx["heads"], mx["dim"], mx["vdim"]
        if layer["type"] == "attention":
            g, size = mx["kv_heads"], mx["mask"]["size"]
            q, k = _lin(x, t[p + "q"]), _lin(x, t[p + "k"])
            qn, kn = (_rms64(q, eps) * t[p + "q.norm"].to(F64)).reshape(B, T, H, d), (_rms64(k, eps) * t[p + "k.norm"].to(F64)).reshape(B, T, g, d)
            o = _attend(rows, qn, kn, k.reshape(B, T, g, d), scale=mx["scale"], see=lambda a, c: a // size == c // size, sink=t[p + "sink"].to(F64))
            y = _lin(o.reshape(B, T, H * d) * torch.sigmoid(_lin(x, t[p + "g"])), t[p + "o"])
        else:
            q, k, v = _lin(x, t[p + "q"]).reshape(B, T, H, d) / math.sqrt(d), _lin(x, t[p + "k"]).reshape(B, T, H, d), _lin(x, t[p + "v"]).reshape(B, T, H, dv)
            a = (torch.sigmoid(_lin(_lin(x, t[p + "a1"]), t[p + "a2"]) + t[p + "a2.b"].to(F64)) ** (1.0 / mx["tau"])).reshape(B, T, H, d)
            S = torch.zeros(B, H, d, dv, dtype=F64, device=DEV)
            o = torch.empty(B, T, H, dv, dtype=F64, device=DEV)
            for n in range(T):
                S.mul_(a[:, n, :, :, None]).add_(k[:, n, :, :, None] * v[:, n, :, None])
                o[:, n] = torch.matmul(q[:, n, :, None], S)[:, :, 0]
            gate = _lin(x, t[p + "g"])
            y = _lin((_rms64(o, eps) * t[p + "norm"].to(F64)).reshape(B, T, H * dv) * torch.nn.functional.silu(gate), t[p + "o"])
        x = x + _rms64(y, eps) * t[f"l{i}.norm1"].to(F64)
        p = f"l{i}.mlp."
        h = x.reshape(B * T, -1)
        weight, chosen = torch.topk(torch.sigmoid(_lin(h, t[p + "router"])), ml["router"]["top"], -1)
        y = _lin(torch.relu(_lin(h, t[p + "shared.up"])) ** 2, t[p + "shared.down"]) * torch.sigmoid(_lin(h, t[p + "shared.sg"]))
        for e in range(ml["router"]["experts"]):
            token, slot = (chosen == e).nonzero(as_tuple=True)
            y.index_add_(0, token, _lin(torch.relu(_lin(h[token] * weight[token, slot][:, None], t[f"{p}e{e}.up"])) ** 2, t[f"{p}e{e}.down"]))
        x = x + (_rms64(y, eps) * t[f"l{i}.norm2"].to(F64)).reshape(B, T, -1)
    return x, lambda rows_of_x: _lin(_rms64(rows_of_x, eps) * t["final.norm"].to(F64), t["head"])


def _zefenex64(config, t, ids, rows):
    B, T = ids.shape
    mx = config["layers"][0]["mixer"]
    H, d, dr, r = mx["heads"], mx["dim"], mx["rot_dim"], mx["kv_rank"]
    dyt = lambda v, n: torch.tanh(t[n + ".alpha"].to(F64) * v) * t[n].to(F64) + t[n + ".b"].to(F64)  # noqa: E731
    pos = torch.arange(T, device=DEV)
    turn = lambda v: torch.stack([_rope64(v[b], pos) for b in range(B)])  # noqa: E731
    x = t["embed"][ids].to(F64)
    h, p = dyt(x, "l0.norm1"), "l0.mix."
    q = _lin(h, t[p + "q"]).reshape(B, T, H, d + dr)
    down = _lin(h, t[p + "dkv"])
    c = _rms64(down[..., :r], 1e-6) * t[p + "dkv.norm"].to(F64)
    kr = turn(down[..., r:].reshape(B, T, 1, dr)).expand(B, T, H, dr)
    k, v = torch.cat((_lin(c, t[p + "uk"]).reshape(B, T, H, d), kr), -1), _lin(c, t[p + "uv"]).reshape(B, T, H, d)
    q = torch.cat((q[..., :d], turn(q[..., d:])), -1)
    o = _attend(rows, q, k, v, scale=mx["scale"], see=lambda i, j: i - j < mx["mask"]["size"], sink=t[p + "sink"].to(F64))
    y = _lin(o.reshape(B, T, H * d) * torch.sigmoid(_lin(h, t[p + "g"])), t[p + "o"])
    x = x + t["l0.ls1"].to(F64) * dyt(y, "l0.norm1b")
    h, p = dyt(x, "l0.norm2"), "l0.mlp."
    y = _lin(torch.relu(_lin(h, t[p + "up"]) + t[p + "up.b"].to(F64)) ** 2, t[p + "down"]) + t[p + "down.b"].to(F64)
    x = x + t["l0.ls2"].to(F64) * dyt(y, "l0.norm2b")
    return x, lambda rows_of_x: 30.0 * torch.tanh(_lin(dyt(rows_of_x, "final.norm"), t["head"]) / 30.0)


def _fedovik64(config, t, ids, rows):
    B, T = ids.shape
    eps = 1e-5
    ln = lambda v, n: (v - v.mean(-1, keepdim=True)) * torch.rsqrt(v.var(-1, unbiased=False, keepdim=True) + eps) * t[n].to(F64) + t[n + ".b"].to(F64)  # noqa: E731
    mx = config["layers"][0]["mixer"]
    x = t["embed"][ids].to(F64)
    y = ln(x, "l0.norm1")
    a, p = mx["left"], "l0.mix.left."
    H, g, d = a["heads"], a["kv_heads"], a["dim"]
    biased = lambda n: _lin(y, t[p + n]) + t[p + n + ".b"].to(F64)  # noqa: E731
    q = _rms64(biased("q").reshape(B, T, H, d), eps) * t[p + "q.norm"].to(F64)
    k = _rms64(biased("k").reshape(B, T, g, d), eps) * t[p + "k.norm"].to(F64)
    r1, r2 = t[p + "r1"].to(F64), t[p + "r2"].to(F64)
    o = _attend(rows, q, k, biased("v").reshape(B, T, g, d), scale=a["scale"], see=lambda i, j: i - j < a["mask"]["size"],
                bias=lambda h, dist: -r1[h] * torch.log1p(r2[h] * dist.to(F64)))
    left = _lin(o.reshape(B, T, H * d), t[p + "o"])
    a, p = mx["right"], "l0.mix.right."
    H, d, dv = a["heads"], a["dim"], a["vdim"]

    def conv(n):  # four causal taps per channel, then silu
        z, taps = torch.nn.functional.pad(_lin(y, t[p + n]), (0, 0, 3, 0)), t[p + n + ".conv"].to(F64)
        return torch.nn.functional.silu(sum(z[:, j:j + T] * taps[:, j] for j in range(4)))

    unit = lambda v: v * torch.rsqrt(v.square().sum(-1, keepdim=True) + 1e-6)  # noqa: E731
    q, k, v = unit(conv("q").reshape(B, T, H, d)) * d ** -0.5, unit(conv("k").reshape(B, T, H, d)), conv("v").reshape(B, T, H, dv)
    beta = torch.sigmoid(_lin(y, t[p + "b"]))
    step = torch.nn.functional.softplus(_lin(_lin(y, t[p + "a1"]), t[p + "a2"]) + t[p + "dt_bias"].to(F64)).reshape(B, T, H, d)
    decay = torch.exp(-torch.exp(t[p + "A_log"].to(F64))[:, None] * step)
    S = torch.zeros(B, H, d, dv, dtype=F64, device=DEV)
    o = torch.empty(B, T, H, dv, dtype=F64, device=DEV)
    for n in range(T):
        S.mul_(decay[:, n, :, :, None])
        u = beta[:, n, :, None] * (v[:, n] - torch.matmul(k[:, n, :, None], S)[:, :, 0])
        S.add_(k[:, n, :, :, None] * u[:, :, None])
        o[:, n] = torch.matmul(q[:, n, :, None], S)[:, :, 0]
    gate = torch.sigmoid(_lin(_lin(y, t[p + "g1"]), t[p + "g2"])).reshape(B, T, H, dv)
    right = _lin((_rms64(o, eps) * t[p + "norm"].to(F64) * gate).reshape(B, T, H * dv), t[p + "o"])
    ff = _lin(torch.relu(_lin(y, t["l0.mlp.gate"])) * _lin(y, t["l0.mlp.up"]), t["l0.mlp.down"])
    x = x + mx["left_scale"] * left + mx["right_scale"] * right + ff
    return x, lambda rows_of_x: _lin(ln(rows_of_x, "final.norm"), t["embed"])


def _exact_list(case, seed):
    config, t, prompts, after = _list_inputs(case, seed)
    ids, rows = _padded(prompts, after)
    x, head = {"vasolix": _vasolix64, "zefenex": _zefenex64, "fedovik": _fedovik64}[case["path"]](config, t, ids, rows)
    ends = torch.stack([x[b, n - 1] for b, n in enumerate(rows)])
    new = torch.stack([x[b, n] for b, n in enumerate(rows)])
    if case["path"] == "vasolix":
        return None if case["decode"] else head(ends), head(new)
    return (head(ends), torch.cat([x[b, :n] for b, n in enumerate(rows)])[None]), (head(new), new[None])


def _seen(first, last, window=0, chunk=0):
    """Keys seen by the queries at positions first .. last - 1."""
    i = np.arange(first, last, dtype=np.int64)
    keys = i % chunk + 1 if chunk else i + 1
    return float((np.minimum(keys, window) if window else keys).sum())


def _work_list(case):
    lens, decode = _ints(case["lens"]), case.get("decode", False)
    n = len(lens)
    passes = ([] if decode else [[(0, t) for t in lens]]) + [[(t, t + 1) for t in lens]]
    total = dict(bytes=0.0, flops=0.0)
    for spans in passes:
        tokens = sum(b - a for a, b in spans)
        if case["path"] == "vasolix":
            z = VASOLIX[case["size"]]
            w = z["width"]
            att = w * (2 * z["heads"] + z["kv_heads"]) * HEAD_DIM + z["heads"] * HEAD_DIM * w
            gd, gv = z["g_heads"] * z["g_dim"], z["g_heads"] * z["g_vdim"]
            gla = w * (2 * gd + 2 * gv + z["rank"]) + z["rank"] * gd + gv * w
            touched, router = min(z["experts"], tokens * z["top"]), w * (z["experts"] + 1)
            keys = sum(_seen(a, b, chunk=z["chunk"]) for a, b in spans)
            rows = sum(min(b, z["chunk"]) if a == 0 else a % z["chunk"] + 1 for a, b in spans)
            state = 4.0 * n * z["g_heads"] * z["g_dim"] * z["g_vdim"]
            total["bytes"] += 2.0 * (2 * att + 2 * gla + 4 * (2 * w * (touched * z["ff"] + z["shared"]) + router) + 32000 * w)
            total["bytes"] += 2 * 2.0 * (2 * z["kv_heads"] * HEAD_DIM * rows) + 2 * state * (1 if spans[0][0] == 0 else 2) + 4.0 * n * 32000
            total["flops"] += 2.0 * tokens * (2 * att + 2 * gla + 4 * (2 * w * (z["top"] * z["ff"] + z["shared"]) + router)) + 2.0 * n * 32000 * w
            total["flops"] += 2 * 4.0 * z["heads"] * HEAD_DIM * keys + 2 * 5.0 * tokens * z["g_heads"] * z["g_dim"] * z["g_vdim"]
        elif case["path"] == "zefenex":
            z = ZEFENEX[case["size"]]
            w, H, r, d, dr = z["width"], z["heads"], z["rank"], 128, 64
            params = w * H * (d + dr) + 2 * w * H * d + w * (r + dr) + 2 * H * d * r + 2 * w * z["ff"]
            rows = sum(min(b, z["window"]) if a else b for a, b in spans)
            total["bytes"] += 2.0 * (params + LAYER_VOCAB * w + (r + dr) * rows) + 4.0 * tokens * w + 4.0 * n * LAYER_VOCAB
            total["flops"] += 2.0 * (tokens * params + n * LAYER_VOCAB * w) + 2.0 * H * (d + dr + d) * sum(_seen(a, b, window=z["window"]) for a, b in spans)
        else:
            z = FEDOVIK[case["size"]]
            w, H, g, d, rh, rd, rv, rank = z["width"], z["heads"], z["kv_heads"], HEAD_DIM, z["r_heads"], z["r_dim"], z["r_vdim"], z["rank"]
            params = w * (2 * H + 2 * g) * d + w * (2 * rh * rd + 2 * rh * rv + rh + 2 * rank) + rank * rh * (rd + rv) + 3 * w * z["ff"]
            rows = sum(min(b, z["window"]) if a else b for a, b in spans)
            state = 4.0 * n * rh * rd * rv
            total["bytes"] += 2.0 * (params + LAYER_VOCAB * w + 2 * g * d * rows) + 4.0 * tokens * w + 4.0 * n * LAYER_VOCAB + state * (1 if spans[0][0] == 0 else 2)
            total["flops"] += 2.0 * (tokens * params + n * LAYER_VOCAB * w) + 4.0 * H * d * sum(_seen(a, b, window=z["window"]) for a, b in spans) + 7.0 * tokens * rh * rd * rv
    return total


# ------------------------------------------------------------------------------------------------ what is asked of this file
def prepare(case, seed):
    return {"decode": _prepare_llama, "prefill": _prepare_llama, "head": _prepare_head}.get(case["path"], _prepare_list)(case, seed)


def run(state):
    return {"decode": _run_llama, "prefill": _run_llama, "head": _run_head}.get(state["case"]["path"], _run_list)(state)


def exact(case, seed):
    return {"decode": _exact_llama, "prefill": _exact_llama, "head": _exact_head}.get(case["path"], _exact_list)(case, seed)


def work(case):
    return {"decode": _work_llama, "prefill": _work_llama, "head": _work_head}.get(case["path"], _work_list)(case)


def tolerance(case):
    """About four times what a path differs from 64 bits by: the rounding of its data type, over the layers that the rounding travels through."""
    if case.get("fmt") == "fp32":
        return {"rel": 1.5e-6}
    half = (case.get("dtype") or case["fmt"]) == "fp16"  # three more bits than bfloat16
    rel = {"decode": 2e-2, "prefill": 2e-2, "head": 1.5e-2, "vasolix": 2e-2, "zefenex": 1e-2, "fedovik": 1e-2}[case["path"]]
    return {"rel": rel / 8 if half else rel}
