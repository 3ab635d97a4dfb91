"""Experts of a few tokens, the router's product and the grouping of pairs (csrc/moe.cu) at the edges of their ranges: 1, 8, 9, 16 and 17 tokens, inner
sizes that do not share out evenly over the warps, more experts than lanes, every token choosing the same experts; against the float64 restatement."""
import importlib
import math

import numpy as np
import pytest
import torch

import vasolix_oracle as ref

pytestmark = pytest.mark.gpu


def ambiguous_rows(monkeypatch, config, W, toks, u):
    """-> (the oracle's logits, which tokens a 16-bit router may send elsewhere).  A logit is a sum of products x_i w_i whose x has been rounded three times (u
    each) on its way: its standard error is below sqrt(3) u |x * w|, and a choice is open where the last chosen and the first left out are within four of
    their difference's."""
    open_rows, plain = [], ref.route

    def spy(h, W, p, ml):
        w, top = W[p + "router"], ml["router"]["top"]
        logits = torch.sort(h @ w.T, descending=True, dim=-1).values
        if top < w.shape[0]:
            error = math.sqrt(6) * u * (h ** 2 @ (w ** 2).T).max(-1).values.sqrt()
            open_rows.append(logits[:, top - 1] - logits[:, top] < 4 * error)
        else:
            open_rows.append(torch.zeros(len(h), dtype=torch.bool))
        return plain(h, W, p, ml)

    with monkeypatch.context() as m:
        m.setattr(ref, "route", spy)
        want = ref.forward(config, W, toks).numpy()
    return want, torch.stack(open_rows).any(0).numpy()


@pytest.mark.parametrize("dtype,tol,u", [("bfloat16", 4e-2, 2.0 ** -8), ("float16", 6e-3, 2.0 ** -11)])
@pytest.mark.parametrize("width,ff,experts,top", [(64, 64, 5, 2), (512, 96, 40, 3), (544, 224, 7, 7), (1024, 512, 70, 4), (2080, 64, 3, 1)])
def test_experts_of_few_tokens(monkeypatch, dtype, tol, u, width, ff, experts, top):
    layer = ref.attention_layer(heads=2, kv_heads=1, dim=16, size=50, mlp=ref.moe(experts=experts, top=top, ff=ff, shared_ff=64))
    config = ref.make_config([layer], width=width, vocab=80)
    W, packed = ref.make_weights(config, seed=2)
    model = importlib.import_module("llm-inference-engine_b200.models.vasolix").VasolixModel(config, packed, dtype=dtype, device="cuda:0", max_tokens=128, max_seqs=20,
                                                                                              max_pages_per_seq=2)
    serving = importlib.import_module("llm-inference-engine_b200.serving")
    for n in (1, 8, 9, 16, 17, 100):
        toks = np.random.default_rng(n).integers(0, 80, n).tolist()
        sess = serving.Session(model, 2560, max_seqs=20, max_batch_tokens=128, poison=True)
        got = sess.feed([(sess.open(), toks, range(n))]).cpu().numpy()
        want, open_rows = ambiguous_rows(monkeypatch, config, W, toks, u)
        assert not np.isnan(got).any()
        err = np.linalg.norm(got - want, axis=-1) / np.linalg.norm(want, axis=-1)
        assert (err[~open_rows] < tol).all(), (n, err, open_rows)
        assert open_rows.mean() <= (0.0 if experts == top else 0.6 if n >= 8 else 1.0), (n, open_rows)


def ordered(h, W, p, ml):
    """The router's choice among equals and among what is not finite: the largest logits, of equals the smaller index first; minus infinity and NaN have no weight
    (which of them is chosen makes no difference: a NaN is left out here, and expert 0 stands in its place)."""
    logits, top = (h @ W[p + "router"].T).tolist(), ml["router"]["top"]
    chosen, weight = torch.zeros(len(logits), top, dtype=torch.long), torch.zeros(len(logits), top, dtype=torch.float64)
    for t, row in enumerate(logits):
        for k, e in enumerate(sorted((e for e in range(len(row)) if row[e] == row[e]), key=lambda e: (-row[e], e))[:top]):
            chosen[t, k], weight[t, k] = e, 0.0 if row[e] == -math.inf else 1.0 / (1.0 + math.exp(-row[e]))
    return chosen, weight


@pytest.mark.parametrize("dtype,tol", [("bfloat16", 4e-2), ("float16", 6e-3), ("float32", 2e-5)])
@pytest.mark.parametrize("experts,top", [(3, 3), (7, 4), (32, 6), (33, 6), (128, 6), (200, 4)])
def test_choices_among_equals_and_what_is_not_finite(monkeypatch, dtype, tol, experts, top):
    """Every routing kernel of csrc/moe.cu: decode batches (16-bit, up to 64 tokens), prompts from 512 tokens on, and what lies between.  A router row has one weight, on
    a channel that is large and of either sign: equal weights give equal logits, 0 and -0 too, an infinite one plus or minus infinity, a NaN NaN."""
    layer = ref.attention_layer(heads=2, kv_heads=1, dim=16, size=50, mlp=ref.moe(experts=experts, top=top, ff=32, shared_ff=32))
    config = ref.make_config([layer], width=64, vocab=80)
    W, packed = ref.make_weights(config, seed=4)
    values = ([math.nan, 0.25, math.inf] if experts == 3 else [math.nan, 0.5, -0.0, 0.5, 0.0, -0.5, math.inf] if experts == 7 else
              [0.5, -0.5, math.nan, 0.0, math.inf, -0.0, -0.5, 0.5, 0.0, 0.0, 0.25, -math.inf, math.inf] + [[0.0, 0.25, -0.25, -0.0][e % 4] for e in range(13, experts)])
    router = torch.zeros(experts, 64)
    router[:, 5] = torch.tensor(values)
    packed["l0.mlp.router"] = router.to(torch.bfloat16)
    packed["embed"][:, 5] = torch.where(torch.arange(80) % 3 == 0, -4.0, 4.0).to(torch.bfloat16)
    for name in ("l0.mlp.router", "embed"):
        W[name] = packed[name].to(torch.float64)
    model = importlib.import_module("llm-inference-engine_b200.models.vasolix").VasolixModel(config, packed, dtype=dtype, device="cuda:0", max_tokens=640, max_seqs=2,
                                                                                              max_pages_per_seq=10)
    serving = importlib.import_module("llm-inference-engine_b200.serving")
    monkeypatch.setattr(ref, "route", ordered)
    for n in (1, 2, 9, 40, 64, 65, 512, 600):
        toks = np.random.default_rng(n).integers(0, 80, n).tolist()
        sess = serving.Session(model, 1280, max_seqs=2, max_batch_tokens=640, poison=True)
        got = sess.feed([(sess.open(), toks, range(n))]).cpu().numpy()
        want = ref.forward(config, W, toks).numpy()
        err = np.linalg.norm(got - want, axis=-1) / np.linalg.norm(want, axis=-1)
        assert (err < tol).all(), (n, err.max())


@pytest.mark.parametrize("dtype,tol,u", [("bfloat16", 4e-2, 2.0 ** -8), ("float16", 6e-3, 2.0 ** -11)])
@pytest.mark.parametrize("experts,top", [(40, 4), (256, 2), (8, 4), (32, 8), (12, 4)])
def test_sparse_choices_of_decode_batches(monkeypatch, dtype, tol, u, experts, top):
    """Up to 64 tokens whose choices scatter over the experts: tiles of one row to about thirty, in passes of eight rows or sixteen (12 and 32 experts: either, by the
    number of tokens); every row whose choice is not open within 16-bit rounding.  The embeddings lean towards the router's rows, so that most choices are sure."""
    layer = ref.attention_layer(heads=2, kv_heads=1, dim=16, size=50, mlp=ref.moe(experts=experts, top=top, ff=96, shared_ff=64))
    config = ref.make_config([layer], width=512, vocab=80)
    W, packed = ref.make_weights(config, seed=3)
    gen = torch.Generator().manual_seed(experts)
    router = W["l0.mlp.router"]
    meant = torch.stack([torch.randperm(experts, generator=gen)[:top] for _ in range(80)])
    lean = torch.zeros(80, experts, dtype=torch.float64).scatter_(1, meant, 12.0) @ torch.nn.functional.normalize(router, dim=-1)
    packed["embed"] = (W["embed"] + lean).to(torch.bfloat16)
    W["embed"] = packed["embed"].to(torch.float64)
    model = importlib.import_module("llm-inference-engine_b200.models.vasolix").VasolixModel(config, packed, dtype=dtype, device="cuda:0", max_tokens=128, max_seqs=20,
                                                                                              max_pages_per_seq=2)
    serving = importlib.import_module("llm-inference-engine_b200.serving")
    for n in (9, 12, 13, 16, 17, 24, 25, 32, 33, 63, 64, 65):
        toks = np.random.default_rng(n).integers(0, 80, n).tolist()
        sess = serving.Session(model, 2560, max_seqs=20, max_batch_tokens=128, poison=True)
        got = sess.feed([(sess.open(), toks, range(n))]).cpu().numpy()
        want, open_rows = ambiguous_rows(monkeypatch, config, W, toks, u)
        err = np.linalg.norm(got - want, axis=-1) / np.linalg.norm(want, axis=-1)
        assert (err[~open_rows] < tol).all(), (n, err, open_rows)
        assert open_rows.mean() <= 0.3, (n, open_rows)


@pytest.mark.parametrize("dtype,tol", [("bfloat16", 4e-2), ("float16", 6e-3)])
@pytest.mark.parametrize("n", [511, 512, 1000, 1023])
def test_prompts_of_one_expert_each(monkeypatch, dtype, tol, n):
    """16-bit prompts of one expert each: from 512 tokens on their choice and their plan run in many CTAs (expert tiles of 128 rows)."""
    layer = ref.attention_layer(heads=2, kv_heads=1, dim=16, size=50, mlp=ref.moe(experts=5, top=1, ff=64, shared_ff=64))
    config = ref.make_config([layer], width=64, vocab=80)
    W, packed = ref.make_weights(config, seed=2)
    model = importlib.import_module("llm-inference-engine_b200.models.vasolix").VasolixModel(config, packed, dtype=dtype, device="cuda:0", max_tokens=1024, max_seqs=1,
                                                                                              max_pages_per_seq=16)
    toks = np.random.default_rng(n).integers(0, 80, n).tolist()
    sess = importlib.import_module("llm-inference-engine_b200.serving").Session(model, 1024, max_seqs=1, max_batch_tokens=1024, poison=True)
    rid = sess.open()
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as prof:
        got = sess.feed([(rid, toks, range(n))]).cpu().numpy()
    want, open_rows = ambiguous_rows(monkeypatch, config, W, toks, 2.0 ** -8 if dtype == "bfloat16" else 2.0 ** -11)
    err = np.linalg.norm(got - want, axis=-1) / np.linalg.norm(want, axis=-1)
    assert (err[~open_rows] < tol).all() and open_rows.mean() <= 0.6
    kernels = " ".join(e.key for e in prof.key_averages())
    if "kernel" not in kernels:
        pytest.skip("no launch was recorded: the route is not seen")
    assert ("moe_route_count_kernel" in kernels) == (n >= 512) and ("moe_plan_kernel" in kernels) == (n < 512), kernels


@pytest.mark.parametrize("dtype,tol", [("bfloat16", 4e-2), ("float16", 6e-3)])
@pytest.mark.parametrize("n", [8, 9, 16])
def test_same_experts_for_every_token_of_a_decode_batch(dtype, tol, n):
    """n sequences of one and the same token: every row of the two experts' tiles is live, the last one too."""
    layer = ref.attention_layer(heads=2, kv_heads=1, dim=16, size=50, mlp=ref.moe(experts=5, top=2, ff=64, shared_ff=64))
    config = ref.make_config([layer], width=64, vocab=80)
    W, packed = ref.make_weights(config, seed=2)
    model = importlib.import_module("llm-inference-engine_b200.models.vasolix").VasolixModel(config, packed, dtype=dtype, device="cuda:0", max_tokens=32, max_seqs=16,
                                                                                              max_pages_per_seq=1)
    sess = importlib.import_module("llm-inference-engine_b200.serving").Session(model, 64 * 16, max_seqs=16, max_batch_tokens=32, poison=True)
    got = sess.feed([(sess.open(), [7], [0]) for _ in range(n)]).cpu().numpy()
    want = ref.forward(config, W, [7]).numpy()
    assert (np.linalg.norm(got - want, axis=-1) / np.linalg.norm(want) < tol).all()


def test_same_experts_for_every_token():
    """33 sequences of the same three tokens in fp32: 99 tokens whose choices fall on a few of five experts, several tiles for each."""
    layer = ref.attention_layer(heads=2, kv_heads=1, dim=16, size=50, mlp=ref.moe(experts=5, top=2, ff=64, shared_ff=64))
    config = ref.make_config([layer], width=64, vocab=80)
    W, packed = ref.make_weights(config, seed=2)
    toks = [7] * 3
    model = importlib.import_module("llm-inference-engine_b200.models.vasolix").VasolixModel(config, packed, dtype="float32", device="cuda:0", max_tokens=128, max_seqs=40,
                                                                                              max_pages_per_seq=1)
    sess = importlib.import_module("llm-inference-engine_b200.serving").Session(model, 64 * 40, max_seqs=40, max_batch_tokens=128, poison=True)
    got = sess.feed([(sess.open(), toks, range(3)) for _ in range(33)]).cpu().numpy().reshape(33, 3, -1)
    want = ref.forward(config, W, toks).numpy()
    assert np.abs(got - want[None]).max() / np.abs(want).max() < 2e-5
