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
