"""Experts of a few tokens, the router's product and the grouping of pairs (csrc/moe.cu) at the edges of their ranges: 1, 8, 9, 16 and 17 tokens, inner
sizes that do not share out evenly over the warps, more experts than lanes, every token choosing the same experts; against the float64 restatement."""
import importlib

import numpy as np
import pytest

import vasolix_oracle as ref

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,tol", [("bfloat16", 4e-2), ("float16", 6e-3)])
@pytest.mark.parametrize("width,ff,experts,top", [(64, 64, 5, 2), (512, 96, 40, 3), (544, 224, 7, 7), (1024, 512, 70, 4), (2080, 64, 3, 1)])
def test_experts_of_few_tokens(dtype, tol, width, ff, experts, top):
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
        want = ref.forward(config, W, toks).numpy()
        assert not np.isnan(got).any()
        # a 16-bit router may choose another expert where two scores are closer than its rounding: such a token is judged by its neighbours
        err = np.linalg.norm(got - want, axis=-1) / np.linalg.norm(want, axis=-1)
        assert np.sort(err)[: max(1, int(0.8 * n))].max() < tol, (n, err)


def test_same_experts_for_every_token():
    """One row per pair of an expert, 100 tokens on the same two of five: counts that no two experts share."""
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
