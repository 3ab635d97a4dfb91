"""What a call of the layer-list decoder copies to the device: the description of its batch (csrc/hybrid.cu, b200_hybrid_forward), in proportion to what is in it.  The
list of decoded tokens (16 bytes each) and the counters of their runs of keys (one per token and query head) cost a prompt nothing."""
import importlib
import json

import numpy as np
import pytest
import torch

import vasolix_oracle as ref

pytestmark = pytest.mark.gpu


def uploaded(calls, path):
    """Bytes that one of some equal calls copies to the device (the largest found: a profiler may miss a copy)."""
    torch.cuda.synchronize()
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as p:
        for call in calls:
            call()
        torch.cuda.synchronize()
    p.export_chrome_trace(str(path))
    return max(e["args"]["bytes"] for e in json.load(open(path))["traceEvents"] if e.get("cat") == "gpu_memcpy" and "HtoD" in e["name"])


def test_a_prompt_uploads_no_list_of_decoded_tokens(tmp_path):
    heads, tokens, pages, layers = 4, 2048, 40, 1
    config = ref.make_config([ref.attention_layer(heads=heads, kv_heads=2, dim=64, size=4096, scale=0.125) for _ in range(layers)], width=64)
    _, packed = ref.make_weights(config, seed=2)
    model = importlib.import_module("llm-inference-engine_b200.models.vasolix").VasolixModel(config, packed, dtype="bfloat16", device="cuda:0", max_tokens=tokens, max_seqs=4,
                                                                                              max_pages_per_seq=pages)
    sess = importlib.import_module("llm-inference-engine_b200.serving").Session(model, 4 * (2048 + 64), max_seqs=4, max_batch_tokens=tokens)
    toks = np.random.default_rng(0).integers(0, config["vocab"], tokens + 1).tolist()
    ids = [sess.open() for _ in range(4)]
    prompt = uploaded([lambda i=i: sess.feed([(i, toks[:tokens], [])]) for i in ids], tmp_path / "p.json")
    decode = uploaded([lambda i=i: sess.feed([(i, toks[tokens:], [0])]) for i in ids], tmp_path / "d.json")
    # ids, sequence, position, wanted rows and short rows of every token; tiles of 64 tokens; start, first position, slot; pages; two counts per layer
    ints = lambda n, listed: 5 * n + 4 * (n // 64 + 2) + 4 + pages + 2 * layers + listed * (4 + heads)  # noqa: E731
    assert prompt == 4 * ints(tokens, 0), (prompt, ints(tokens, 0) * 4)
    assert decode == 4 * ints(1, 1), (decode, ints(1, 1) * 4)


@pytest.mark.parametrize("starts", [[0, 9, 4], [0, 400, 4], [0, 2, 9, 4], [0, 3, 2, 4]])
def test_portions_outside_the_batch_are_refused(starts):
    """Starts that pass the number of tokens and come back, or that fall: refused before anything is written for them."""
    config = ref.make_config([ref.attention_layer(heads=2, kv_heads=1, dim=64, size=100, scale=0.125)], width=64)
    _, packed = ref.make_weights(config, seed=2)
    model = importlib.import_module("llm-inference-engine_b200.models.vasolix").VasolixModel(config, packed, dtype="bfloat16", device="cuda:0", max_tokens=16, max_seqs=4,
                                                                                              max_pages_per_seq=8)
    engine, seqs = model.engine, len(starts) - 1
    engine.set_pools(8 * seqs, seqs)
    call = lambda st: engine.forward([1, 2, 3, 4], st, [0] * seqs, range(seqs), np.arange(8 * seqs), [3])  # noqa: E731
    with pytest.raises(importlib.import_module("llm-inference-engine_b200").B200Error, match="bad portion"):
        call(starts)
    assert torch.isfinite(call([0] * seqs + [4])).all()
