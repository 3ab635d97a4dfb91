"""Decoded tokens of the per-token attention kernels (csrc/attention_chunked.cu, csrc/attention_scored.cu): contexts of a few keys and of several
rounds of the block, blocks and windows that end inside a page; against the float64 restatements of the designs, pools poisoned with NaN."""
import importlib

import numpy as np
import pytest

import fedovik_oracle
import pamulix_oracle
import vasolix_oracle

pytestmark = pytest.mark.gpu
LENGTHS = {"a": 3, "b": 5, "c": 11, "d": 132, "e": 703}
LAYERS = [
    ("vasolix", vasolix_oracle, vasolix_oracle.attention_layer(heads=2, kv_heads=1, dim=16, size=1000, scale=0.3)),
    ("vasolix", vasolix_oracle, vasolix_oracle.attention_layer(heads=4, kv_heads=2, dim=12, size=130, scale=0.3)),
    ("vasolix", vasolix_oracle, vasolix_oracle.attention_layer(heads=2, kv_heads=2, dim=128, size=701, scale=0.1)),
    ("fedovik", fedovik_oracle, fedovik_oracle.pair_layer(heads=2, kv_heads=1, window=600)),
    ("fedovik", fedovik_oracle, fedovik_oracle.attention_layer(heads=2, kv_heads=1)),
    ("pamulix", pamulix_oracle, pamulix_oracle.attention(heads=2, kv_heads=1, chunk=640, v_mix=False)),
]


# fp32: sums of a few hundred terms in another order; 16 bits: the roundings of the stored rows
@pytest.mark.parametrize("dtype,tol", [("float32", 2e-5), ("bfloat16", 2.5e-2)])
@pytest.mark.parametrize("name,oracle,layer", LAYERS, ids=["block", "odd-dim", "tile-dim", "window", "sigmoid", "slope"])
def test_decoded_tokens(name, oracle, layer, dtype, tol):
    config = oracle.make_config([layer])
    W, packed = oracle.make_weights(config, seed=5)
    cls = getattr(importlib.import_module("llm-inference-engine_b200.models." + name), name.capitalize() + "Model")
    model = cls(config, packed, dtype=dtype, device="cuda:0", max_tokens=1024, max_seqs=5, max_pages_per_seq=16)
    sess = importlib.import_module("llm-inference-engine_b200.serving").Session(model, 2048, max_seqs=5, max_batch_tokens=1024, poison=True)
    rng = np.random.default_rng(9)
    tokens = {k: rng.integers(0, config["vocab"], n).tolist() for k, n in LENGTHS.items()}
    rid = {k: sess.open() for k in tokens}
    sess.feed([(rid[k], t[:-2], []) for k, t in tokens.items()])
    for at in (-2, -1):
        got = sess.feed([(rid[k], t[at:len(t) + at + 1], [0]) for k, t in tokens.items()]).cpu().numpy()
        for row, t in zip(got, tokens.values()):
            want = oracle.forward(config, W, t).numpy()[at]
            assert np.linalg.norm(row - want) / np.linalg.norm(want) < tol, (len(t), at, np.linalg.norm(row - want) / np.linalg.norm(want))
