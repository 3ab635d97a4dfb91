"""The tiled preparation of the delta rule's prompts (csrc/recurrent.cu) at the edges of its tiles: channel counts that end inside a warp and inside a
block, portions that continue another's convolution, last tiles of one to eight rows; against the float64 restatement of the design."""
import importlib

import numpy as np
import pytest

import fedovik_oracle as ref

pytestmark = pytest.mark.gpu


# 16-bit rows rounded at every step of the layer and of the head: a few roundings of 2^-8 (bf16) and 2^-11 (fp16)
@pytest.mark.parametrize("dtype,tol", [("bfloat16", 2.5e-2), ("float16", 4e-3)])
@pytest.mark.parametrize("heads,kv_heads,dim,vdim", [(1, 1, 128, 24), (2, 1, 128, 16), (4, 4, 32, 40), (2, 2, 64, 256), (3, 1, 128, 72)])
def test_channels_that_end_anywhere(dtype, tol, heads, kv_heads, dim, vdim):
    layer = ref.pair_layer(heads=2, kv_heads=1, dim=16, vdim=8, window=24, r_heads=heads, r_kv_heads=kv_heads, r_dim=dim, r_vdim=vdim, conv=4)
    config = ref.make_config([layer])
    W, packed = ref.make_weights(config, seed=7)
    model = importlib.import_module("llm-inference-engine_b200.models.fedovik").FedovikModel(config, packed, dtype=dtype, device="cuda:0", max_tokens=512, max_seqs=2,
                                                                                             max_pages_per_seq=8)
    sess = importlib.import_module("llm-inference-engine_b200.serving").Session(model, 1024, max_seqs=2, max_batch_tokens=512, poison=True)
    rng = np.random.default_rng(2)
    tokens = {k: rng.integers(0, config["vocab"], n).tolist() for k, n in {"a": 150, "b": 99}.items()}
    rid, fed, got = {k: sess.open() for k in tokens}, {k: 0 for k in tokens}, {k: [] for k in tokens}
    for step in ([("a", 65), ("b", 2)], [("b", 97), ("a", 85)]):
        out, at = sess.feed([(rid[k], tokens[k][fed[k]:fed[k] + n], range(n)) for k, n in step]).cpu().numpy(), 0
        for k, n in step:
            got[k].append(out[at:at + n])
            fed[k], at = fed[k] + n, at + n
    for k, toks in tokens.items():
        want, g = ref.forward(config, W, toks).numpy(), np.concatenate(got[k])
        assert not np.isnan(g).any()
        assert np.linalg.norm(g - want) / np.linalg.norm(want) < tol, (k, np.linalg.norm(g - want) / np.linalg.norm(want))
