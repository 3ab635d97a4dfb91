"""The tcgen05 attention of prompt portions (csrc/prompt_attn_tc.cu) at the edges of its tiles: portions on both sides of 64 tokens, that continue inside
a page, blocks and windows shorter than a page and longer than the prompt, two heads per CTA of one and of several kv heads, a sink that outweighs
the keys, logits with a distance penalty, a slope, blocks and a sink; against the float64 restatements of the designs, pools poisoned with NaN."""
import importlib

import numpy as np
import pytest

import fedovik_oracle
import pamulix_oracle
import vasolix_oracle
import zefenex_oracle

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def session(name, config, packed, dtype):
    cls = getattr(importlib.import_module("llm-inference-engine_b200.models." + name), name.capitalize() + "Model")
    model = cls(config, packed, dtype=dtype, device=DEV, max_tokens=1024, max_seqs=3, max_pages_per_seq=8)
    return importlib.import_module("llm-inference-engine_b200.serving").Session(model, 1536, max_seqs=3, max_batch_tokens=1024, poison=True)


def check(name, oracle, layer, dtype, tol, sink=None):
    config = oracle.make_config([layer])
    W, packed = oracle.make_weights(config, seed=11)
    if sink is not None:
        W["l0.mix.sink"][:] = sink
        packed["l0.mix.sink"][:] = sink
    rng = np.random.default_rng(3)
    requests = {k: rng.integers(0, config["vocab"], n).tolist() for k, n in {"a": 64 + 63 + 1, "b": 9 + 65 + 130, "c": 333}.items()}
    sess = session(name, config, packed, dtype)
    rid, fed, got = {k: sess.open() for k in requests}, {k: 0 for k in requests}, {k: [] for k in requests}
    for step in ([("a", 64), ("b", 9)], [("b", 65), ("c", 333), ("a", 63)], [("a", 1), ("b", 130)]):
        out, at = sess.feed([(rid[k], requests[k][fed[k]:fed[k] + n], range(n)) for k, n in step]).cpu().numpy(), 0
        for k, n in step:
            got[k].append(out[at:at + n])
            fed[k], at = fed[k] + n, at + n
    for k, toks in requests.items():
        want, g = oracle.forward(config, W, toks).numpy(), np.concatenate(got[k])
        assert not np.isnan(g).any(), k
        assert np.linalg.norm(g - want) / np.linalg.norm(want) < tol, (k, np.linalg.norm(g - want) / np.linalg.norm(want))


# stored rows rounded to the engine's type at every step of the layer and of the head: a few roundings of 2^-8 (bf16) and 2^-11 (fp16)
TYPES = [("bfloat16", 2.5e-2), ("float16", 4e-3)]


@pytest.mark.parametrize("dtype,tol", TYPES)
@pytest.mark.parametrize("heads,kv_heads,size", [(2, 1, 24), (4, 2, 64), (8, 2, 100), (4, 1, 1000), (6, 3, 127)])
def test_chunked(dtype, tol, heads, kv_heads, size):
    check("vasolix", vasolix_oracle, vasolix_oracle.attention_layer(heads=heads, kv_heads=kv_heads, dim=128, size=size, scale=0.1), dtype, tol)


@pytest.mark.parametrize("dtype,tol", TYPES)
@pytest.mark.parametrize("heads,rank,window", [(2, 128, 24), (4, 192, 64), (2, 192, 65), (6, 256, 200), (2, 192, 0), (4, 128, 1)])
def test_latent(dtype, tol, heads, rank, window):
    layer = zefenex_oracle.latent_layer(heads=heads, dim=32, rot_dim=64, vdim=32, kv_rank=rank, window=window or None, scale=0.1)
    if not window:
        layer["mixer"].pop("mask")
    check("zefenex", zefenex_oracle, layer, dtype, tol)


@pytest.mark.parametrize("dtype,tol", TYPES)
@pytest.mark.parametrize("heads,kv_heads,window", [(2, 1, 24), (4, 2, 64), (8, 2, 65), (4, 1, 1000), (6, 3, 1)])
def test_scored_with_a_distance_penalty(dtype, tol, heads, kv_heads, window):
    check("fedovik", fedovik_oracle, fedovik_oracle.pair_layer(heads=heads, kv_heads=kv_heads, dim=128, vdim=128, window=window), dtype, tol)


@pytest.mark.parametrize("dtype,tol", TYPES)
@pytest.mark.parametrize("heads,kv_heads,chunk", [(2, 1, 24), (4, 2, 64), (8, 2, 100), (4, 1, 1000)])
def test_scored_with_a_slope_and_blocks(dtype, tol, heads, kv_heads, chunk):
    check("pamulix", pamulix_oracle, pamulix_oracle.attention(heads=heads, kv_heads=kv_heads, dim=128, vdim=128, chunk=chunk, v_mix=False), dtype, tol)


@pytest.mark.parametrize("sink", [-30.0, 12.0])
def test_sink_far_from_the_scores(sink):
    """A sink far below the scores vanishes; one far above them takes nearly all the weight and sets the running maximum from the start."""
    check("vasolix", vasolix_oracle, vasolix_oracle.attention_layer(heads=2, kv_heads=1, dim=128, size=90, scale=0.1), "float16", 4e-3, sink)
    check("zefenex", zefenex_oracle, zefenex_oracle.latent_layer(heads=2, dim=32, rot_dim=64, vdim=32, kv_rank=192, window=70, scale=0.1), "float16", 4e-3, sink)
