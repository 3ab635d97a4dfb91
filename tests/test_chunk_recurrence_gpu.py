"""The token-parallel recurrences (csrc/chunk_recurrence.cu) at the sizes where they can go wrong: portions on both sides of the shortest one
they take and of a chunk's edge, portions that continue from a state, beside shorter ones in the same batch; keys shared by heads; decays that
underflow; more chunks than the scratch holds at once.  Against the float64 restatements of the designs, in fp32 (every position) and bf16."""
import importlib

import numpy as np
import pytest
import torch

import fedovik_oracle
import silonex_oracle
import vasolix_oracle

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def session(name, config, packed, dtype, most):
    cls = getattr(importlib.import_module("llm-inference-engine_b200.models." + name), name.capitalize() + "Model")
    model = cls(config, packed, dtype=dtype, device=DEV, max_tokens=most, max_seqs=4, max_pages_per_seq=most // 64 + 1)
    return importlib.import_module("llm-inference-engine_b200.serving").Session(model, 4 * most, max_seqs=4, max_batch_tokens=most, poison=True)


def replay(sess, requests, steps):
    rid = {k: sess.open() for k in requests}
    fed, got = {k: 0 for k in requests}, {k: [] for k in requests}
    for step in steps:
        entries = [(rid[k], requests[k][fed[k]:fed[k] + n], range(n)) for k, n in step]
        out, at = sess.feed(entries).cpu().numpy(), 0
        for k, n in step:
            got[k].append(out[at:at + n])
            fed[k], at = fed[k] + n, at + n
    return {k: np.concatenate(v) for k, v in got.items()}


def worst(got, want):
    assert not np.isnan(got).any()
    return float((np.linalg.norm(got - want, axis=-1) / np.linalg.norm(want, axis=-1)).max())


LAYERS = {
    "gla_64": ("vasolix", vasolix_oracle, [vasolix_oracle.gla_layer(heads=3, dim=64, vdim=48)]),
    "gla_128": ("vasolix", vasolix_oracle, [vasolix_oracle.gla_layer(heads=2, dim=128, vdim=16)]),
    "gla_strong_decay": ("vasolix", vasolix_oracle, [vasolix_oracle.gla_layer(heads=2, dim=64, vdim=16, tau=0.02)]),
    "delta_64": ("fedovik", fedovik_oracle, [fedovik_oracle.pair_layer(r_heads=4, r_kv_heads=2, r_dim=64, r_vdim=16)]),
    "delta_128": ("fedovik", fedovik_oracle, [fedovik_oracle.pair_layer(r_heads=2, r_kv_heads=2, r_dim=128, r_vdim=32)]),
    "delta_one_decay": ("silonex", silonex_oracle, [silonex_oracle.pair_layer(r_heads=2, r_dim=64, r_vdim=16)]),
    "state_space": ("silonex", silonex_oracle, [silonex_oracle.mamba_layer(heads=4, vdim=16, state=64, groups=2, norm_groups=2)]),
    "constant_decay": ("silonex", silonex_oracle, [silonex_oracle.lightning_layer(heads=2, dim=128, vdim=16)]),
}


def model(name, oracle, layers, **kw):
    config = oracle.make_config(layers, **kw)
    W, packed = (oracle.random_model if hasattr(oracle, "random_model") else oracle.make_weights)(config, seed=5)
    return config, W, packed


@pytest.mark.parametrize("which", LAYERS)
@pytest.mark.parametrize("dtype,tol", [("float32", 2e-5), ("bfloat16", 4e-2)])
def test_portions_match_the_oracle(which, dtype, tol):
    """fp32: the tolerance the serial kernels are held to (sums of a few hundred terms in fp32, through a norm that divides by the read-out's
    size); bf16: 2^-9 per stored row through the layer and the head, at the worst of several hundred positions."""
    name, oracle, layers = LAYERS[which]
    config, W, packed = model(name, oracle, layers)
    rng = np.random.default_rng(7)
    lens = {"a": 64 + 33 + 1, "b": 63 + 65 + 7, "c": 129 + 96, "d": 160}
    requests = {k: rng.integers(0, config["vocab"], n).tolist() for k, n in lens.items()}
    steps = [[("a", 64), ("b", 63), ("c", 129)], [("b", 65), ("a", 33), ("d", 160)], [("c", 96), ("a", 1), ("b", 7)]]
    got = replay(session(name, config, packed, dtype, 512), requests, steps)
    for k, toks in requests.items():
        want = np.asarray(oracle.forward(config, W, toks))
        if dtype == "float32":
            assert worst(got[k], want) < tol, k
        else:
            assert np.linalg.norm(got[k] - want) / np.linalg.norm(want) < tol, k


def test_more_chunks_than_the_scratch_holds():
    """32 heads of 128 channels: 64 MB hold 36 chunks, so two prompts of 700 and 500 tokens run in several rounds, the state carried between them."""
    config, W, packed = model("vasolix", vasolix_oracle, [vasolix_oracle.gla_layer(heads=32, dim=128, vdim=16)])
    rng = np.random.default_rng(8)
    requests = {k: rng.integers(0, config["vocab"], n).tolist() for k, n in {"a": 700, "b": 500, "c": 100}.items()}
    got = replay(session("vasolix", config, packed, "float32", 1408), requests, [[("a", 700), ("b", 500), ("c", 100)]])
    for k, toks in requests.items():
        assert worst(got[k], vasolix_oracle.forward(config, W, toks).numpy()) < 2e-5, k


def test_scratch_size_follows_the_limits():
    """Sizes the kernels do not take ask for no scratch; the others grow with the token limit up to 64 MB."""
    sizes = []
    for dim, most in ((48, 4096), (64, 1024), (64, 4096)):
        config, _, packed = model("vasolix", vasolix_oracle, [vasolix_oracle.gla_layer(heads=2, dim=dim, vdim=16)])
        sess = session("vasolix", config, packed, "float32", most)
        sizes.append(sess.engine._scratch.numel() / most)
    assert sizes[1] > sizes[0]
    assert abs(sizes[2] / sizes[1] - 1) < 0.2
