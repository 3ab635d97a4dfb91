"""Decode steps of gated linear attention in one launch (csrc/gla.cu gla_decode_kernel): head sizes and ranks at the edges of what it takes (values of 32 to 256, keys
fewer and more than a pass of its lanes, ranks of 8 to 128), sequences of different ages in a batch and a state that is carried; against the float64 restatement.
Sizes beside them (values of 24 or 288, ranks of 6) keep the three launches."""
import importlib

import numpy as np
import pytest
import torch

import vasolix_oracle as ref

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,tol", [("bfloat16", 4e-2), ("float16", 6e-3)])
@pytest.mark.parametrize("heads,dim,vdim,rank", [(1, 8, 32, 8), (2, 64, 64, 16), (3, 132, 32, 24), (2, 128, 256, 64), (1, 300, 128, 128), (2, 16, 24, 8), (1, 16, 288, 32), (2, 32, 64, 6)])
def test_steps(dtype, tol, heads, dim, vdim, rank):
    config = ref.make_config([ref.gla_layer(heads=heads, dim=dim, vdim=vdim, tau=4.0)], width=64)
    W, packed = ref.make_weights(config, seed=heads + dim, decay_rank=rank)
    model = importlib.import_module("llm-inference-engine_b200.models.vasolix").VasolixModel(config, packed, dtype=dtype, device="cuda:0", max_tokens=128, max_seqs=4,
                                                                                              max_pages_per_seq=2)
    serving = importlib.import_module("llm-inference-engine_b200.serving")
    sess = serving.Session(model, 512, max_seqs=4, max_batch_tokens=128, poison=True)
    before, steps = [0, 1, 5, 40], 12
    toks = [np.random.default_rng(i).integers(0, config["vocab"], n + steps).tolist() for i, n in enumerate(before)]
    ids = [sess.open() for _ in before]
    for i, n in enumerate(before):
        if n:
            sess.feed([(ids[i], toks[i][:n], [])])
    got = [[] for _ in before]
    for k in range(steps):
        out = sess.feed([(ids[i], toks[i][n + k:n + k + 1], [0]) for i, n in enumerate(before)]).cpu().numpy()
        for i in range(len(before)):
            got[i].append(out[i])
    for i, n in enumerate(before):
        want = ref.forward(config, W, toks[i]).numpy()[n:]
        lg = np.stack(got[i])
        assert not np.isnan(lg).any()
        err = np.linalg.norm(lg - want, axis=-1) / np.linalg.norm(want, axis=-1)
        assert err.max() < tol, (n, float(err.max()))


@pytest.mark.parametrize("heads,dim,vdim,rank", [(8, 64, 128, 16), (8, 128, 256, 64)])
def test_a_token_by_itself(heads, dim, vdim, rank):
    """A decoded token's row has the same bits by itself, among others, and beside portions of several tokens (sixteen rows in all: the range in which the linears around
    it have), step after step over the state that it leaves; and the portions beside it are what they are without it."""
    config = ref.make_config([ref.gla_layer(heads=heads, dim=dim, vdim=vdim, tau=4.0) for _ in range(2)], width=128)
    _, packed = ref.make_weights(config, seed=heads + dim, decay_rank=rank)
    model = importlib.import_module("llm-inference-engine_b200.models.vasolix").VasolixModel(config, packed, dtype="float16", device="cuda:0", max_tokens=128, max_seqs=4,
                                                                                              max_pages_per_seq=2)
    serving = importlib.import_module("llm-inference-engine_b200.serving")
    before, steps, beside = [0, 1, 5, 40], 4, [1, 5, 1, 7]  # tokens that each sequence brings to a step
    toks = [np.random.default_rng(i).integers(0, config["vocab"], n + steps * k).tolist() for i, (n, k) in enumerate(zip(before, beside))]
    rows = {}
    for how in ("alone", "together"):
        sess = serving.Session(model, 512, max_seqs=4, max_batch_tokens=128, poison=True)
        ids = [sess.open() for _ in before]
        for i, n in enumerate(before):
            if n:
                sess.feed([(ids[i], toks[i][:n], [])])
        for s in range(steps):
            entries = [(ids[i], toks[i][n + s * k:n + (s + 1) * k], list(range(k))) for i, (n, k) in enumerate(zip(before, beside))]
            rows[how, s] = torch.cat([sess.feed([e]) for e in entries]) if how == "alone" else sess.feed(entries)
    for s in range(steps):
        assert not torch.isnan(rows["together", s]).any()
        assert torch.equal(rows["alone", s], rows["together", s]), s
