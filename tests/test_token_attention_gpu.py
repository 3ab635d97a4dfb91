"""Attention of decoded tokens by key head (csrc/attention_token.cu) against the float64 restatements: query heads per key head on both sides of every block of
heads (1, 2, 3, 4, 5, 8, 9), head sizes of 64 and 128 (256 keeps the per-token kernel), contexts of one key, of a page's edge (63, 64, 65), and of more blocks of keys
than one; batches whose tokens share out their keys beside batches that do not; portions of several decoded tokens; windows, blocks, a sink, distance penalties and
un-normalised weights."""
import importlib

import numpy as np
import pytest
import torch

import fedovik_oracle
import vasolix_oracle

pytestmark = pytest.mark.gpu
TOL = {"bfloat16": 4e-2, "float16": 6e-3}  # as the other tests of 16-bit engines: rounding of a layer's rows, eight or eleven bits


def run(name, ref, config, dtype, contexts, steps, seqs):
    W, packed = ref.make_weights(config, seed=5)
    cls = {"vasolix": "VasolixModel", "fedovik": "FedovikModel"}[name]
    longest = max(contexts) + steps
    model = getattr(importlib.import_module("llm-inference-engine_b200.models." + name), cls)(config, packed, dtype=dtype, device="cuda:0", max_tokens=2048, max_seqs=seqs,
                                                                                              max_pages_per_seq=(longest + 63) // 64)
    serving = importlib.import_module("llm-inference-engine_b200.serving")
    sess = serving.Session(model, (longest + 64) * seqs, max_seqs=seqs, max_batch_tokens=2048, poison=True)
    toks = [np.random.default_rng(i).integers(0, config["vocab"], n + steps).tolist() for i, n in enumerate(contexts)]
    ids = [sess.open() for _ in contexts]
    for i, n in enumerate(contexts):
        if n:
            sess.feed([(ids[i], toks[i][:n], [])])
    got = [[] for _ in contexts]
    at = list(contexts)
    while any(a < len(t) for a, t in zip(at, toks)):
        some = [i for i in range(len(toks)) if at[i] < len(toks[i])]
        take = {i: min(1 + (i + at[i]) % 3, len(toks[i]) - at[i]) for i in some}  # portions of one to three tokens
        out = sess.feed([(ids[i], toks[i][at[i]:at[i] + take[i]], list(range(take[i]))) for i in some]).cpu().numpy()
        o = 0
        for i in some:
            got[i].append(out[o:o + take[i]])
            o += take[i]
            at[i] += take[i]
    for i, n in enumerate(contexts):
        want = ref.forward(config, W, toks[i])
        want = (want[0] if isinstance(want, tuple) else want).numpy()[n:]
        lg = np.concatenate(got[i])
        assert not np.isnan(lg).any()
        err = np.linalg.norm(lg - want, axis=-1) / np.linalg.norm(want, axis=-1)
        assert err.max() < TOL[dtype], (n, int(err.argmax()), float(err.max()))


EDGES = [0, 1, 30, 31, 32, 62, 63, 64, 95, 290]


@pytest.mark.parametrize("dtype", ["bfloat16", "float16"])
@pytest.mark.parametrize("heads,kv,dim,chunk", [(1, 1, 64, 40), (2, 1, 128, 64), (6, 2, 64, 100), (4, 1, 128, 1000), (5, 1, 64, 200), (8, 1, 64, 33), (9, 1, 64, 128), (2, 2, 256, 96)])
def test_blocks_of_positions_with_a_sink(dtype, heads, kv, dim, chunk):
    config = vasolix_oracle.make_config([vasolix_oracle.attention_layer(heads=heads, kv_heads=kv, dim=dim, size=chunk, scale=dim ** -0.5)], width=64)
    run("vasolix", vasolix_oracle, config, dtype, EDGES, 5, 10)
    run("vasolix", vasolix_oracle, config, dtype, [700], 4, 1)


@pytest.mark.parametrize("dtype", ["bfloat16", "float16"])
@pytest.mark.parametrize("heads,kv,dim,vdim,window", [(2, 1, 32, 64, 33), (4, 2, 64, 128, 64), (3, 1, 96, 64, 200), (8, 2, 128, 128, 500), (8, 1, 64, 256, 70)])
def test_windows_with_a_distance_penalty(dtype, heads, kv, dim, vdim, window):
    layer = fedovik_oracle.pair_layer(heads=heads, kv_heads=kv, dim=dim, vdim=vdim, window=window, mlp=fedovik_oracle.dense())
    config = fedovik_oracle.make_config([layer], width=64)
    run("fedovik", fedovik_oracle, config, dtype, EDGES, 5, 10)
    run("fedovik", fedovik_oracle, config, dtype, [600], 4, 1)


@pytest.mark.parametrize("dtype", ["bfloat16", "float16"])
@pytest.mark.parametrize("heads,kv,dim,vdim", [(4, 2, 64, 64), (3, 1, 32, 128)])
def test_unnormalised_weights(dtype, heads, kv, dim, vdim):
    config = fedovik_oracle.make_config([fedovik_oracle.attention_layer(heads=heads, kv_heads=kv, dim=dim, vdim=vdim)], width=64)
    run("fedovik", fedovik_oracle, config, dtype, EDGES, 5, 10)
    run("fedovik", fedovik_oracle, config, dtype, [400], 4, 1)


@pytest.mark.parametrize("design,heads,kv,dim,size,contexts", [
    ("vasolix", 16, 4, 128, 8192, [1, 100, 126, 127, 128, 254, 255, 256, 300, 511, 700, 1000, 1500, 2500, 4094, 4200]),  # one block of keys to 32, and longer ones
    ("vasolix", 16, 2, 128, 1000, [40, 990, 1010, 2400]),  # blocks of positions
    ("fedovik", 16, 4, 128, 0, [5, 300, 599, 601, 1200, 3000]),  # un-normalised weights
    ("vasolix", 32, 16, 64, 4096, [2300 + 7 * i for i in range(16)])])  # more blocks than a launch's scratch holds
def test_a_token_by_itself(design, heads, kv, dim, size, contexts):
    """The keys of a decoded token are cut by its own context: its row has the same bits by itself, where its blocks of keys are shared out over the device, and in a
    batch of up to sixteen, the range in which the linears around it have."""
    if design == "vasolix":
        ref, config = vasolix_oracle, vasolix_oracle.make_config([vasolix_oracle.attention_layer(heads=heads, kv_heads=kv, dim=dim, size=size, scale=dim ** -0.5)], width=128)
    else:
        ref, config = fedovik_oracle, fedovik_oracle.make_config([fedovik_oracle.attention_layer(heads=heads, kv_heads=kv, dim=dim, vdim=dim)], width=128)
    _, packed = ref.make_weights(config, seed=9)
    model = getattr(importlib.import_module("llm-inference-engine_b200.models." + design), design.capitalize() + "Model")(
        config, packed, dtype="float16", device="cuda:0", max_tokens=2048, max_seqs=len(contexts), max_pages_per_seq=80)
    serving = importlib.import_module("llm-inference-engine_b200.serving")
    toks = [np.random.default_rng(i).integers(0, config["vocab"], n + 3).tolist() for i, n in enumerate(contexts)]
    rows = {}
    for how in ("alone", "together"):
        sess = serving.Session(model, sum(n + 67 for n in contexts), max_seqs=len(contexts), max_batch_tokens=2048, poison=True)
        ids = [sess.open() for _ in contexts]
        for i, n in enumerate(contexts):
            for a in range(0, n, 2000):
                sess.feed([(ids[i], toks[i][a:min(a + 2000, n)], [])])
        for k in range(3):
            entries = [(ids[i], toks[i][n + k:n + k + 1], [0]) for i, n in enumerate(contexts)]
            rows[how, k] = torch.cat([sess.feed([e]) for e in entries]) if how == "alone" else sess.feed(entries)
    for k in range(3):
        same = (rows["alone", k] == rows["together", k]).all(dim=-1)
        assert same.all(), [contexts[i] for i in range(len(contexts)) if not same[i]]


@pytest.mark.parametrize("heads,kv", [(1, 1), (8, 1)])
def test_long_contexts(heads, kv):
    """Contexts beyond the sizes at which blocks of keys change their number and their length (4096, 32768 and 131072 keys): the last tokens of a prompt decoded one by
    one against the same tokens as a portion of eight, which the prompt kernel takes.  Both round their rows to 16 bits."""
    config = vasolix_oracle.make_config([vasolix_oracle.attention_layer(heads=heads, kv_heads=kv, dim=64, size=1 << 20, scale=0.125)], width=64)
    _, packed = vasolix_oracle.make_weights(config, seed=3)
    model = importlib.import_module("llm-inference-engine_b200.models.vasolix").VasolixModel(config, packed, dtype="float16", device="cuda:0", max_tokens=4096, max_seqs=1,
                                                                                              max_pages_per_seq=2200)
    serving = importlib.import_module("llm-inference-engine_b200.serving")
    toks = np.random.default_rng(0).integers(0, config["vocab"], 140000).tolist()
    rows = {}
    for how in ("portions", "decoded"):
        sess = serving.Session(model, len(toks) + 64, max_seqs=1, max_batch_tokens=4096, poison=True)
        i, at = sess.open(), 0
        for stop in (5000, 33000, 140000):
            while at < stop - 8:
                n = min(4096, stop - 8 - at)
                sess.feed([(i, toks[at:at + n], [])])
                at += n
            part = toks[at:stop]
            rows[how, stop] = sess.feed([(i, part, list(range(8)))]) if how == "portions" else torch.cat([sess.feed([(i, [x], [0])]) for x in part])
            at = stop
    for stop in (5000, 33000, 140000):
        a, b = rows["portions", stop].double(), rows["decoded", stop].double()
        assert not torch.isnan(b).any() and ((a - b).norm(dim=-1) / a.norm(dim=-1)).max() < TOL["float16"], stop


@pytest.mark.parametrize("each", [1, 7])
def test_the_same_every_time(each):
    """Forty sequences of a dozen blocks of keys, shared out over two CTAs a token and key head (one token each) or all of them in one CTA (seven): a step repeated from
    the same state gives every bit again, whatever the order in which warps and CTAs come to their sums."""
    config = vasolix_oracle.make_config([vasolix_oracle.attention_layer(heads=16, kv_heads=4, dim=128, size=4096, scale=128 ** -0.5)], width=128)
    _, packed = vasolix_oracle.make_weights(config, seed=4)
    seqs, pages = 40, 25
    model = importlib.import_module("llm-inference-engine_b200.models.vasolix").VasolixModel(config, packed, dtype="float16", device="cuda:0", max_tokens=2048, max_seqs=seqs,
                                                                                              max_pages_per_seq=pages)
    engine = model.engine
    engine.set_pools(seqs * pages, seqs)
    rng = np.random.default_rng(each)
    table = np.arange(seqs * pages).reshape(seqs, pages)
    lens = [1400 + 4 * i for i in range(seqs)]
    for i, n in enumerate(lens):
        engine.forward(rng.integers(0, config["vocab"], n), [0, n], [0], [i], table[i], [])
    ids, starts, rows = rng.integers(0, config["vocab"], seqs * each), [each * i for i in range(seqs + 1)], range(seqs * each)
    step = lambda: engine.forward(ids, starts, lens, range(seqs), table.reshape(-1), rows)  # noqa: E731
    want = step()
    assert not torch.isnan(want).any()
    for _ in range(150):
        assert torch.equal(step(), want)
