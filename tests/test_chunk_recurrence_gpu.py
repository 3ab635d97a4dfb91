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


@pytest.mark.parametrize("which", LAYERS)
@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
def test_a_token_that_is_not_finite(which, dtype):
    """A token whose vectors overflow spoils itself and what comes after it, not what comes before it and not its neighbours in the batch: the same rows are
    finite, with the same values, as in portions that the serial kernels run."""
    name, oracle, layers = LAYERS[which]
    config, W, packed = model(name, oracle, layers)
    at, spoilt = 77, config["vocab"] - 1
    packed["embed"] = packed["embed"].copy() if isinstance(packed["embed"], np.ndarray) else packed["embed"].clone()
    packed["embed"][spoilt] = 3e38
    rng = np.random.default_rng(9)
    requests = {k: rng.integers(0, spoilt, 128).tolist() for k in "ab"}
    requests["a"][at] = spoilt
    whole = replay(session(name, config, packed, dtype, 512), requests, [[("a", 128), ("b", 128)]])
    parts = replay(session(name, config, packed, dtype, 512), requests, [[("a", 32), ("b", 32)]] * 4)
    for k in requests:
        whole[k], parts[k] = whole[k][:, :spoilt], parts[k][:, :spoilt]  # (a tied head's column of that token is not finite anywhere)
        finite = np.isfinite(parts[k]).all(-1)
        assert finite.tolist() == [k == "b" or t < at for t in range(128)], k
        assert (np.isfinite(whole[k]).all(-1) == finite).all(), k
        err = np.linalg.norm(whole[k][finite] - parts[k][finite], axis=-1) / np.linalg.norm(parts[k][finite], axis=-1)
        # fp32: both are sums of a few hundred terms; bf16: stored rows rounded on either side
        assert np.sort(err)[-1] < 2e-5 if dtype == "float32" else np.median(err) < 2e-2, (k, err.max())


b200 = importlib.import_module("llm-inference-engine_b200")
GLA, DELTA, LINEAR = 2, 5, 8  # b200_mixer_kind_t


def in_64_bits(q, k, v, g, beta):
    """One sequence: q, k, g [T, H, d], v [T, H, n], beta [T, H] or None -> read-outs, last state."""
    S, out = torch.zeros(q.shape[1], q.shape[2], v.shape[2], dtype=torch.float64, device=DEV), []
    for t in range(len(q)):
        S = S * g[t, :, :, None]
        u = v[t] if beta is None else beta[t, :, None] * (v[t] - torch.einsum("hdn,hd->hn", S, k[t]))
        S = S + k[t, :, :, None] * u[:, None]
        out.append(torch.einsum("hdn,hd->hn", S, q[t]))
    return torch.stack(out), S


@pytest.mark.parametrize("kind", ["gla", "delta", "linear"])
@pytest.mark.parametrize("dim", [64, 128])
@pytest.mark.parametrize("decays", ["slow", "mixed", "fast"])
@pytest.mark.parametrize("lens", [(64,), (200, 77), (1024,)], ids=str)
def test_no_further_from_64_bits_than_the_serial_kernels(kind, dim, decays, lens):
    """fp32 vectors, decays near 1, around 0.7 and around 0.15: read-outs and states of the chunked form against 64 bits, beside those of the serial form."""
    H, n, T = 2, 32, sum(lens)
    gen = torch.Generator(device=DEV).manual_seed(dim + T)
    rand = lambda *s: torch.randn(*s, generator=gen, device=DEV)  # noqa: E731
    per = (T, H, dim if kind != "linear" else 1)
    g = {"slow": 1 - 0.01 * torch.rand(*per, generator=gen, device=DEV), "mixed": torch.sigmoid(2 * rand(*per) + 1), "fast": torch.sigmoid(rand(*per) - 2)}[decays].contiguous()
    q, k, v, beta = rand(T, H, dim), rand(T, H, dim), rand(T, H, n), None
    if kind == "delta":
        q, k, beta = torch.nn.functional.normalize(q, dim=-1) / dim ** 0.5, torch.nn.functional.normalize(k, dim=-1), torch.sigmoid(rand(T, H))
    flat = lambda t: t.reshape(T, -1)  # noqa: E731
    none = torch.zeros(T, H * n, device=DEV)
    parts = {"gla": [q, k, v], "delta": [q, k, v, g, none, beta], "linear": [q, k, v, none, g]}[kind]
    rows = torch.cat([torch.nn.functional.pad(flat(p), (0, -flat(p).shape[1] % 4)) for p in parts], 1).contiguous()
    starts = [sum(lens[:i]) for i in range(len(lens) + 1)]
    meta = [torch.tensor(m, dtype=torch.int32, device=DEV) for m in (starts, [0] * len(lens), list(range(len(lens))))]
    lib, ptr = b200.lib(), lambda t: t.data_ptr()
    size = lib.b200_chunk_recurrence_scratch_bytes({"gla": GLA, "delta": DELTA, "linear": LINEAR}[kind], H, dim, T, len(lens))
    scratch = torch.empty(size, dtype=torch.uint8, device=DEV)
    want = [in_64_bits(*(p[a:b].double() for p in (q * (dim ** -0.5 if kind == "gla" else 1), k, v, g)), None if beta is None else beta[a:b].double())
            for a, b in zip(starts, starts[1:])]
    want = torch.cat([w[0] for w in want]), torch.stack([w[1] for w in want])
    errors = []
    for chunked in (False, True):
        state, o = torch.full((len(lens), H, dim, n), float("nan"), device=DEV), torch.zeros(T, H, n, device=DEV)
        at = (ptr(state), ptr(o), *map(ptr, meta), len(lens), H)
        if chunked:
            rc = lib.b200_chunk_recurrence({"gla": GLA, "delta": DELTA, "linear": LINEAR}[kind], ptr(rows), rows.shape[1], ptr(g), *at, H, dim, n, ptr(scratch), size, T,
                                           max(lens), b200.F32, b200.stream())
        elif kind == "gla":
            rc = lib.b200_gla_recurrent(ptr(rows), rows.shape[1], ptr(g), *at, dim, n, b200.F32, b200.stream())
        else:
            rc = (lib.b200_delta_rule_recurrent if kind == "delta" else lib.b200_decay_recurrent)(ptr(rows), *at, H, dim, n, b200.stream())
        b200.check(rc)
        errors.append([float((got.double() - w).norm() / w.norm()) for got, w in zip((o, state), want)])
    # (the same roundings in another order: 5 % for the spread of two samples of a few thousand values)
    assert all(c <= 1.05 * s for s, c in zip(*errors)), errors


@pytest.mark.parametrize("kind", ["gla", "delta", "linear"])
@pytest.mark.parametrize("dim", [64, 128])
@pytest.mark.parametrize("tail", [1, 2, 3, 4, 5, 8, 27, 28, 29, 31, 32, 33])
def test_last_chunks_of_every_length(kind, dim, tail):
    """The scan's update takes tokens in fours and the last four apart: portions that end anywhere in a chunk, beside one that ends with it."""
    test_no_further_from_64_bits_than_the_serial_kernels(kind, dim, "mixed", (96 + tail, 64))


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16], ids=["bf16", "f16"])
@pytest.mark.parametrize("rank", [32, 64, 256])
def test_decays_on_the_tensor_cores(dtype, rank):
    """Against 64 bits, beside the general kernel (which takes columns that do not start on a 16-byte boundary)."""
    T, channels, tau = 515, 1000, 16.0
    gen = torch.Generator(device=DEV).manual_seed(rank)
    rand = lambda *s: torch.randn(*s, generator=gen, device=DEV)  # noqa: E731
    x, w, bias = rand(T, rank).to(dtype), (2 * rand(channels, rank) / rank ** 0.5).to(dtype), rand(channels)
    want = torch.exp(torch.nn.functional.logsigmoid(x.double() @ w.double().T + bias.double()) / tau)
    errors = []
    for col0 in (1, 8):
        proj = torch.zeros(T, rank + 8, dtype=dtype, device=DEV)
        proj[:, col0:col0 + rank] = x
        got = torch.zeros(T, channels, device=DEV)
        b200.check(b200.lib().b200_gla_decay(proj.data_ptr(), rank + 8, col0, w.data_ptr(), bias.data_ptr(), tau, got.data_ptr(), T, rank, channels, b200.dtype_code(x), b200.stream()))
        errors.append(float((got.double().log() - want.log()).norm() / want.log().norm()))
    assert errors[1] <= 1.02 * errors[0], errors
