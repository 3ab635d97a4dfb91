"""Experts of prompts on row tiles of 32, 64 and 128 rows (hybrid.cu expert_tile, csrc/gemm_tc.cu launch_gemm_tc_grouped): rows per expert on both sides of every
size's range, experts that nobody chooses, one that all choose, inner sizes that fill no column tile; against the float64 restatement, as the other expert tests."""
import importlib

import numpy as np
import pytest
import torch

import vasolix_oracle as ref
from test_few_rows_gpu import ambiguous_rows

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,tol,u", [("bfloat16", 4e-2, 2.0 ** -8), ("float16", 6e-3, 2.0 ** -11)])
@pytest.mark.parametrize("tokens,experts,top,width,ff", [(65, 16, 2, 64, 72), (65, 3, 1, 128, 64), (85, 8, 2, 64, 64), (170, 8, 2, 128, 200), (196, 8, 2, 64, 64), (250, 16, 3, 64, 520),
                                                         (767, 8, 2, 64, 64), (769, 8, 2, 128, 136), (1500, 5, 1, 64, 264), (600, 3, 3, 64, 64),
                                                         # 32 rows an expert or fewer, planned by many CTAs (512 tokens and more)
                                                         (512, 26, 1, 64, 64), (700, 128, 3, 64, 72)])
def test_row_tiles(monkeypatch, dtype, tol, u, tokens, experts, top, width, ff):
    layer = ref.attention_layer(heads=2, kv_heads=1, dim=16, size=50, mlp=ref.moe(experts=experts, top=top, ff=ff, shared_ff=64))
    config = ref.make_config([layer], width=width, vocab=80)
    W, packed = ref.make_weights(config, seed=tokens)
    model = importlib.import_module("llm-inference-engine_b200.models.vasolix").VasolixModel(config, packed, dtype=dtype, device="cuda:0", max_tokens=tokens, max_seqs=2,
                                                                                              max_pages_per_seq=(tokens + 63) // 64)
    serving = importlib.import_module("llm-inference-engine_b200.serving")
    toks = np.random.default_rng(tokens).integers(0, 80, tokens).tolist()
    sess = serving.Session(model, 2 * (tokens + 64), max_seqs=2, max_batch_tokens=tokens, poison=True)
    got = sess.feed([(sess.open(), toks, range(tokens))]).cpu().numpy()
    want, open_rows = ambiguous_rows(monkeypatch, config, W, toks, u)
    assert not np.isnan(got).any()
    err = np.linalg.norm(got - want, axis=-1) / np.linalg.norm(want, axis=-1)
    assert (err[~open_rows] < tol).all(), (float(err[~open_rows].max()), int(err.argmax()))
    assert open_rows.mean() <= (0.0 if experts == top else 0.6)
