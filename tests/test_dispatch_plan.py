"""scripts/dispatch_plan.py restates the host-side kernel selection (decoder.cu / gemv_f32.cu / linear.cu / gemv_inst.cuh / gemv_qd.cuh / gemv_sr.cuh /
gemv_rs.cuh / gemv_mma.cuh) so that the plan of a decode step can be read without a GPU.  These cases pin it to the geometries of the dispatch (six 16 KB stages
per group for the bf16 GEMV at one token; whole-unit stages of gemv_rs, whose ring and sums share the SM; the sizes gemv_rs refuses; the forms of gemv_qd)."""
import os
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(ROOT, "scripts"))
import dispatch_plan as dp  # noqa: E402


def test_dense_batch1_geometry_matches_the_design_document():
    g = dp.gemv_nk_plan(1, 4096, "dense")
    assert g == dict(kernel="gemv_nk", pieces=1, piece_bytes=8192, stages=6)  # 6 stages x 16 KB x 2 groups = 192 KB in flight per SM
    g = dp.gemv_nk_plan(1, 11008, "dense")
    assert g["pieces"] == 3 and g["piece_bytes"] % 512 == 0 and g["pieces"] * g["piece_bytes"] >= 11008 * 2


@pytest.mark.parametrize("fmt", ["dense", "fp8", "int4"])
@pytest.mark.parametrize("k", [128, 4096, 4224, 11008, 28672])
@pytest.mark.parametrize("m", [1, 2, 8, 9, 16])
def test_streaming_gemv_geometry(fmt, k, m):
    """Parts cover the row in whole groups of 128 that a warp's eight blocks reach, and at least two stages fit beside the tiles and the parts' sums."""
    g = dp.gemv_rs_plan(m, k, 4096, fmt)
    if fmt == "dense" and m == 1:
        assert g is None
        return
    assert g["parts"] == max(1, -(-k // 4096)) and g["part_k"] % 128 == 0 and g["part_k"] <= 16 * 8 * 32
    assert g["parts"] * g["part_k"] >= k > (g["parts"] - 1) * g["part_k"]
    rows, nt = (8 if fmt == "dense" else 16), (2 if m > 8 else 1)
    stage = rows * (-(-g["piece_bytes"] // 128) * 128 + 64)
    tile, sums = (128, 128) if fmt == "dense" else (160 * nt, 128 * nt)
    units = -(-(-(-4096 // rows)) // 148)
    assert 2 <= g["stages"] <= 12
    assert g["stages"] * stage + 28 * 8 + 2 * 16 * tile * 4 + (units * sums * 4 if g["parts"] > 1 else 0) <= 226 * 1024


def test_streaming_gemv_stages():
    """16 tokens at K = 4096: two 64 KB FP8 stages beside the tiles, five INT4 ones, three dense ones; K = 11008 goes in three parts."""
    stages = {fmt: dp.gemv_rs_plan(16, 4096, 4096, fmt)["stages"] for fmt in ("dense", "fp8", "int4")}
    assert stages == {"dense": 3, "fp8": 2, "int4": 5}
    assert dp.gemv_rs_plan(16, 11008, 4096, "fp8")["parts"] == 3


def test_decode_batches_read_the_weights_once():
    """Every decode batch up to 16 is ONE pass over the weights, in every format, behind a norm kernel; one dense or INT4 token has the norm inside the GEMV."""
    for fmt in ("dense", "fp8", "int4"):
        for m in (1, 2, 4, 8, 16):
            for k, n in ((4096, 12288), (11008, 4096), (8192, 1280)):
                path, passes, geo = dp.linear_plan(m, k, n, fmt)
                streamed = fmt == "int4" and m <= 8 and not (k == 11008 and m == 8)  # (whose 8 tokens leave no room for what is in flight)
                want = "fused gemv_nk" if fmt == "dense" and m == 1 else "fused gemv_qd" if streamed and m == 1 else "norm_kernel + gemv_qd" if streamed else "norm_kernel + gemv_rs"
                assert passes == 1 and path == want, (fmt, m, k, path)
    # the linears without a norm in front (O, down), one behind a tensor-parallel exchange, and rows too long for the norm's registers
    assert dp.linear_plan(1, 4096, 4096, "int4", norm=False)[0] == "gemv_qd" and dp.linear_plan(1, 11008, 4096, "fp8", norm=False)[0] == "gemv_rs"
    assert dp.linear_plan(1, 2048, 4096, "dense", norm=False)[0] == "gemv_qd" and dp.linear_plan(1, 4096, 4096, "dense", norm=False)[0] == "gemv_nk"
    assert dp.linear_plan(1, 4096, 1536, "int4", tp=True)[0] == "norm_kernel + gemv_qd" and dp.linear_plan(1, 28672, 4096, "int4")[0] == "norm_kernel + gemv_qd"
    path, passes, _ = dp.linear_plan(32, 4096, 4096, "fp8")
    assert passes == 2 and path == "un-fused gemv_rs x 2 passes of <= 16 tokens"


@pytest.mark.parametrize("k", [128, 1024, 2048, 2176, 3072, 4096, 4224, 5120, 8192, 8832, 8960, 11008, 14336, 28672])
def test_int4_ring_of_registers(k):
    """Two CTAs of 8 warps per SM to 4096 k, while both hold the activations; else one of 16, which up to 8832 k holds 8 tokens; then the tokens that fit."""
    for m in range(1, 9):
        g = dp.gemv_qd_plan(m, k, 4096, "int4")
        one = 256 + 2 * 16 * 8 * 20 * 4 + m * (2 * k + 64) > 80 * 1024  # too much for two CTAs
        if g is None:
            assert k > 8832 and m >= (7 if k == 11008 else 5 if k == 14336 else 3 if k == 28672 else 8), m
            assert dp.gemv_any(m, k, 4096, "int4")["kernel"] == "gemv_rs"
            continue
        assert g["warps"] == (16 if k > 4096 or one else 8) and g["smem"] <= g["budget"] * g["warps"] // 16 and g["barriers"] == (1 if k <= 4096 else -(-k // 4096))
    assert dp.gemv_any(9, k, 4096, "int4")["kernel"] == "gemv_rs"
    assert dp.gemv_qd_plan(4, k, 2 * 12, "int4", swiglu=True) is None


def test_dense_ring_of_registers():
    """Every number of tokens to 3072 k, none beyond, whatever the output's type: a token's result does not depend on those beside it."""
    for k in range(128, 3072 + 1, 128):
        for m in range(1, 17):
            g = dp.gemv_qd_plan(m, k, 4096, "dense")
            assert g["kernel"] == "gemv_qd" and g["smem"] <= g["budget"] * g["warps"] // 16, (m, k)
            if m <= 8:
                assert g["warps"] == (8 if k <= 2048 else 16) and g["budget"] == 108 * 1024
    assert dp.gemv_qd_plan(16, 1024, 4096, "dense")["warps"] == 8 and dp.gemv_qd_plan(16, 1152, 4096, "dense")["warps"] == 16
    assert dp.gemv_qd_plan(16, 2048, 4096, "dense")["budget"] == 108 * 1024 and dp.gemv_qd_plan(16, 2176, 4096, "dense")["budget"] == 148 * 1024
    assert dp.gemv_qd_plan(2, 3200, 4096, "dense") is None and dp.gemv_any(2, 3200, 4096, "dense")["kernel"] == "gemv_rs"
    assert dp.gemv_qd_plan(17, 1024, 4096, "dense") is None and dp.gemv_qd_plan(2, 1000, 4096, "dense") is None


def test_whole_rows_per_warp():
    """One 16-bit token of at most 3072 k, one to four fp32 tokens of at most 1536 k: the rows' length says so for all numbers of tokens."""
    assert dp.linear_plan(1, 2048, 4096, "dense")[0] == "fused gemv_sr" and dp.linear_plan(1, 3328, 4096, "dense")[0] == "fused gemv_nk"
    assert dp.linear_plan(1, 2176, 4096, "dense")[0] == "fused gemv_nk"  # (no whole number of a warp's pieces)
    for m in range(1, 5):
        assert dp.gemv_sr_plan(m, 1536, 4)["smem"] <= 64 * 1024 and dp.gemv_sr_plan(m, 1664, 4) is None
    assert dp.gemv_sr_plan(5, 1024, 4) is None and dp.gemv_sr_plan(2, 1024, 2) is None
    # a tensor-parallel rank's partial: the kernels that push it to the other ranks
    assert dp.linear_plan(1, 1024, 8192, "dense", push=True)[0] == "fused gemv_nk" and dp.linear_plan(8, 1024, 8192, "dense", push=True)[0] == "norm_kernel + gemv_rs"


def test_sums_of_a_vocabulary_leave_no_ring():
    """Rows of more than 4096 k with vocabulary-sized outputs: the parts' sums fill the SM, and the kernel with the activations in shared memory takes over."""
    assert dp.linear_plan(16, 8192, 128256, "fp8")[0] == "norm_kernel + gemv_rs"
    path, passes, geo = dp.linear_plan(16, 8192, 152064, "fp8")
    assert (path, passes) == ("norm_kernel + gemv_mma", 1) and geo["parts"] * geo["part_k"] >= 8192 and geo["stages"] >= 3


def test_dense_batches_beyond_16_go_to_the_tensor_core_gemm():
    for m in (17, 32, 128):
        assert dp.linear_plan(m, 4096, 4096, "dense")[0].startswith("un-fused gemm_tc")
