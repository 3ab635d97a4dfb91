#!/usr/bin/env python
"""Which kernel, how many passes over the weights and which ring geometry each linear of a decode step gets -- a Python MODEL of the host-side
dispatch (no GPU): decoder.cu norm_linear (norm inside the GEMV for one dense or INT4 token, a norm kernel in front otherwise) and plain_linear, gemv_f32.cu launch_gemv_nk
(gemv_qd for up to 8 tokens of INT4 and short dense rows, gemv_rs, what its ring refuses on gemv_mma, gemv_sr for one token of short rows, the SIMT GEMV for up
to 4 tokens), linear.cu (GEMV passes, tcgen05 GEMM for dense M > 16), gemv_inst.cuh, gemv_qd.cuh launch_gemv_qd_t, gemv_sr.cuh launch_gemv_sr_t, gemv_rs.cuh
gemv_rs_geometry and gemv_mma.cuh gemv_mma_geometry.  It restates those few formulas; when they change, this file must follow
(tests/test_dispatch_plan.py).
usage: python scripts/dispatch_plan.py > profiles/<tag>_dispatch_plan.txt"""
BUDGET = 224 * 1024
GROUPS, GW, MAX_STAGES, ROWS, PIECE = 2, 8, 8, 2, 8192
MMA_WARPS, MMA_ROWS = 16, 8
WARPS = GROUPS * GW


def gemv_nk_plan(M, K, fmt, ebytes=2):
    """gemv_inst.cuh launch_gemv_inst: None when unsupported, else dict(pieces, piece_bytes, stages)."""
    if M > 4:
        return None
    MB = 1 if M <= 1 else (2 if M <= 2 else 4)
    row_bytes = {"dense": K * ebytes, "fp8": K, "int4": K // 2}[fmt]
    pieces = -(-row_bytes // PIECE)
    piece_bytes = row_bytes if pieces == 1 else (-(-row_bytes // pieces) + 511) // 512 * 512
    pieces = -(-row_bytes // piece_bytes)
    stage_bytes = ROWS * ((piece_bytes + 127) // 128 * 128)
    block = {"dense": 1, "fp8": 512, "int4": 1024}[fmt]
    xs_bytes = ebytes if fmt == "dense" else 4
    Kp = -(-K // block) * block
    fixed = (MB * Kp * xs_bytes + 127) // 128 * 128 + GROUPS * (2 * MAX_STAGES + 4) * 8 + GROUPS * GW * 2 * ROWS * MB * 32 * 4
    per_stage = GROUPS * stage_bytes
    if fixed + 3 * per_stage > BUDGET:
        return None
    return dict(kernel="gemv_nk", pieces=pieces, piece_bytes=piece_bytes, stages=min((BUDGET - fixed) // per_stage, MAX_STAGES))


def gemv_mma_plan(M, K, fmt, max_units=8):
    """gemv_mma.cuh gemv_mma_geometry (16-bit activations, 1..16 tokens): None when unsupported."""
    if M < 1 or M > 16 or K % 128:
        return None
    dense = fmt == "dense"
    tok = 8 if M <= 8 else 16
    xs_rows = tok if M == tok else M + 1
    k_round = -(-K // 512) * 512
    best, best_score = None, -1
    piece_bytes0 = 2048 if fmt == "int4" else 4096
    while piece_bytes0 >= 1024:
        piece_bytes = piece_bytes0
        piece_bytes0 //= 2
        piece_k = piece_bytes // 2 if dense else (piece_bytes if fmt == "fp8" else piece_bytes * 2)
        if piece_k > k_round:
            piece_k = k_round
            piece_bytes = piece_k * 2 if dense else (piece_k if fmt == "fp8" else piece_k // 2)
        if fmt == "int4" and (piece_k // MMA_WARPS) % 128:
            continue
        if fmt == "int4" and piece_k // MMA_WARPS > 256:
            continue
        rg = 2 if fmt == "fp8" else 1  # row groups of 8 weight rows per unit
        row_stride = piece_bytes + (64 if dense else (32 if fmt == "fp8" else 16))
        stage_bytes = MMA_ROWS * rg * row_stride
        pieces_total = -(-K // piece_k)
        for parts in range(1, pieces_total + 1):
            ppp = -(-pieces_total // parts)
            if -(-pieces_total // ppp) != parts:
                continue
            part_k = ppp * piece_k
            tile = 16 * MMA_ROWS * rg * 4
            fixed = (xs_rows * (part_k + 32) * 2 + 127) // 128 * 128 + (2 * MAX_STAGES + 6) * 8 + 2 * MMA_WARPS * tile + (max_units * tile if parts > 1 else 0)
            if fixed + 3 * stage_bytes > 226 * 1024:
                continue
            stages = min((226 * 1024 - fixed) // stage_bytes, MAX_STAGES)
            score = min(stages * stage_bytes, 196608) + (49152 if piece_bytes >= 4096 else (0 if piece_bytes >= 2048 else -49152)) - (49152 if M <= 8 else 8192) * (parts - 1)
            if best is None or score > best_score:
                best_score = score
                best = dict(kernel="gemv_mma", pieces=pieces_total, piece_bytes=piece_bytes, stages=stages, parts=parts, part_k=part_k)
    return best


RS_BLOCKS, RS_STAGES, SMS = 8, 12, 148


def gemv_rs_plan(M, K, N, fmt, swiglu=False):
    """gemv_rs.cuh gemv_rs_geometry (16-bit activations, 1..16 tokens): None when unsupported."""
    if M < 1 or M > 16 or K % 128 or (fmt == "dense" and M == 1):
        return None
    dense, nt = fmt == "dense", 2 if M > 8 else 1
    rows = 8 if dense else 16
    units = -(-(N // 2) // (rows // 2)) if swiglu else -(-N // rows)
    max_units = -(-units // max(1, min(SMS, units)))
    groups = K // 128
    parts = -(-groups * 4 // (MMA_WARPS * RS_BLOCKS))
    part_k = -(-groups // parts) * 128
    parts = -(-K // part_k)
    row = {"dense": part_k * 2, "fp8": part_k, "int4": part_k // 2}[fmt]
    stage = rows * (-(-row // 128) * 128 + 64)
    tile, vals = (128, 128) if dense else (8 * nt * 20, 128 * nt)
    fixed = (2 * RS_STAGES + 4) * 8 + 2 * MMA_WARPS * tile * 4 + (max_units * vals * 4 if parts > 1 else 0)
    if fixed + 2 * stage > 226 * 1024:
        return None
    return dict(kernel="gemv_rs", pieces=parts, piece_bytes=row, stages=min((226 * 1024 - fixed) // stage, RS_STAGES), parts=parts, part_k=part_k)


def gemv_qd_plan(M, K, N, fmt, swiglu=False):
    """gemv_qd.cuh launch_gemv_qd_t (16-bit activations; INT4 in groups of 128 of 1..8 tokens, dense rows of at most 3072 k of 1..16): None when unsupported.
    warps: of a CTA (8: two CTAs per SM); barriers: of a unit of 16 rows."""
    dense = fmt == "dense"
    if fmt == "fp8" or M < 1 or M > (16 if dense else 8) or K % 128 or (dense and K > 3072) or (swiglu and N // 2 % 8):
        return None

    def smem(warps):
        return M * (2 * K + 64) + 256 + 2 * (warps if dense else 16) * (16 if M > 8 else 8) * 20 * 4

    budget = (108 if dense else 160) * 1024
    warps = 16 if K > (2048 if dense else 4096) or smem(8) > budget // 2 else 8
    if dense and warps == 16 and smem(16) > budget:
        budget = 148 * 1024
    if smem(warps) > budget * warps // 16:
        return None
    return dict(kernel="gemv_qd", warps=warps, smem=smem(warps), budget=budget, barriers=1 if dense or warps == 8 else -(-K // 4096))


def gemv_sr_plan(M, K, ebytes=2):
    """gemv_sr.cuh launch_gemv_sr_t (dense rows, norm in front or not; one 16-bit token, one to four fp32 tokens): None when unsupported."""
    if M < 1 or M > (1 if ebytes == 2 else 4) or K > (3072 if ebytes == 2 else 1536) or K % (32 * 16 // ebytes):
        return None
    return dict(kernel="gemv_sr", smem=(M if M <= 2 else 4) * K * 4 + K * ebytes)


def gemv_any(M, K, N, fmt, swiglu=False, push=False):
    """gemv_f32.cu launch_gemv_nk for a 16-bit model; push: a tensor-parallel rank's partial, which the kernels with a ring of registers leave to the others."""
    g = gemv_qd_plan(M, K, N, fmt, swiglu)
    if g and not push:
        return g
    if M <= 16 and (M >= 2 or fmt != "dense"):
        rows = 16 if fmt == "fp8" else 8
        units = -(-(N // 2) // (rows // 2)) if swiglu else -(-N // rows)
        g = gemv_rs_plan(M, K, N, fmt, swiglu) or gemv_mma_plan(M, K, fmt, -(-units // max(1, min(SMS, units))))
        if g:
            return g
    return (fmt == "dense" and not push and gemv_sr_plan(M, K)) or gemv_nk_plan(M, K, fmt)


def linear_plan(M, K, N, fmt, fused_rows=16, swiglu=False, push=False, norm=True, tp=False):
    """One linear of the decode step: (path, passes over the weights, geometry).  norm: residual and norm in front (QKV, gate-up); tp: a tensor-parallel exchange too."""
    if norm and M == 1 and fmt == "dense":  # the norm / residual / tensor-parallel prologue inside the GEMV
        g = (not push and gemv_sr_plan(M, K)) or gemv_nk_plan(M, K, fmt)
        if g:
            return ("fused " + g["kernel"], 1, g)
    if norm and M == 1 and fmt == "int4" and not tp and not push and K <= 16384:  # residual and norm in the norm kernel's order of summation
        g = gemv_qd_plan(M, K, N, fmt, swiglu)
        if g:
            return ("fused " + g["kernel"], 1, g)
    if M <= fused_rows:
        g = gemv_any(M, K, N, fmt, swiglu, push)
        if g:
            return (("norm_kernel + " if norm else "") + g["kernel"], 1, g)
    if fmt == "dense" and M > 4:
        return ("un-fused gemm_tc", 1, None)
    for step in (16, 8, 4):  # linear.cu: quantised weights in passes
        if M > (8 if step == 16 else 4) * step:
            continue
        plans = [gemv_any(min(step, M - m0), K, N, fmt) for m0 in range(0, M, step)]
        if all(plans):
            return (f"un-fused {plans[0]['kernel']} x {len(plans)} passes of <= {step} tokens", len(plans), plans[0])
    return ("un-fused generic SIMT fallback (launch_simt, linear.cu)", 1, None)


def step_plan(name, hidden, heads, kv_heads, d, inter, tp, batch, fmt):
    fused_rows = 16  # decoder.cu gemv_max_rows (16-bit models)
    shapes = [("qkv", hidden, (heads + 2 * kv_heads) * d // tp), ("o", heads * d // tp, hidden), ("gate_up", hidden, 2 * inter // tp),
              ("down", inter // tp, hidden)]
    lines = [f"{name}, batch {batch}, weights {fmt}" + (f", TP-{tp} (one rank)" if tp > 1 else "")]
    for lin, K, N in shapes:
        path, passes, g = linear_plan(batch, K, N, fmt, fused_rows, lin == "gate_up", tp > 1 and lin in ("o", "down"), lin in ("qkv", "gate_up"), tp > 1)
        if g and g["kernel"] == "gemv_qd":
            geo = f"ring of registers, {16 // g['warps']} CTAs of {g['warps']} warps per SM, barriers per 16 rows: {g['barriers']}"
        elif g and g["kernel"] == "gemv_sr":
            geo = "ring of registers, 2 CTAs of 8 warps per SM, a row per warp"
        else:
            geo = (f"pieces {g['pieces']} x {g['piece_bytes']} B, {g['stages']} stages" + (f", {g['parts']} activation parts of {g['part_k']} k" if g.get("parts") else "")) if g else "-"
        wbytes = K * N * {"dense": 2, "fp8": 1, "int4": 0.5}[fmt]
        lines.append(f"  {lin:8s} K={K:6d} N={N:6d}  {path:58s} weights read {passes} x {wbytes / 1e6:7.1f} MB   {geo}")
    return lines


CASES = [("Llama-2-7B", 4096, 32, 32, 128, 11008, 1, b, f) for f in ("dense", "fp8", "int4") for b in (1, 4, 8, 16, 32)] + \
        [("Llama-2-70B-shaped", 8192, 64, 8, 128, 28672, 8, b, "dense") for b in (1, 8)]

if __name__ == "__main__":
    print(__doc__.split("usage:")[0].strip() + "\n")
    for c in CASES:
        print("\n".join(step_plan(*c)) + "\n")
