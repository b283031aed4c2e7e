"""GPU parity of the tensor-core (tcgen05) skinny GEMM used for 9..64 activation rows.

The contraction runs on the tensor cores in K-slices, so the fp32 summation order differs from
the SIMT kernels and from the reference: the checks are the north-star tolerance (fp32 value
before the final round within 1e-3 of fp64 truth, relative to |value| + the row's RMS) and bf16
outputs within one rounding step of bf16(oracle).  Rows are independent in the reference kernel,
so the oracle for more than 8 rows is the reference arithmetic applied row by row."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

MODEL_SHAPES = [  # (out_features, in_features)
    (4096, 2048), (2048, 2048), (2048, 6144), (3072, 2048), (1024, 2048),
    (4096, 1024), (1024, 3072), (2048, 1024),
    (200, 64), (129, 128), (64, 192),      # ragged channel counts, short K
]


def case(orc, seed, n, k, rows):
    rng = np.random.default_rng(seed)
    w = rng.integers(-127, 128, size=(n, k), dtype=np.int8)
    s = (rng.uniform(0.5, 1.5, size=n) / (73.6 * np.sqrt(k))).astype(np.float32)
    x = orc.to_bf16(rng.standard_normal((rows, k)).astype(np.float32))
    return w, s, x


def check_bf16(orc, got, want, summand=None):
    """One bf16 rounding step of the value, or of the largest summand that was itself rounded
    to bf16 on the way (a residual add can cancel down to a small value)."""
    g, w = orc.from_bf16(got), orc.from_bf16(want)
    rms = np.sqrt((w ** 2).mean(axis=-1, keepdims=True))
    mag = np.maximum(np.abs(w), 0.25 * rms)
    if summand is not None:
        mag = np.maximum(mag, np.abs(orc.from_bf16(summand)).reshape(mag.shape))
    step = 2.0 ** -7 * mag
    bad = np.abs(g - w) > step
    assert not bad.any(), (int(bad.sum()), float(np.abs(g - w).max()))
    assert (g != w).mean() < 0.02, float((g != w).mean())


@pytest.mark.parametrize("n,k", MODEL_SHAPES)
@pytest.mark.parametrize("rows", [9, 16, 17, 33, 64])
def test_plain(orc, ops, n, k, rows):
    w, s, x = case(orc, rows, n, k, rows)
    out = ops.int8_gemm(w, s, x, want_f32=True)
    truth = orc.int8_gemm_rows_f64(w, s, x)
    rel = np.abs(out["f32"] - truth) / (np.abs(truth) + np.sqrt((truth ** 2).mean()))
    assert rel.max() <= 1.0e-3, rel.max()
    assert np.array_equal(out["y"], orc.to_bf16(out["f32"]))
    check_bf16(orc, out["y"], orc.int8_gemm_rows(w, s, x))


@pytest.mark.parametrize("n,k,rows", [(2048, 2048, 64), (2048, 6144, 20), (130, 256, 12)])
def test_residual(orc, ops, n, k, rows):
    w, s, x = case(orc, 1, n, k, rows)
    base = orc.to_bf16(np.random.default_rng(2).standard_normal((rows, n)).astype(np.float32))
    got = ops.int8_gemm_rows(w, s, x, y_in=base, mode=1)
    check_bf16(orc, got, orc.int8_gemm_rows(w, s, x, y_in=base, mode=1), summand=base)


@pytest.mark.parametrize("rows", [33, 47, 48, 49])
def test_row_tile_edges(orc, ops, rows):
    """Around the tile of 48 rows, with K in ragged slices and a last channel tile that is not full."""
    n, k = 1100, 1408
    w, s, x = case(orc, rows, n, k, rows)
    base = orc.to_bf16(np.random.default_rng(rows).standard_normal((rows, n)).astype(np.float32))
    got = ops.int8_gemm_rows(w, s, x, y_in=base, mode=1)
    check_bf16(orc, got, orc.int8_gemm_rows(w, s, x, y_in=base, mode=1), summand=base)


@pytest.mark.parametrize("n,k,rows", [(6144, 2048, 64), (3072, 1024, 16), (100, 128, 9), (64, 64, 33)])
def test_gate_up_silu(orc, ops, n, k, rows):
    rng = np.random.default_rng(3)
    w = rng.integers(-127, 128, size=(2 * n, k), dtype=np.int8)
    s = (rng.uniform(0.5, 1.5, size=2 * n) / (73.6 * np.sqrt(k))).astype(np.float32)
    x = orc.to_bf16(rng.standard_normal((rows, k)).astype(np.float32))
    got = ops.int8_gemm_rows(w, s, x, mode=2)
    check_bf16(orc, got, orc.int8_gate_up_silu_rows(w, s, x))


@pytest.mark.parametrize("rows", [12, 64])
def test_bias_epilogues_and_norm(orc, ops, rows):
    k, n = 2048, 1024
    rng = np.random.default_rng(4)
    w, s, x = case(orc, 4, n, k, rows)
    bias = orc.to_bf16((0.1 * rng.standard_normal(n)).astype(np.float32))
    resid = orc.to_bf16(rng.standard_normal((rows, n)).astype(np.float32))
    plain = orc.int8_gemm_rows(w, s, x)
    check_bf16(orc, ops.int8_gemm(w, s, x, epilogue=ops.EPI_BIAS, bias=bias)["y"],
               orc.bias_activation_rows(plain, bias, False))
    check_bf16(orc, ops.int8_gemm(w, s, x, epilogue=ops.EPI_BIAS_SILU, bias=bias)["y"],
               orc.bias_activation_rows(plain, bias, True))
    got = ops.int8_gemm(w, s, x, epilogue=ops.EPI_BIAS_ADD, bias=bias, resid=resid)["resid"]
    check_bf16(orc, got, orc.add(resid, orc.bias_activation_rows(plain, bias, False)).reshape(rows, n),
               summand=resid)
    # RMSNorm in front: same normalised rows as the stand-alone operator
    nw = orc.to_bf16((1.0 + 0.02 * rng.standard_normal(k)).astype(np.float32))
    fused = ops.int8_gemm(w, s, x, norm_w=nw, want_norm=True)
    normed = ops.rms_norm_rows(x, nw)
    assert np.array_equal(fused["norm"], normed)
    assert np.array_equal(fused["y"], ops.int8_gemm_rows(w, s, normed))


def test_deterministic_and_healthy(q3t, orc, ops):
    w, s, x = case(orc, 5, 2048, 2048, 64)
    a = ops.int8_gemm_rows(w, s, x)
    b = ops.int8_gemm_rows(w, s, x)
    assert np.array_equal(a, b)                       # K-slices are summed in slice order
    # a row's result does not depend on how many rows ride along, as long as the tile width is the same
    c = ops.int8_gemm_rows(w, s, x[:40])
    assert np.array_equal(a[:40], c)
    assert q3t.library().q3t_kernel_error_count() == 0


def prompt_case(orc, n, k, rows, gate_up=False):
    w, s, x = case(orc, n + rows, 2 * n if gate_up else n, k, rows)
    rng = np.random.default_rng(rows)
    return w, s, x, orc.to_bf16((0.1 * rng.standard_normal(n)).astype(np.float32)), orc.to_bf16(rng.standard_normal((rows, n)).astype(np.float32))


@pytest.mark.parametrize("kernel", [1, 2, 3])
@pytest.mark.parametrize("n,k,rows", [(300, 384, 65), (128, 128, 128), (129, 1152, 129), (640, 256, 161), (257, 512, 300), (1100, 2048, 128)])
def test_prompt_kernels(q3t, orc, ops, kernel, n, k, rows):
    """Projections of more than 64 rows: 128 rows and one or two tiles of channels a CTA (1, 2), or the lockstep kernel's row
    blocks side by side (3), with every epilogue that they have, at the edges of row blocks and of channel tiles (a last tile
    that is short, a second one that is not there), fewer steps than the rings hold and more."""
    w, s, x, bias, base = prompt_case(orc, n, k, rows)
    plain = orc.int8_gemm_rows(w, s, x)
    check_bf16(orc, ops.int8_gemm(w, s, x, prompt_kernel=kernel)["y"], plain)
    check_bf16(orc, ops.int8_gemm(w, s, x, epilogue=ops.EPI_ADD, y_in=base, prompt_kernel=kernel)["y"],
               orc.int8_gemm_rows(w, s, x, y_in=base, mode=1), summand=base)
    # the product is rounded to bf16 before the bias is added, and its rounding may fall the other way: an ulp of it, at most
    # 2^-7 |product|, through SiLU (slope at most 1.1) and a rounding of the result, 2^-8 (|product| + |bias|)
    summand = orc.to_bf16(1.6 * (np.abs(orc.from_bf16(plain)) + np.abs(orc.from_bf16(bias))).astype(np.float32))
    for epilogue, silu in ((ops.EPI_BIAS, False), (ops.EPI_BIAS_SILU, True)):
        check_bf16(orc, ops.int8_gemm(w, s, x, epilogue=epilogue, bias=bias, prompt_kernel=kernel)["y"],
                   orc.bias_activation_rows(plain, bias, silu), summand=summand)
    got = ops.int8_gemm(w, s, x, epilogue=ops.EPI_BIAS_ADD, bias=bias, resid=base, prompt_kernel=kernel)["resid"]
    check_bf16(orc, got, orc.add(base, orc.bias_activation_rows(plain, bias, False)).reshape(rows, n),
               summand=orc.to_bf16(np.maximum(np.abs(orc.from_bf16(base)), orc.from_bf16(summand)).astype(np.float32)))
    w, s, x, _, _ = prompt_case(orc, n, k, rows, gate_up=True)
    check_bf16(orc, ops.int8_gemm(w, s, x, epilogue=ops.EPI_GATE_UP_SILU, prompt_kernel=kernel)["y"],
               orc.int8_gate_up_silu_rows(w, s, x))
    assert q3t.library().q3t_kernel_error_count() == 0


@pytest.mark.parametrize("kernel", [96, 128, 160])
@pytest.mark.parametrize("n,k,rows", [(300, 384, 65), (128, 128, 97), (129, 1152, 161), (257, 512, 300), (2048, 6144, 150), (4096, 2048, 640)])
def test_tall_tiles(q3t, orc, ops, kernel, n, k, rows):
    """The lockstep kernel in blocks of 96, 128 or 160 rows: one step of K and many, K unsplit and in up to eight slices (whose
    exchange lies over the rings), rows that end inside a block and inside an owner's share, channels that end inside a tile."""
    w, s, x, bias, base = prompt_case(orc, n, k, rows)
    plain = orc.int8_gemm_rows(w, s, x)
    check_bf16(orc, ops.int8_gemm(w, s, x, prompt_kernel=kernel)["y"], plain)
    out = ops.int8_gemm(w, s, x, epilogue=ops.EPI_ADD, y_in=base, prompt_kernel=kernel)["y"]
    check_bf16(orc, out, orc.int8_gemm_rows(w, s, x, y_in=base, mode=1), summand=base)
    assert np.array_equal(out, ops.int8_gemm(w, s, x, epilogue=ops.EPI_ADD, y_in=base, prompt_kernel=kernel)["y"])
    # tolerance: as in test_prompt_kernels
    summand = orc.to_bf16(1.6 * (np.abs(orc.from_bf16(plain)) + np.abs(orc.from_bf16(bias))).astype(np.float32))
    check_bf16(orc, ops.int8_gemm(w, s, x, epilogue=ops.EPI_BIAS_SILU, bias=bias, prompt_kernel=kernel)["y"],
               orc.bias_activation_rows(plain, bias, True), summand=summand)
    w, s, x, _, _ = prompt_case(orc, n, k, rows, gate_up=True)
    check_bf16(orc, ops.int8_gemm(w, s, x, epilogue=ops.EPI_GATE_UP_SILU, prompt_kernel=kernel)["y"],
               orc.int8_gate_up_silu_rows(w, s, x))
    assert q3t.library().q3t_kernel_error_count() == 0


@pytest.mark.parametrize("n,k,rows", [(256, 128, 1), (300, 384, 65), (129, 1152, 161), (257, 512, 300), (512, 2048, 257)])
def test_pairs(q3t, orc, ops, n, k, rows):
    """Pairs of CTAs: one step of K and many, rows and channels that end inside a block, a chunk of sixteen and a CTA's half; each
    value within a rounding step of the oracle's, and the same twice.  Tolerance: as in test_prompt_kernels."""
    w, s, x, bias, base = prompt_case(orc, n, k, rows)
    plain = orc.int8_gemm_rows(w, s, x)
    check_bf16(orc, ops.int8_gemm(w, s, x, prompt_kernel=256)["y"], plain)
    out = ops.int8_gemm(w, s, x, epilogue=ops.EPI_ADD, y_in=base, prompt_kernel=256)["y"]
    check_bf16(orc, out, orc.int8_gemm_rows(w, s, x, y_in=base, mode=1), summand=base)
    assert np.array_equal(out, ops.int8_gemm(w, s, x, epilogue=ops.EPI_ADD, y_in=base, prompt_kernel=256)["y"])
    summand = orc.to_bf16(1.6 * (np.abs(orc.from_bf16(plain)) + np.abs(orc.from_bf16(bias))).astype(np.float32))
    for epilogue, silu in ((ops.EPI_BIAS, False), (ops.EPI_BIAS_SILU, True)):
        check_bf16(orc, ops.int8_gemm(w, s, x, epilogue=epilogue, bias=bias, prompt_kernel=256)["y"],
                   orc.bias_activation_rows(plain, bias, silu), summand=summand)
    got = ops.int8_gemm(w, s, x, epilogue=ops.EPI_BIAS_ADD, bias=bias, resid=base, prompt_kernel=256)["resid"]
    check_bf16(orc, got, orc.add(base, orc.bias_activation_rows(plain, bias, False)).reshape(rows, n),
               summand=orc.to_bf16(np.maximum(np.abs(orc.from_bf16(base)), orc.from_bf16(summand)).astype(np.float32)))
    w, s, x, _, _ = prompt_case(orc, n, k, rows, gate_up=True)
    check_bf16(orc, ops.int8_gemm(w, s, x, epilogue=ops.EPI_GATE_UP_SILU, prompt_kernel=256)["y"],
               orc.int8_gate_up_silu_rows(w, s, x))
    for bad in (dict(epilogue=ops.EPI_BIAS_ADD, bias=bias), dict(want_f32=True), dict(epilogue=ops.EPI_BIAS)):
        with pytest.raises(RuntimeError):
            ops.int8_gemm(w[:n], s[:n], x, prompt_kernel=256, **bad)
    assert q3t.library().q3t_kernel_error_count() == 0


@pytest.mark.parametrize("n,k,rows,gate_up", [(4096, 256, 1500, False), (2048, 1152, 2048, False), (4097, 384, 1201, False), (6144, 256, 1500, True), (6100, 640, 700, True)])
def test_pairs_of_several_tiles(q3t, orc, ops, n, k, rows, gate_up):
    """More tiles than pairs: every sum is made of the same products in the same order as with one tile a CTA, so every bit is."""
    w, s, x, _, base = prompt_case(orc, n, k, rows, gate_up)
    args = dict(epilogue=ops.EPI_GATE_UP_SILU) if gate_up else dict(epilogue=ops.EPI_ADD, y_in=base)
    assert np.array_equal(ops.int8_gemm(w, s, x, prompt_kernel=256, **args)["y"], ops.int8_gemm(w, s, x, prompt_kernel=1, **args)["y"])
    assert q3t.library().q3t_kernel_error_count() == 0


@pytest.mark.parametrize("rows,kernels", [(65, (96,)), (96, (96,)), (97, (128, 256)), (128, (128, 256))])
def test_gate_up_of_short_prompts(q3t, ops, rows, kernels):
    """The talker's gate/up of 65 to 128 rows goes to a kernel that was measured the shortest there or within 0.8 us of it, not to
    one tile a CTA (1.7 us longer than the tall tiles at 65 rows); the bits are the same, so they do not tell."""
    d = ops.GemmDescC()
    d.struct_size = C.sizeof(d)
    d.epilogue, d.in_features, d.out_features, d.rows = ops.EPI_GATE_UP_SILU, 2048, 6144, rows
    assert q3t.library().q3t_test_prompt_gemm_kernel(C.byref(d)) in kernels


@pytest.mark.parametrize("n,k,rows,gate_up", [(2048, 6144, 700, False), (4096, 2048, 1200, False), (2048, 2048, 2048, False), (6144, 2048, 600, True)])
def test_prompt_kernels_over_several_waves(q3t, orc, ops, n, k, rows, gate_up):
    """More CTAs than the GPU holds at once, at the talker's shapes; rows are compared with the lockstep kernel's, each within
    a rounding step of the other (both sum in fp32, in another order), and the choice by estimate is one of the three."""
    w, s, x, _, base = prompt_case(orc, n, k, rows, gate_up)
    args = dict(epilogue=ops.EPI_GATE_UP_SILU) if gate_up else dict(epilogue=ops.EPI_ADD, y_in=base)
    outs = [ops.int8_gemm(w, s, x, prompt_kernel=i, **args)["y"] for i in (0, 1, 2, 3)]
    blocks = np.concatenate([ops.int8_gemm(w, s, x[i:i + 64], **dict(args, **({} if gate_up else {"y_in": base[i:i + 64]})))["y"]
                             for i in range(0, rows, 64)])
    for out in outs:
        check_bf16(orc, out, blocks, summand=None if gate_up else base)
    assert any(np.array_equal(outs[0], out) for out in outs[1:])
    assert q3t.library().q3t_kernel_error_count() == 0


def test_prompt_kernels_refuse(ops, orc):
    w, s, x, bias, base = prompt_case(orc, 128, 128, 65)
    for bad in (dict(epilogue=ops.EPI_BIAS_ADD, bias=bias), dict(want_f32=True), dict(epilogue=ops.EPI_BIAS)):
        for kernel in (1, 2):
            with pytest.raises(RuntimeError):
                ops.int8_gemm(w, s, x, prompt_kernel=kernel, **bad)
    with pytest.raises(RuntimeError):
        ops.int8_gemm(w[:, :64].copy(), s, x[:, :64].copy(), prompt_kernel=1)      # K in steps of 128
    with pytest.raises(RuntimeError):
        ops.int8_gemm(w, s, np.resize(x, (2049, 128)), prompt_kernel=1)
