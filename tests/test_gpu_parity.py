"""GPU parity tests: every CUDA kernel, called through the C ABI, against the CPU oracle and the
golden vectors produced by the reference's own kernels.  Integer outputs and scales must match
bit for bit; bf16 results within 1e-2 relative Frobenius error (far tighter in practice)."""
import os

import numpy as np
import pytest
import torch

from golden_inputs import make_inputs
from oracle import ref_semantics as R

pytestmark = pytest.mark.gpu

if torch.cuda.is_available():
    from triton_int8_b200 import _lib as L
    from triton_int8_b200 import block_channel as BC
    from triton_int8_b200 import double_channel as DC
    from triton_int8_b200 import fused as FU
    from triton_int8_b200 import kernels as K

DEV = "cuda"
TOL_BF16 = 1e-2  # relative Frobenius error allowed for bf16 outputs


def _golden(golden_dir, name):
    return np.load(os.path.join(golden_dir, name + ".npz"))


def _same(t: torch.Tensor, ref, what=""):
    ref = torch.as_tensor(np.asarray(ref)) if not isinstance(ref, torch.Tensor) else ref
    t = t.detach().cpu()
    assert t.shape == ref.shape, f"{what}: shape {tuple(t.shape)} vs {tuple(ref.shape)}"
    bad = (t != ref).sum().item()
    assert bad == 0, f"{what}: {bad} of {t.numel()} entries differ"


def _status():
    return torch.zeros(1, dtype=torch.int32, device=DEV)


def _randq(g, *shape):
    return torch.randint(-127, 128, shape, generator=g, dtype=torch.int8)


# ------------------------------------------------------------------------------ quantizers
@pytest.mark.parametrize("case", ["small", "edge", "c1"])
def test_quant_tile_and_token_match_reference(golden_dir, case):
    a, w, b3 = make_inputs(case)
    aq_ref, as_ref = R.quant_tile128(a)
    q, s = BC.triton_per_block_quant(a.to(DEV))
    _same(q, aq_ref, "tile int8"); _same(s, as_ref, "tile scale")
    wq_ref, ws_ref = R.quant_token(w)
    q, s = BC.triton_per_token_quant(w.to(DEV))
    _same(q, wq_ref, "token int8"); _same(s, ws_ref, "token scale")
    if case != "c1":
        g = _golden(golden_dir, "block_channel_" + case)
        _same(BC.triton_per_block_quant(a.to(DEV))[0], g["aq"], "tile int8 vs golden")
        _same(BC.triton_per_block_quant(b3.to(DEV))[1], g["b_s_bwd"], "tile scale vs golden")


@pytest.mark.parametrize("gran", ["tile", "group"])
@pytest.mark.parametrize("mode", ["triton", "rne", "fused"])
def test_quant_tile_modes_and_transposed_output(gran, mode):
    g = torch.Generator().manual_seed(7)
    x = (torch.randn(2, 256, 384, generator=g) * 3).to(torch.bfloat16)
    x[0, :128, :128] = 0
    x[1, 5, 200] = 40.0
    G = L.GRAN_TILE128 if gran == "tile" else L.GRAN_GROUP128
    Mo = {"triton": L.QMODE_TRITON, "rne": L.QMODE_RNE, "fused": L.QMODE_FUSED}[mode]
    q, s, qt, st = K.quant_tile(x.to(DEV), G, Mo, 0, natural=True, transposed=True)

    def oracle(t):
        if mode == "triton":
            return R.quant_tile128(t) if gran == "tile" else R.quant_rowgroup128(t)
        if mode == "rne":
            return R.quant_tile128_rne(t) if gran == "tile" else R.quant_rowgroup128_rne(t)
        B, M, Kd = t.shape
        v = t.float().view(B, M // 128, 128, Kd // 128, 128) if gran == "tile" else t.float().view(B, M, Kd // 128, 128)
        am = v.abs().amax(dim=(2, 4) if gran == "tile" else 3, keepdim=True) + 1e-5
        sc = torch.full_like(am, 127.0) / am
        qq = torch.floor(v * sc + 0.5).to(torch.int8).view(B, M, Kd)
        return qq, sc.view(B, M // 128, Kd // 128) if gran == "tile" else sc.view(B, M, Kd // 128)

    q_ref, s_ref = oracle(x)
    _same(q, q_ref, "natural int8"); _same(s, s_ref, "natural scale")
    xt = x.transpose(1, 2).contiguous()
    qt_ref, st_ref = oracle(xt)
    _same(qt, qt_ref, "transposed int8"); _same(st, st_ref, "transposed scale")


def test_quant_row_modes_and_col_t():
    a, w, _ = make_inputs("dc_small")
    q, s = DC.triton_per_row_quant_3d(a.to(DEV))
    q_ref, s_ref = R.quant_row(a)
    _same(q, q_ref, "row int8"); _same(s, s_ref, "row scale")
    g = torch.Generator().manual_seed(11)
    w = (torch.randn(384, 1280, generator=g) * 0.02).to(torch.bfloat16)   # K not a power of two
    w[7] = 0
    q, s = BC.triton_per_token_quant(w.to(DEV))
    q_ref, s_ref = R.quant_token(w)
    _same(q, q_ref); _same(s, s_ref)
    q, s = BC.triton_per_token_quant(w.to(DEV), round="rne")
    q_ref, s_ref = R.quant_token_rne(w)
    _same(q, q_ref); _same(s, s_ref)
    qt, st = K.quant_col_t(w.to(DEV), L.QMODE_TRITON)          # W^T per input channel, for dX
    q_ref, s_ref = R.quant_token(w.t().contiguous())
    _same(qt, q_ref, "col_t int8"); _same(st, s_ref.view(-1), "col_t scale")
    qt, st = K.quant_col_t(w.to(DEV), L.QMODE_TRITON, hadamard=128)   # rotated along the rows of w (N)
    q_ref, s_ref = R.quant_token(R.hadamard(w.t().contiguous(), 128))
    _same(qt, q_ref, "rotated col_t int8"); _same(st, s_ref.view(-1), "rotated col_t scale")
    for had in (0, 128):   # the double_channel scale (127 / absmax as a reciprocal): transposed operands of its backward
        qt, st = K.quant_col_t(w.to(DEV), L.QMODE_ROWRCP, hadamard=had)
        wt = w.t().contiguous()
        q_ref, s_ref = R.quant_row((R.hadamard(wt, 128) if had else wt)[None])
        _same(qt, q_ref[0], f"rowrcp col_t int8, hadamard={had}"); _same(st, s_ref.view(-1), "rowrcp col_t scale")


@pytest.mark.parametrize("kind", ["tile128", "row128", "rowfull"])
def test_hadamard_fused_quantizers(kind):
    g = torch.Generator().manual_seed(13)
    if kind == "rowfull":
        x = torch.randn(2, 128, 2048, generator=g).to(torch.bfloat16)
        q, s = DC.triton_per_row_quant_3d(x.to(DEV), hadamard="full")
        q_ref, s_ref = R.quant_row(R.hadamard(x))
    elif kind == "row128":
        x = (torch.randn(256, 640, generator=g) * 0.02).to(torch.bfloat16)
        q, s = BC.triton_per_token_quant(x.to(DEV), hadamard=128)
        q_ref, s_ref = R.quant_token(R.hadamard(x, 128))
    else:
        x = torch.randn(2, 256, 384, generator=g).to(torch.bfloat16)
        q, s = BC.triton_per_block_quant(x.to(DEV), hadamard=128)
        q_ref, s_ref = R.quant_tile128(R.hadamard(x, 128))
    # same butterfly order as the oracle -> bit-equal; a different FWHT order could differ by 1 LSB on ties
    _same(q, q_ref, "rotated int8"); _same(s, s_ref, "rotated scale")


# ------------------------------------------------------------------------------ int32 accumulators
@pytest.mark.parametrize("shape", [(1, 128, 128, 128), (1, 128, 256, 256), (2, 256, 384, 640),
                                   (1, 2048, 4096, 512), (3, 128, 128, 1152)])
@pytest.mark.parametrize("b_batched", [False, True])
def test_gemm_int32_accumulators_bit_exact(shape, b_batched):
    B, M, N, Kd = shape
    g = torch.Generator().manual_seed(B * 1000 + M + N + Kd)
    aq = _randq(g, B, M, Kd)
    bq = _randq(g, B, N, Kd) if b_batched else _randq(g, N, Kd)
    st = _status()
    out = K.gemm_dump_i32(aq.to(DEV), bq.to(DEV), per_block=False, status=st)
    assert st.item() == 0
    _same(out, R.gemm_i32(aq, bq), "whole-K int32")
    outb = K.gemm_dump_i32(aq.to(DEV), bq.to(DEV), per_block=True, status=st)
    assert st.item() == 0
    ref = torch.stack([R.gemm_i32(aq[:, :, k:k + 128].contiguous(), bq[..., k:k + 128].contiguous())
                       for k in range(0, Kd, 128)], dim=1)
    _same(outb, ref, "per-K-block int32")


def test_gemm_int32_extreme_values():
    """All operands at +-127/-128: partial sums reach 128*128*128 per K block, K*16129 overall."""
    aq = torch.full((1, 128, 1024), -128, dtype=torch.int8)
    bq = torch.full((256, 1024), -128, dtype=torch.int8)
    bq[::2] = 127
    out = K.gemm_dump_i32(aq.to(DEV), bq.to(DEV))
    _same(out, R.gemm_i32(aq, bq))


# ------------------------------------------------------------------------------ scaled GEMMs
@pytest.mark.parametrize("case", ["small", "edge"])
def test_block_channel_exact_mode_equals_reference_kernels(golden_dir, case):
    g = _golden(golden_dir, "block_channel_" + case)
    a, w, b3 = make_inputs(case)
    aq, a_s = BC.triton_per_block_quant(a.to(DEV))
    wq, w_s = BC.triton_per_token_quant(w.to(DEV))
    c = BC.triton_gemm(aq, wq, a_s, w_s, out_dtype=torch.float32, exact=True)
    _same(c, g["c_fwd"], "fwd fp32 vs reference kernel output")
    bq, b_s = BC.triton_per_block_quant(b3.to(DEV))
    c2 = BC.triton_gemm(aq, bq, a_s, b_s, out_dtype=torch.float32, exact=True)
    _same(c2, g["c_bwd"], "bwd fp32 vs reference kernel output")
    # default (fast) path: same integers, scale factors regrouped -> within tolerance, bf16 output
    y = BC.fwd_32(a.to(DEV), w.to(DEV))
    assert R.rel_fro(y.cpu().float(), torch.as_tensor(g["c_fwd"])) < TOL_BF16
    y2 = BC.bwd_33(a.to(DEV), b3.to(DEV))
    assert R.rel_fro(y2.cpu().float(), torch.as_tensor(g["c_bwd"])) < TOL_BF16
    _same(BC.fwd_32(a.to(DEV), w.to(DEV), exact=True), torch.as_tensor(g["c_fwd"]).to(torch.bfloat16), "bf16 exact")


def test_block_channel_config1_both_wordings():
    """The 512x1024x1024 configuration (8 outlier columns): reference scaling (tile128, half up) and the
    per-(row,128)/RNE wording, forward + dX + dW by composition of the two primitives."""
    a, w, dy = make_inputs("c1")
    x = a[0]
    y_ref, dx_ref, dw_ref = R.linear_block_channel(x, w, dy[0])
    xd, wd, dyd = x.to(DEV), w.to(DEV), dy[0].to(DEV)
    y = BC.fwd_32(xd[None], wd)[0]
    dx = BC.fwd_32(dyd[None], wd.t().contiguous())[0]
    dw = BC.bwd_33(dyd.t().contiguous()[None], xd.t().contiguous()[None])[0]
    for got, ref, name in ((y, y_ref, "Y"), (dx, dx_ref, "dX"), (dw, dw_ref, "dW")):
        err = R.rel_fro(got.cpu().float(), ref.float())
        assert err < TOL_BF16, f"{name}: rel fro {err}"
    # row128 / rne wording
    aq, a_s = R.quant_rowgroup128_rne(a)
    wq, w_s = R.quant_token_rne(w)
    ref = R.gemm_block_general(aq, wq, a_s, w_s.view(-1), 1, "channel").to(torch.bfloat16)
    got = BC.fwd_32(xd[None], wd, scaling="row128", round="rne")
    assert R.rel_fro(got.cpu().float(), ref.float()) < TOL_BF16
    got_exact = BC.fwd_32(xd[None], wd, scaling="row128", round="rne", exact=True)
    _same(got_exact, ref, "row128/rne exact bf16")


def test_double_channel_matches_reference_kernels(golden_dir):
    g = _golden(golden_dir, "double_channel_small")
    a, w, b3 = make_inputs("dc_small")
    aq, a_s = DC.triton_per_row_quant_3d(a.to(DEV))
    wq, w_s = DC.triton_per_row_quant_2d(w.to(DEV))
    _same(aq, g["aq"]); _same(a_s, g["a_s"]); _same(wq, g["wq"]); _same(w_s, g["w_s"])
    _same(DC.triton_gemm(aq, wq, a_s, w_s, out_dtype=torch.float32), g["c_fwd"], "fwd fp32")
    bq, b_s = DC.triton_per_row_quant_3d(b3.to(DEV))
    _same(DC.triton_gemm(aq, bq, a_s, b_s, out_dtype=torch.float32), g["c_bwd"], "bwd fp32")
    # whole pipeline incl. the rotation and the bf16 `C * 1/K` pass, against the oracle
    _same(DC.fwd_32(a.to(DEV), w.to(DEV)), R.double_channel_fwd_32(a, w), "fwd_32 bf16")
    _same(DC.bwd_33(a.to(DEV), b3.to(DEV)), R.double_channel_bwd_33(a, b3), "bwd_33 bf16")
    _same(DC.fwd_32(a.to(DEV), w.to(DEV), hadamard=None), R.double_channel_fwd_32(a, w, use_hadamard=False))


def test_fused_matches_reference_kernels(golden_dir):
    g = _golden(golden_dir, "fused_small")
    a, w, b3 = make_inputs("small")
    _same(FU.fused_int8_gemm(a.to(DEV), w.to(DEV), out_dtype=torch.float32, exact=True), g["c_fwd"], "fused fwd fp32")
    _same(FU.fused_int8_gemm(a.to(DEV), b3.to(DEV), out_dtype=torch.float32, exact=True), g["c_bwd"], "fused bwd fp32")
    # default (fast) path: reciprocal instead of division, fused accumulation
    for got, ref in ((FU.fused_int8_gemm(a.to(DEV), w.to(DEV), out_dtype=torch.float32), g["c_fwd"]),
                     (FU.fused_int8_gemm(a.to(DEV), b3.to(DEV), out_dtype=torch.float32), g["c_bwd"])):
        assert R.rel_fro(got.cpu(), torch.as_tensor(ref)) < 1e-5
    assert R.rel_fro(FU.fwd_32(a.to(DEV), w.to(DEV)).cpu().float(), torch.as_tensor(g["c_fwd"])) < TOL_BF16
    assert R.rel_fro(FU.bwd_33(a.to(DEV), b3.to(DEV)).cpu().float(), torch.as_tensor(g["c_bwd"])) < TOL_BF16


def test_reference_acceptance_gate():
    """calc_diff < 1e-3 against the bf16 product on N(0,1) inputs: the reference's own check
    (triton/block_channel_fwd32.py:257-272 and siblings), at 2 x 1024^3."""
    g = torch.Generator().manual_seed(3)
    a = torch.randn(2, 1024, 1024, generator=g).to(torch.bfloat16).to(DEV)
    w = torch.randn(1024, 1024, generator=g).to(torch.bfloat16).to(DEV)
    b3 = torch.randn(2, 1024, 1024, generator=g).to(torch.bfloat16).to(DEV)
    ref_f = torch.matmul(a, w.t())
    ref_b = torch.matmul(a, b3.transpose(1, 2))
    for mod in (BC, DC, FU):
        assert mod.calc_diff(mod.fwd_32(a, w), ref_f) < 1e-3
        assert mod.calc_diff(mod.bwd_33(a, b3), ref_b) < 1e-3


def test_bias_and_hadamard128_forward():
    g = torch.Generator().manual_seed(5)
    x = torch.randn(1, 256, 512, generator=g).to(torch.bfloat16)
    w = (torch.randn(384, 512, generator=g) * 0.02).to(torch.bfloat16)
    bias = (torch.randn(384, generator=g) * 0.01).to(torch.bfloat16)
    y_ref, _, _ = R.linear_block_channel(x[0], w, torch.zeros(256, 384, dtype=torch.bfloat16), hadamard128=True, bias=bias)
    y = BC.fwd_32(x.to(DEV), w.to(DEV), hadamard=128, bias=bias.to(DEV))[0]
    assert R.rel_fro(y.cpu().float(), y_ref.float()) < TOL_BF16
    y = BC.fwd_32(x.to(DEV), w.to(DEV), hadamard=128, bias=bias.to(DEV), exact=True)[0]
    _same(y, y_ref, "hadamard128 + bias, exact order")


# ------------------------------------------------------------------------------ error behaviour
def test_errors_are_reported_not_swallowed():
    from triton_int8_b200 import I8LError
    x = torch.zeros(1, 100, 128, dtype=torch.bfloat16, device=DEV)
    with pytest.raises(I8LError, match="SHAPE"):
        BC.triton_per_block_quant(x)
    with pytest.raises(ValueError):
        BC.triton_per_block_quant(torch.zeros(1, 128, 128, dtype=torch.bfloat16))   # CPU tensor: no fallback
    with pytest.raises(TypeError):
        BC.triton_per_block_quant(torch.zeros(1, 128, 128, device=DEV))             # fp32 input


@pytest.mark.parametrize("gran", ["tile", "group"])
def test_hadamard_along_tokens_for_transposed_operand(gran):
    """The dW operands are x^T rotated along the tokens (rows of x): bit-equal to the oracle applied to
    the materialised transpose."""
    g = torch.Generator().manual_seed(17)
    x = (torch.randn(2, 256, 384, generator=g) * 2).to(torch.bfloat16)
    x[0, 3, 5] = 60.0
    G = L.GRAN_TILE128 if gran == "tile" else L.GRAN_GROUP128
    _, _, qt, st = K.quant_tile(x.to(DEV), G, L.QMODE_TRITON, 128, natural=False, transposed=True)
    xt_rot = R.hadamard(x.transpose(1, 2).contiguous(), 128)
    q_ref, s_ref = R.quant_tile128(xt_rot) if gran == "tile" else R.quant_rowgroup128(xt_rot)
    _same(qt, q_ref, "rotated transposed int8"); _same(st, s_ref, "rotated transposed scale")


# ------------------------------------------------------------------------------ TileLang variant numerics
@pytest.mark.parametrize("case", ["small", "edge"])
def test_tilelang_variant_quantizers_and_gemm(golden_dir, case):
    """scaling="tile128x256_bf16scale": activation scale per 128 x 256, scales rounded to bf16, scale
    product first (tilelang/block_channel_fwd.py:33,75-81,185-204).  The quantizers are checked against
    the reference's own Triton kernels (golden, unrounded scales + the bf16 rounding a GPU store applies),
    the GEMM against the cited restatement."""
    g = _golden(golden_dir, "tilelang_quantizers")
    a, w, b3 = make_inputs(case)
    aq, a_s = BC.triton_per_block256_quant(a.to(DEV))
    wq, w_s = BC.triton_per_token_quant_bf16scale(w.to(DEV))
    _same(aq, g[f"{case}__aq"], "128x256 int8"); _same(wq, g[f"{case}__wq"], "row int8")
    _same(a_s, torch.as_tensor(g[f"{case}__a_s_f32"]).to(torch.bfloat16).float(), "128x256 scale (bf16-rounded)")
    _same(w_s, torch.as_tensor(g[f"{case}__w_s_f32"]).to(torch.bfloat16).float(), "row scale (bf16-rounded)")
    ref = R.tilelang_fwd_32(a, w, return_fp32=True)
    got = BC.fwd_32(a.to(DEV), w.to(DEV), scaling="tile128x256_bf16scale", exact=True, out_dtype=torch.float32)
    _same(got, ref, "TileLang forward numerics, exact order, fp32")
    fast = BC.fwd_32(a.to(DEV), w.to(DEV), scaling="tile128x256_bf16scale")
    assert R.rel_fro(fast.cpu().float(), ref) < TOL_BF16
    ref_b = R.tilelang_bwd_33(a, b3, return_fp32=True)
    got_b = BC.bwd_33(a.to(DEV), b3.to(DEV), scaling="tilelang_tile128", exact=True, out_dtype=torch.float32)
    _same(got_b, ref_b, "TileLang backward numerics, exact order, fp32")
    assert R.rel_fro(BC.bwd_33(a.to(DEV), b3.to(DEV), scaling="tilelang_tile128").cpu().float(), ref_b) < TOL_BF16


def test_rowcol_fp32_output_applies_post_scale_and_bias():
    """double_channel pipeline with an fp32 result: the 1/K rescale and the bias are applied in fp32
    (the reference multiplies its GEMM output, whatever its type, by 1/K:
    triton/double-channle_fwd32.py:284)."""
    a, w, _ = make_inputs("dc_small")
    bias = (torch.arange(w.shape[0], dtype=torch.float32) * 1e-3).to(torch.bfloat16)
    for had in ("full", 128, None):
        rot = (lambda t: R.hadamard(t)) if had == "full" else ((lambda t: R.hadamard(t, 128)) if had == 128 else (lambda t: t))
        aq, a_s = R.quant_row(rot(a)); wq, w_s = R.quant_row(rot(w))
        post = 1.0 / a.shape[-1] if had == "full" else (1.0 / 128 if had == 128 else 1.0)
        ref = R.gemm_rowcol(aq, wq, a_s, w_s) * post + bias.float()
        got = DC.int8_gemm_pipeline(a.to(DEV), w.to(DEV), out_dtype=torch.float32, hadamard=had, bias=bias.to(DEV))
        _same(got, ref, f"fp32 double_channel pipeline, hadamard={had}")


@pytest.mark.parametrize("mode", ["triton", "rne"])
def test_rotated_operand_pair_from_one_read(mode):
    """hadamard=128 with both outputs requested: q (rotated along the columns) and qt (the transpose,
    rotated along the rows) come from one kernel that reads each tile once; both must equal the oracle,
    and the two single-output kernels, bit for bit."""
    g = torch.Generator().manual_seed(23)
    x = (torch.randn(2, 384, 256, generator=g) * 2).to(torch.bfloat16)
    x[0, :128, :128] = 0
    x[1, 130, 7] = -90.0
    x[0, 200:210, 129] = 33.0
    Mo = L.QMODE_TRITON if mode == "triton" else L.QMODE_RNE
    oracle = R.quant_tile128 if mode == "triton" else R.quant_tile128_rne
    q, s, qt, st = K.quant_tile(x.to(DEV), L.GRAN_TILE128, Mo, 128, natural=True, transposed=True)
    q_ref, s_ref = oracle(R.hadamard(x, 128))
    qt_ref, st_ref = oracle(R.hadamard(x.transpose(1, 2).contiguous(), 128))
    _same(q, q_ref, "q"); _same(s, s_ref, "scale"); _same(qt, qt_ref, "qt"); _same(st, st_ref, "scale_t")
    q1, s1, _, _ = K.quant_tile(x.to(DEV), L.GRAN_TILE128, Mo, 128, natural=True, transposed=False)
    _, _, qt1, st1 = K.quant_tile(x.to(DEV), L.GRAN_TILE128, Mo, 128, natural=False, transposed=True)
    assert torch.equal(q, q1) and torch.equal(s, s1) and torch.equal(qt, qt1) and torch.equal(st, st1)


@pytest.mark.parametrize("spread", ["smooth", "wild"])
def test_fast_block_epilogue_accuracy_deep_k(spread):
    """The fast block-scaled epilogue takes the int32 partials as floats shifted by a constant, whose multiple the
    accumulators carry for four K blocks at a time.
    At K = 32768 (256 K blocks), with per-tile scales that are smooth or jump by three decades from one
    K block to the next, the fp32 result must stay within 1e-4 (relative Frobenius) of the float64 value of
    sum_kb P_kb * a_s * b_s, like the reference-order mode."""
    M, N, Kd = 256, 512, 32768
    g = torch.Generator().manual_seed(41)
    aq, bq = _randq(g, 1, M, Kd), _randq(g, N, Kd)
    if spread == "smooth":
        a_s = torch.rand(1, M // 128, Kd // 128, generator=g) * 0.5 + 0.75
    else:
        a_s = 10.0 ** (torch.rand(1, M // 128, Kd // 128, generator=g) * 3.0 - 1.5)
    b_s = torch.rand(N, generator=g) + 0.5
    ref = torch.zeros(M, N, dtype=torch.float64)
    for kb in range(Kd // 128):
        P = R.int_mm(aq[0, :, kb * 128:(kb + 1) * 128], bq[:, kb * 128:(kb + 1) * 128]).double()
        ref += P * a_s[0, :, kb].double().repeat_interleave(128).view(M, 1)
    ref *= b_s.double().view(1, N)
    args = (aq.to(DEV), bq.to(DEV), a_s.to(DEV), b_s.to(DEV))
    fast = K.gemm_block(*args, flags=L.GEMM_OUT_F32)[0].cpu().double()
    exact = K.gemm_block(*args, flags=L.GEMM_OUT_F32 | L.GEMM_EXACT_ORDER)[0].cpu().double()
    e_fast, e_exact = R.rel_fro(fast, ref), R.rel_fro(exact, ref)
    assert e_exact < 1e-6, e_exact
    assert e_fast < 1e-4, (e_fast, e_exact)
    # tile x tile scales (the dW layout) through the same kind
    b_t = torch.rand(N // 128, Kd // 128, generator=g) + 0.5
    ref2 = torch.zeros(M, N, dtype=torch.float64)
    for kb in range(Kd // 128):
        P = R.int_mm(aq[0, :, kb * 128:(kb + 1) * 128], bq[:, kb * 128:(kb + 1) * 128]).double()
        ref2 += P * a_s[0, :, kb].double().repeat_interleave(128).view(M, 1) * b_t[:, kb].double().repeat_interleave(128).view(1, N)
    fast2 = K.gemm_block(args[0], args[1], args[2], b_t.to(DEV), b_kind=L.BSCALE_TILE, flags=L.GEMM_OUT_F32)[0].cpu().double()
    assert R.rel_fro(fast2, ref2) < 1e-4


def test_single_kernel_fused_matches_reference_kernels(golden_dir):
    """i8l_fused_gemm: bf16 in, result out, operand tiles quantized inside the GEMM.  Reference operation
    order: bit-equal to the reference's fused kernels (golden); default order: equal to the two-step path."""
    g = _golden(golden_dir, "fused_small")
    a, w, b3 = make_inputs("small")
    ad, wd, bd = a.to(DEV), w.to(DEV), b3.to(DEV)
    _same(FU.fused_int8_gemm(ad, wd, out_dtype=torch.float32, exact=True, single_kernel=True), g["c_fwd"], "single-kernel fwd fp32")
    _same(FU.fused_int8_gemm(ad, bd, out_dtype=torch.float32, exact=True, single_kernel=True), g["c_bwd"], "single-kernel bwd fp32")
    for other in (wd, bd):
        one = FU.fused_int8_gemm(ad, other, out_dtype=torch.float32, single_kernel=True)
        two = FU.fused_int8_gemm(ad, other, out_dtype=torch.float32)
        assert R.rel_fro(one.cpu(), two.cpu()) < 1e-6
        assert torch.equal(FU.fused_int8_gemm(ad, other, single_kernel=True), FU.fused_int8_gemm(ad, other).to(torch.bfloat16)) or \
            R.rel_fro(FU.fused_int8_gemm(ad, other, single_kernel=True).cpu().float(), two.cpu()) < TOL_BF16
    # a shape with more tiles than SMs and a deeper K, against the exact product (the reference's gate)
    gen = torch.Generator().manual_seed(9)
    a2 = torch.randn(1, 2048, 2048, generator=gen).to(torch.bfloat16).to(DEV)
    w2 = torch.randn(1536, 2048, generator=gen).to(torch.bfloat16).to(DEV)
    y = FU.fwd_32(a2, w2, single_kernel=True)
    assert FU.calc_diff(y, torch.matmul(a2, w2.t())) < 1e-3
    assert R.rel_fro(y.cpu().float(), FU.fwd_32(a2, w2).cpu().float()) < 1e-2
    K.check_status(DEV)


def test_fast_block_epilogue_more_than_512_k_blocks():
    """K = 73728 = 576 K blocks: the factors of a tile are handed over in three chunks (256 + 256 + 64); int32
    partials via the dump entry, fp32 result against float64."""
    M, N, Kd = 128, 256, 128 * 576
    g = torch.Generator().manual_seed(43)
    aq, bq = _randq(g, 1, M, Kd), _randq(g, N, Kd)
    a_s = torch.rand(1, 1, Kd // 128, generator=g) + 0.5
    b_s = torch.rand(N, generator=g) + 0.5
    P = K.gemm_dump_i32(aq.to(DEV), bq.to(DEV), per_block=True)[0].cpu()          # [KB, M, N]
    ref = (P.double() * a_s[0, 0].double().view(-1, 1, 1)).sum(0) * b_s.double().view(1, N)
    for b_scale, kind in ((b_s, L.BSCALE_CHANNEL),):
        fast = K.gemm_block(aq.to(DEV), bq.to(DEV), a_s.to(DEV), b_scale.to(DEV), b_kind=kind, flags=L.GEMM_OUT_F32)[0].cpu().double()
        assert R.rel_fro(fast, ref) < 1e-4
    K.check_status(DEV)


@pytest.mark.parametrize("cols", [384, 8192, 8192 + 384])
def test_rotated_row_quantizer_both_kernels(cols):
    """Per-row scale with the 128-point rotation: rows of up to 8192 elements take the kernel that keeps the
    rotated row in registers, longer rows the two-sweep kernel; both must equal the oracle bit for bit."""
    g = torch.Generator().manual_seed(cols)
    w = (torch.randn(160, cols, generator=g) * 0.05).to(torch.bfloat16)
    w[3] = 0
    w[7, cols - 1] = 9.0
    q, s = K.quant_row(w.to(DEV), L.QMODE_TRITON, 128)
    q_ref, s_ref = R.quant_token(R.hadamard(w, 128))
    _same(q, q_ref, "rotated row int8"); _same(s, s_ref.view(-1), "rotated row scale")


@pytest.mark.parametrize("kb,n,values,decade", [
    (1, 256, "random", 0), (2, 384, "random", 0), (3, 128, "random", 30), (5, 256, "random", -30), (6, 640, "random", 0),
    (7, 256, "lowest", 0), (4, 256, "opposite", 0), (257, 128, "random", 0)])
def test_fast_block_epilogue_shift(kb, n, values, decade):
    """The tensor core adds 32 * 255^2 to every partial product so that its bits are a float: the extreme int8
    operands (all products 128 * 128, all -128 * 127), numbers of K blocks around the group of four after which
    the shift is taken out and around the 256 staged at a time, partial tiles, and factors far from one.
    Bound: an fp32 operation on a value up to |sum| + two shifts rounds by 2^-24 of it; one per K block, one per
    four for the correction, three at the end."""
    g = torch.Generator().manual_seed(100 + kb)
    M, Kd = 128, 128 * kb
    aq, bq = _randq(g, 1, M, Kd), _randq(g, n, Kd)
    if values == "lowest":
        aq.fill_(-128), bq.fill_(-128)
    elif values == "opposite":
        aq.fill_(-128), bq.fill_(127)
    a_s = (torch.rand(1, 1, kb, generator=g) + 0.5) * 10.0 ** decade
    b_t = torch.rand(n // 128, kb, generator=g) + 0.5
    P = torch.stack([R.int_mm(aq[0, :, k * 128:(k + 1) * 128], bq[:, k * 128:(k + 1) * 128]) for k in range(kb)]).double()
    for b_s, kind in ((torch.rand(n, generator=g) + 0.5, L.BSCALE_CHANNEL), (b_t, L.BSCALE_TILE)):
        f = a_s[0, 0].double().view(-1, 1, 1)
        f = f * (b_s.double().view(1, 1, n) if kind == L.BSCALE_CHANNEL else b_s.double().t().repeat_interleave(128, 1).view(kb, 1, n))
        ref = (P * f).sum(0)
        bound = (1.25 * kb + 3) * 2.0 ** -24 * ((P * f).abs().sum(0) + 2 * 2080800 * f.max()) + 2.0 ** -23 * (P * f).abs().sum(0)
        out = K.gemm_block(aq.to(DEV), bq.to(DEV), a_s.to(DEV), b_s.to(DEV), b_kind=kind, flags=L.GEMM_OUT_F32)[0].cpu().double()
        assert ((out - ref).abs() <= bound).all(), float(((out - ref).abs() / bound).max())
    K.check_status(DEV)


@pytest.mark.parametrize("scaling", ["tile128", "row128"])
def test_rotated_tile_quantizer_infinite_and_nan(scaling):
    """A rotated group with a NaN is all NaN: it leaves the maximum alone and quantizes to 0; one with an infinity
    has scale factor 127/inf = 0 and quantizes to 0 with stored scale inf."""
    gran = L.GRAN_TILE128 if scaling == "tile128" else L.GRAN_GROUP128
    g = torch.Generator().manual_seed(3)
    x = torch.randn(1, 256, 384, generator=g).to(torch.bfloat16)
    clean = x.clone()
    x[0, 3, 5], x[0, 9, 140] = float("nan"), float("inf")
    q, s, qt, st = K.quant_tile(x.to(DEV), gran, L.QMODE_TRITON, 128, transposed=True)
    q0, s0, qt0, st0 = K.quant_tile(clean.to(DEV), gran, L.QMODE_TRITON, 128, transposed=True)
    assert (q[0, 3, :128] == 0).all() and (q[0, 9, 128:256] == 0).all()
    assert torch.equal(q[0, 128:], q0[0, 128:]) and torch.equal(qt[0, :, 128:], qt0[0, :, 128:])
    assert (qt[0, 5, :128] == 0).all() and (qt[0, 140, :128] == 0).all()
    if gran == L.GRAN_GROUP128:
        assert torch.isinf(s[0, 9, 1]) and torch.isinf(st[0, 140, 0])
        assert abs(float(s[0, 3, 0]) - 1e-4 / 127) < 1e-9    # no finite value: the floor of the maximum
        keep = [r for r in range(128) if r not in (3, 9)]
        assert torch.equal(q[0, keep], q0[0, keep]) and torch.equal(s[0, keep], s0[0, keep])
    else:
        assert torch.isinf(s[0, 0, 1]) and torch.isinf(st[0, 1, 0]) and torch.equal(s[0, 0, 2], s0[0, 0, 2])


@pytest.mark.parametrize("rows,cols", [(1, 128), (9, 256), (3, 2048), (130, 2176), (6, 4096), (5, 4224), (3, 8320), (2, 16384), (2, 16512)])
@pytest.mark.parametrize("had", [0, 128])
def test_row_quantizer_row_lengths(rows, cols, had):
    """Row lengths at which the number of threads or rows per CTA changes, and row counts that fill no CTA."""
    g = torch.Generator().manual_seed(rows + cols)
    w = torch.randn(rows, cols, generator=g).to(torch.bfloat16)
    w[rows - 1, cols - 1] = -77.0
    q, s = K.quant_row(w.to(DEV), L.QMODE_TRITON, had)
    q_ref, s_ref = R.quant_token(R.hadamard(w, 128) if had else w)
    _same(q, q_ref, "int8"); _same(s, s_ref.view(-1), "scale")
    w[0, 5], w[0, 6] = float("nan"), 3.0     # without a rotation the NaN becomes 0 and leaves the maximum alone
    if not had:
        q, s = K.quant_row(w.to(DEV), L.QMODE_TRITON, had)
        w[0, 5] = 0.0
        q_ref, s_ref = R.quant_token(w)
        _same(q, q_ref, "int8 with a NaN"); _same(s, s_ref.view(-1), "scale with a NaN")


@pytest.mark.parametrize("rows,cols", [(3100, 256), (1600, 512), (801, 1024), (401, 2048), (197, 4096), (99, 8192), (49, 16384),
                                       (5, 128), (70, 256), (3, 16384), (2, 32768)])
def test_whole_row_rotation_both_kernels(rows, cols):
    """Rows of every power of two on both sides of the size from which a CTA takes whole rows of 128 groups, with a
    last CTA that is not full; a NaN or an infinity spoils its own row only."""
    g = torch.Generator().manual_seed(rows)
    x = torch.randn(rows, cols, generator=g).to(torch.bfloat16)
    x[rows - 1, cols - 1], x[1, :] = 60.0, 0
    q, s = K.quant_row(x.to(DEV), L.QMODE_ROWRCP, -1)
    q_ref, s_ref = R.quant_row(R.hadamard(x, cols)[None])
    _same(q, q_ref[0], "int8"); _same(s, s_ref.view(-1), "scale")
    if rows >= 40:
        x[2, 7], x[30, 9] = float("nan"), float("inf")
        q2, s2 = K.quant_row(x.to(DEV), L.QMODE_ROWRCP, -1)
        keep = [r for r in range(rows) if r not in (2, 30)]
        assert torch.equal(q2[keep], q[keep]) and torch.equal(s2[keep], s[keep])
        assert (q2[2] == 0).all() and (q2[30] == 0).all() and torch.isinf(s2[30])


@pytest.mark.parametrize("kb,n,values,decade", [(1, 256, "random", 0), (2, 384, "random", 0), (5, 128, "random", 30), (6, 640, "random", -25),
                                                (3, 256, "lowest", 0), (4, 256, "opposite", 0)])
@pytest.mark.parametrize("b_kind", ["channel", "tile", "group", "column"])
def test_row_and_column_factor_epilogues(kb, n, values, decade, b_kind):
    """Per-(row, K block) A scales with every kind of B scale, and per-tile A scales with per-(column, K block) ones
    ("column", as products and, for moderate sizes, as divisors).  The shifted partial product is brought back exactly, so
    each K block costs three fp32 roundings (product of the scales, of the factors, the sum) and the end three more."""
    g = torch.Generator().manual_seed(200 + kb)
    M, Kd = 256, 128 * kb
    aq, bq = _randq(g, 1, M, Kd), _randq(g, n, Kd)
    if values == "lowest":
        aq.fill_(-128), bq.fill_(-128)
    elif values == "opposite":
        aq.fill_(-128), bq.fill_(127)
    P = torch.stack([R.int_mm(aq[0, :, k * 128:(k + 1) * 128], bq[:, k * 128:(k + 1) * 128]) for k in range(kb)]).double()
    if b_kind == "column":
        a_s = (torch.rand(1, M // 128, kb, generator=g) + 0.5) * 10.0 ** decade
        fa = a_s[0].double().t().repeat_interleave(128, 1)[:, :, None]
    else:
        a_s = (torch.rand(1, M, kb, generator=g) + 0.5) * 10.0 ** decade
        fa = a_s[0].double().t()[:, :, None]
    if b_kind == "channel":
        b_s, kind = torch.rand(n, generator=g) + 0.5, L.BSCALE_CHANNEL
        fb = b_s.double().view(1, 1, n)
    elif b_kind == "tile":
        b_s, kind = torch.rand(n // 128, kb, generator=g) + 0.5, L.BSCALE_TILE
        fb = b_s.double().t().repeat_interleave(128, 1)[:, None, :]
    else:
        b_s, kind = torch.rand(n, kb, generator=g) + 0.5, L.BSCALE_GROUP
        fb = b_s.double().t()[:, None, :]
    a_kind = L.ASCALE_TILE if b_kind == "column" else L.ASCALE_GROUP
    modes = [(0, fa * fb)] + ([(L.GEMM_DIVIDE, 1.0 / (fa * fb))] if b_kind == "column" and decade == 0 else [])
    for flag, f in modes:
        ref, mag = (P * f).sum(0), (P * f).abs().sum(0)
        out = K.gemm_block(aq.to(DEV), bq.to(DEV), a_s.to(DEV), b_s.to(DEV), a_kind, kind, flags=L.GEMM_OUT_F32 | flag)[0].cpu().double()
        assert ((out - ref).abs() <= (3 * kb + 3) * 2.0 ** -24 * mag).all(), float(((out - ref).abs() / mag.clamp_min(1e-300)).max())
    K.check_status(DEV)


@pytest.mark.parametrize("kb,n,share", [(1, 256, 1.0), (3, 128, 1.0), (8, 384, 1.0), (64, 256, 1.0), (258, 128, 1.0), (64, 384, 0.5),
                                        (256, 256, 0.25)])
@pytest.mark.parametrize("kind", ["channel", "tile"])
def test_fast_block_epilogue_repeated_factors(kb, n, share, kind):
    """A factor that repeats (an all-zero 128-row block, whose scales sit on the quantizers' floor; clipped data) must not
    let the roundings of the shift add up along K.  Where all factors are equal nothing is rounded but the sum itself:
    zero rows give exactly zero and small constant partial products their exact sum, times c and the column scale (three
    roundings).  Where `share` of them are, the other K blocks round like distinct ones: three roundings in four K blocks, each
    within a quarter of the factor and uniform (standard deviation f / 7), so five standard deviations of their sum
    for the rows whose products are zero."""
    g = torch.Generator().manual_seed(300 + kb)
    M, Kd = 128, 128 * kb
    aq, bq = torch.zeros(1, M, Kd, dtype=torch.int8), torch.zeros(n, Kd, dtype=torch.int8)
    aq[0, 40:, ::128] = 1                    # rows 40-: partial product 1 or -3 in every K block
    bq[:, ::128] = 1
    bq[1::2, ::128] = -3
    a_s = torch.rand(1, 1, kb, generator=g) + 0.5
    same = int(share * kb)
    a_s[0, 0, :same] = a_s[0, 0, 0]
    if kind == "channel":
        b_s, b_kind = torch.rand(n, generator=g) + 0.5, L.BSCALE_CHANNEL
        fb = b_s.double().view(1, n)
    else:
        b_s, b_kind = (torch.rand(n // 128, 1, generator=g) + 0.5).expand(-1, kb).contiguous(), L.BSCALE_TILE
        fb = b_s[:, 0].double().repeat_interleave(128).view(1, n)
    P = torch.zeros(M, n, dtype=torch.double)
    P[40:] = bq[:, 0].double()
    ref = P * a_s.double().sum() * fb
    out = K.gemm_block(aq.to(DEV), bq.to(DEV), a_s.to(DEV), b_s.to(DEV), b_kind=b_kind, flags=L.GEMM_OUT_F32)[0].cpu().double()
    err = (out - ref).abs()
    if share == 1.0:
        assert (out[:40] == 0).all(), float(out[:40].abs().max())
        assert (err <= 4 * 2.0 ** -24 * ref.abs()).all()
    else:
        unit = float(a_s.max()) * fb
        assert (err <= 5 / 7 * (0.75 * (kb - same)) ** 0.5 * unit).all(), float((err / unit).max())
    K.check_status(DEV)


def test_fast_block_epilogue_zero_rows_and_a_dominant_block():
    """The rounding of the shift is an absolute error, a fraction of the tile's largest factor: rows of zeros beside
    other rows come out within it (five standard deviations, see above), and a row that is zero in the one K block whose
    scale is 1e4 times the others is off by no more than the roundings around that block (four times a quarter of its
    factor)."""
    g = torch.Generator().manual_seed(400)
    kb, n = 64, 256
    aq, bq = _randq(g, 1, 256, 128 * kb), _randq(g, n, 128 * kb)
    aq[0, 5], aq[0, 77] = 0, 0
    a_s, b_s = torch.rand(1, 2, kb, generator=g) + 0.5, torch.rand(n, generator=g) + 0.5
    a_s[0, 1, 30] = 1e4
    aq[0, 200:, 30 * 128:31 * 128] = 0
    out = K.gemm_block(aq.to(DEV), bq.to(DEV), a_s.to(DEV), b_s.to(DEV), flags=L.GEMM_OUT_F32)[0].cpu().double()
    unit = b_s.double().view(1, n)
    bound = 5 / 7 * (0.75 * kb) ** 0.5 * float(a_s[0, 0].max())
    assert (out[[5, 77]].abs() <= bound * unit).all(), float((out[[5, 77]].abs() / unit).max())
    P = torch.stack([R.int_mm(aq[0, 128:, k * 128:(k + 1) * 128], bq[:, k * 128:(k + 1) * 128]) for k in range(kb)]).double()
    ref = (P * a_s[0, 1].double().view(-1, 1, 1)).sum(0) * unit
    err = (out[128:] - ref).abs() / unit
    assert (err[72:] <= 1e4 + bound).all(), float(err[72:].max())
    K.check_status(DEV)


@pytest.mark.parametrize("kb", [1, 3, 4])
@pytest.mark.parametrize("kind", ["row_channel", "row_tile", "outer", "column", "column_div", "tile_div", "outer_exact", "column_exact"])
def test_row_and_column_factors_over_many_tiles_of_one_cta(kind, kb):
    """Two CTAs for all tiles, so that each runs many in a row, with odd and even numbers of K blocks: the column factors
    are published through two buffers that alternate over the K blocks of all tiles.  Bound as in
    test_row_and_column_factor_epilogues; the reference's operation order is met bit for bit."""
    g = torch.Generator().manual_seed(500 + kb)
    M, n, Kd = 512, 1152, 128 * kb
    aq, bq = _randq(g, 1, M, Kd), _randq(g, n, Kd)
    rnd = lambda *shape: torch.rand(*shape, generator=g) + 0.5
    a_tile, a_row = rnd(1, M // 128, kb), rnd(1, M, kb)
    flags, exact = (L.GEMM_DIVIDE if "div" in kind else 0), "exact" in kind
    a_s, a_kind = (a_row, L.ASCALE_GROUP) if kind.startswith(("row", "outer")) else (a_tile, L.ASCALE_TILE)
    if kind == "row_channel":
        b_s, b_kind = rnd(n), L.BSCALE_CHANNEL
        fb = b_s.view(1, 1, n)
    elif kind in ("row_tile", "tile_div"):
        b_s, b_kind = rnd(n // 128, kb), L.BSCALE_TILE
        fb = b_s.t().repeat_interleave(128, 1)[:, None, :]
    else:
        b_s, b_kind = rnd(n, kb), L.BSCALE_GROUP
        fb = b_s.t()[:, None, :]
    fa = (a_s[0].t() if a_kind == L.ASCALE_GROUP else a_s[0].t().repeat_interleave(128, 1))[:, :, None]
    P = torch.stack([R.int_mm(aq[0, :, k * 128:(k + 1) * 128], bq[:, k * 128:(k + 1) * 128]) for k in range(kb)])
    with K.cta_limit(2):
        out = K.gemm_block(aq.to(DEV), bq.to(DEV), a_s.to(DEV), b_s.to(DEV), a_kind, b_kind,
                           flags=L.GEMM_OUT_F32 | flags | (L.GEMM_EXACT_ORDER if exact else 0))[0].cpu()
    if exact:
        acc = torch.zeros(M, n)
        for k in range(kb):
            acc = acc + (P[k].float() * fa[k]) * fb[k]
        assert torch.equal(out, acc)
    else:
        f = 1.0 / (fa.double() * fb.double()) if flags else fa.double() * fb.double()
        mag = (P.double() * f).abs().sum(0)
        err = (out.double() - (P.double() * f).sum(0)).abs()
        assert (err <= (3 * kb + 3) * 2.0 ** -24 * mag).all(), float((err / mag.clamp_min(1e-300)).max())
    K.check_status(DEV)
