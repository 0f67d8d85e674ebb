"""Small operands of a product are quantized in one launch: the product equals that of the separate quantizers bit for bit."""
import pytest
import torch

pytestmark = pytest.mark.gpu

if torch.cuda.is_available():
    from triton_int8_b200 import _lib as L
    from triton_int8_b200 import kernels as K

DEV = "cuda"


@pytest.mark.parametrize("B,M,N,Kd", [(1, 128, 128, 128), (3, 256, 640, 384), (1, 640, 128, 2176), (1, 256, 384, 4096), (1, 2048, 1024, 1024),
                                      (2, 128, 2048, 4224)])   # the last: rows too long for it
@pytest.mark.parametrize("a_gran,b_gran,qmode", [("tile", "row", 0), ("group", "row", 1), ("row", "row", 3), ("tile", "tile", 0),
                                                 ("tile", "tile", 2), ("tile", "group", 2), ("tile", "row", 1)])
def test_pair_equals_separate_quantizers(B, M, N, Kd, a_gran, b_gran, qmode):
    g = torch.Generator(device=DEV).manual_seed(M + N)
    G = {"tile": L.GRAN_TILE128, "group": L.GRAN_GROUP128, "row": L.GRAN_ROW}
    batched = b_gran != "row" and B > 1
    a = torch.randn(B, M, Kd, device=DEV, generator=g).to(torch.bfloat16)
    b = torch.randn(*((B,) if batched else ()), N, Kd, device=DEV, generator=g).to(torch.bfloat16)
    flags = L.GEMM_DIVIDE if qmode == 2 else 0

    def quant(t, gran):
        if gran == "row":
            return K.quant_row(t, qmode)
        t3 = t if t.dim() == 3 else t[None]
        q, s = K.quant_tile(t3, G[gran], qmode)[:2]
        return (q, s) if t.dim() == 3 else (q[0], s[0])

    (aq, a_s), (bq, b_s) = quant(a, a_gran), quant(b, b_gran)
    if a_gran == "row":
        ref = K.gemm_rowcol(aq, bq, a_s, b_s)
    else:
        bk = {"row": L.BSCALE_CHANNEL, "tile": L.BSCALE_TILE, "group": L.BSCALE_GROUP}[b_gran]
        ref = K.gemm_block(aq, bq, a_s, b_s, L.ASCALE_TILE if a_gran == "tile" else L.ASCALE_GROUP, bk, flags=flags)
    for want in ((False, True) if B == 1 and b_gran == "row" else (False,)):
        out, (qt, st) = K.quant_gemm(a, b, G[a_gran], G[b_gran], qmode, 0, None, 1.0, flags, want)
        assert torch.equal(out, ref)
        if want:
            if a_gran == "row":
                qt_ref, st_ref = (t[None] for t in K.quant_col_t(a[0], qmode))
            else:
                qt_ref, st_ref = K.quant_tile(a, G[a_gran], qmode, natural=False, transposed=True)[2:]
            assert torch.equal(qt, qt_ref) and torch.equal(st, st_ref)
