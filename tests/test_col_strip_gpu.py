"""Per-column scales in one pass (columns of up to 4096 elements) and in two: the bytes and scales of the row quantizer on the
transposed matrix."""
import pytest
import torch

pytestmark = pytest.mark.gpu

if torch.cuda.is_available():
    from triton_int8_b200 import kernels as K

DEV = "cuda"


@pytest.mark.parametrize("qmode", [0, 1, 3])
@pytest.mark.parametrize("rows", [128, 256, 384, 512, 640, 896, 1024, 1152, 2176, 3968, 4096, 4224])   # 1 to 33 blocks of 128
@pytest.mark.parametrize("cols", [128, 1152])
def test_columns_equal_rows_of_the_transpose(rows, cols, qmode):
    g = torch.Generator(device=DEV).manual_seed(rows + cols)
    x = torch.randn(rows, cols, device=DEV, generator=g).to(torch.bfloat16)
    x[:, 3] = 0
    x[rows - 1, 64] = -50.0
    x[0, 65] = 127.0
    x[1:, 65] = 0.5
    x[5, 70] = float("inf")
    x[7, 71] = float("nan")
    q, s = K.quant_col_t(x, qmode)
    q_ref, s_ref = K.quant_row(x.t().contiguous(), qmode)
    assert torch.equal(q, q_ref) and torch.equal(s, s_ref)
