"""Column sums (the bias gradient) against float64."""
import pytest
import torch

pytestmark = pytest.mark.gpu

if torch.cuda.is_available():
    from triton_int8_b200 import kernels as K

DEV = "cuda"


@pytest.mark.parametrize("rows,cols", [(128, 128), (512, 1024), (640, 128), (1024, 384), (4224, 256), (8192, 128), (33024, 128),
                                       (65536, 256), (1152, 19072)])
def test_col_sum(rows, cols):
    g = torch.Generator(device=DEV).manual_seed(rows)
    x = torch.randn(rows, cols, device=DEV, generator=g).to(torch.bfloat16)
    x[:, 5] = 1.0
    x[rows - 1, 5] = -3.0
    x[3, 77] = float("inf")
    x[4, 78] = float("nan")
    got, ref = K.col_sum(x), x.double().sum(0)
    for _ in range(3):   # the order depends on the shape only
        torch.cuda._sleep(10_000)
        assert torch.equal(got.view(torch.int16), K.col_sum(x).view(torch.int16))
    fin = ref.isfinite()
    assert torch.equal(got.double()[~fin].isnan(), ref[~fin].isnan()) and got[77] == float("inf")
    # one rounding to bf16, behind fp32 sums of at most 128 values and their 3 levels
    bound = ref.abs() * 2.0 ** -8 + x.double().abs().nan_to_num(0, 0).sum(0) * 2.0 ** -24 * 131
    assert ((got.double() - ref).abs() <= bound)[fin].all()
    assert got[5] == torch.tensor(rows - 4.0).to(torch.bfloat16)
