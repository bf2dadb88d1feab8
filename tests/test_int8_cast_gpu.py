"""f32 rows of the int8 projection: their cast to bf16, aligned to 16 bytes or not (needs a B200)."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("m,k", [(1, 16), (3, 1032), (17, 256), (40, 2048)])
@pytest.mark.parametrize("offset", [0, 1])
def test_cast_rows_equal_bf16_rows(m, k, offset):
    from tlaloc_b200 import ops

    x = torch.randn((m * k + offset,), device=DEV)[offset:].view(m, k)
    codes, scales = torch.randint(-127, 128, (k, 256), dtype=torch.int8, device=DEV), torch.rand((256,), device=DEV)
    assert torch.equal(ops.int8_gemm(x, codes, scales), ops.int8_gemm(x.bfloat16(), codes, scales))
