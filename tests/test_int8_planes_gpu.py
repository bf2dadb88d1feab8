"""The int8 tensor-core projection's own quantizer: rows of every number of words a thread keeps, and rows it reads twice."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("k", [64, 4096, 4112, 8192, 8208, 16384, 16400, 32768, 32784])
@pytest.mark.parametrize("offset", [0, 2])
def test_whole_activations_give_exact_sums(k, dtype, offset):
    """Whole activations of up to 8 are exact in the planes; k * 8 * 127 < 2^25.1 keeps every result a whole number that the int32 sums hold, and the last
    rounding to f32 is that of the f64 reference."""
    from tlaloc_b200 import ops

    rows = 17
    g = torch.Generator(device=DEV).manual_seed(k)
    x = torch.randint(-8, 9, (rows * k + offset,), generator=g, device=DEV).to(dtype)[offset:].view(rows, k)
    x[3] = 0
    codes = torch.randint(-127, 128, (k, 256), dtype=torch.int8, generator=g, device=DEV)
    scales = torch.full((256,), 0.5, device=DEV)
    want = (x.double() @ codes.double() * 0.5).float()
    for const in (False, True):
        assert torch.equal(ops.int8_gemm(x, codes, scales, i8_mma=True, weights_const=const), want)
    x[5, k // 2] = float("nan")
    got = ops.int8_gemm(x, codes, scales, i8_mma=True)
    assert bool(torch.isnan(got[5]).all()) and torch.equal(got[:5], want[:5]) and torch.equal(got[6:], want[6:])
