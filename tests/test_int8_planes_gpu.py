"""The int8 tensor-core projection's own quantizer: rows of every number of words a thread keeps, and rows it reads twice."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("dtype,offset", [(torch.float32, 0), (torch.float32, 2), (torch.bfloat16, 0)])
@pytest.mark.parametrize("k", [64, 4096, 4112, 8192, 8208, 16384, 16400, 32768, 32784, 49168])
def test_whole_activations_give_exact_sums(k, dtype, offset):
    """Whole activations of up to 8 are exact in the planes; k * 8 * 127 < 2^25.6 keeps every result a whole number that the int32 sums hold, and the last
    rounding to f32 is that of the f64 reference.  f32 rows may start anywhere; bf16 rows off a 16-byte boundary never reach the quantizer."""
    from tlaloc_b200 import _native, ops

    rows = 17
    g = torch.Generator(device=DEV).manual_seed(k)
    x = torch.randint(-8, 9, (rows * k + offset,), generator=g, device=DEV).to(dtype)[offset:].view(rows, k)
    x[3] = 0
    codes = torch.randint(-127, 128, (k, 256), dtype=torch.int8, generator=g, device=DEV)
    scales = torch.full((256,), 0.5, device=DEV)
    want = (x.double() @ codes.double() * 0.5).float()
    for const in (False, True):
        before = _native.lib().tlaloc_b200_launch_count()
        assert torch.equal(ops.int8_gemm(x, codes, scales, i8_mma=True, weights_const=const), want)
        assert _native.lib().tlaloc_b200_launch_count() - before == 2  # the quantizer and the projection
    x[5, k // 2] = float("nan")
    got = ops.int8_gemm(x, codes, scales, i8_mma=True)
    assert bool(torch.isnan(got[5]).all()) and torch.equal(got[:5], want[:5]) and torch.equal(got[6:], want[6:])


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("rows", [17, 40, 128])
def test_codes_written_right_in_front_are_the_ones_read(rows, dtype):
    """Without weights_const the projection asks for its codes only behind its quantizer's wait: what the kernel before both has written.  That kernel
    (gather_rows) lets its successors start as early as any of the library's."""
    from tlaloc_b200 import ops

    k, n, count = 4096, 4096, 12
    g = torch.Generator(device=DEV).manual_seed(rows)
    x = torch.randint(-8, 9, (rows, k), generator=g, device=DEV).to(dtype)
    sources = [torch.randint(-127, 128, (k, n), dtype=torch.int8, device=DEV, generator=g) for _ in range(2)]
    factors = [torch.full((1, n), f, device=DEV) for f in (0.5, 0.25)]
    want = [(x.double() @ c.double() * f[0]).float() for c, f in zip(sources, factors)]
    codes, scales = torch.zeros((k, n), dtype=torch.int8, device=DEV), torch.zeros((1, n), device=DEV)
    order = torch.arange(k, dtype=torch.int32, device=DEV)
    outs = [torch.empty((rows, n), device=DEV) for _ in range(count)]
    scratch = torch.empty(ops.int8_gemm_scratch_bytes(rows, k, n) // 4, device=DEV)
    for i, out in enumerate(outs):
        ops.gather_rows(factors[i % 2], order[:1], scales)
        ops.gather_rows(sources[i % 2], order, codes)
        ops.int8_gemm(x, codes, scales[0], i8_mma=True, out=out, scratch=scratch)
    for i, out in enumerate(outs):
        assert torch.equal(out, want[i % 2]), i
