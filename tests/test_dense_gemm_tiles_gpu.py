"""bf16 projections of more than 128 rows: every height of a tile, whole and cut, against f64 (needs a B200)."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


# heights by rows and columns (148 CTAs): 256; 224; 192; 160, cut; 128, whole and cut
@pytest.mark.parametrize("m,n,k", [(256, 18944, 128), (2007, 4096, 512), (192, 18944, 192), (2047, 2560, 648), (150, 2560, 256), (165, 2048, 4096), (300, 1100, 2056)])
@pytest.mark.parametrize("act", [0, 1, 3])
def test_heights(m, n, k, act):
    from tlaloc_b200 import _native, ops

    n = n // 32 * 32
    g = torch.Generator(device=DEV)
    g.manual_seed(m + n + k)
    x, w = (torch.randn(s, device=DEV, generator=g).bfloat16() for s in ((m, k), (n, k)))
    b, r = torch.randn((n,), device=DEV, generator=g), torch.randn((m, n), device=DEV, generator=g)
    z = x.double() @ w.double().T
    # the tensor core's accumulator is cut, not rounded, after each 16 products: 2^-23 of it at most, k / 16 times; twice that through the square
    exact = (k / 16 + 8) * 2.0 ** -22
    for f32 in (True, False):
        y = torch.full((m + 1, n // 2 if act == 3 else n), 7.0, device=DEV, dtype=torch.float32 if f32 else torch.bfloat16)
        if act == 3:
            ops.dense_gemm(ops.dense(x, w, y[:m], act=3), weights_const=True)
            u = z.view(m, -1, 2, 16)
            want = (torch.nn.functional.gelu(u[:, :, 0], approximate="tanh") * u[:, :, 1]).reshape(m, -1)
        else:
            ops.dense_gemm(ops.dense(x, w, y[:m], bias=b, act=act, residual=r if f32 else None))
            want = z + b.double()
            want = (want.clamp_min(0) ** 2 if act else want) + (r.double() if f32 else 0)
        assert float((y[:m].double() - want).norm() / want.norm()) < (exact if f32 else exact + 2.0 ** -8)
        assert bool((y[m] == 7).all())
    assert _native.lib().tlaloc_b200_device_status() == 0
