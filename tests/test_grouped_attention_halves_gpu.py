"""Attention over grouped heads in grids of more CTAs than SMs, where large groups' keys and values travel on their own (three halves, or two of each) and others as one, against f64."""
import pytest
import torch

from tlaloc_b200 import ops

pytestmark = pytest.mark.gpu
DEV, BF16 = "cuda:0", torch.bfloat16


@pytest.fixture(autouse=True)
def no_wait_runs_out():
    yield
    from tlaloc_b200 import _native

    torch.cuda.synchronize()
    assert _native.lib().tlaloc_b200_device_status() == 0


# heads of queries (with maps), value heads, maps, dim, vdim.  Keys and values on their own: 8 + 8 KB, 8 + 8 of which 240 channels are used, 4 + 8 (two maps of 64, one of 128), 8 + 4,
# 4 + 6, 2 + 8; whole groups in as large a grid: 4 + 4 (small enough as they are), 8 + 6 (halves of two do not leave room for a second CTA)
@pytest.mark.parametrize("heads,groups,maps,dim,vdim", [(16, 4, 2, 128, 256), (8, 4, 2, 128, 240), (16, 4, 2, 64, 256), (8, 4, 1, 128, 256), (16, 4, 2, 112, 128), (8, 4, 2, 48, 192),
                                                        (16, 4, 1, 64, 256), (16, 4, 2, 64, 128), (16, 4, 2, 128, 192)])
@pytest.mark.parametrize("window,keep,slices", [(0, 0, 1), (70, 0, 1), (70, 9, 1), (33, 40, 2), (0, 0, 3)])
def test_more_ctas_than_sms(heads, groups, maps, dim, vdim, window, keep, slices):
    lens = [1, 15, 16, 17, 31, 32, 33, 47, 48, 49, 63, 64, 65, 80, 95, 96, 97, 111, 112, 127, 128, 129, 143, 144, 145, 159, 160, 200, 255, 256, 257, 300, 319, 320, 321, 350, 383, 384,
            385, 400]
    g = torch.Generator(device=DEV).manual_seed(dim + vdim)
    T, M, v_first = len(lens), 7, groups * maps * dim
    pool = torch.randn((T * M + 1, 64, v_first + groups * vdim), generator=g, device=DEV).to(BF16)
    tables = (1 + torch.randperm(T * M, generator=g, device=DEV)).view(T, M).int()
    for t, n in enumerate(lens):  # what lies behind a row's end may be anything
        if n < M * 64:
            pool[tables[t, n // 64].long(), n % 64:] = float("nan")
    q, scale = torch.randn((T, heads, dim), generator=g, device=DEV).to(BF16), 1.5 * dim ** -0.5
    records = torch.full((slices, T, heads, vdim + 2), float("nan"), device=DEV)
    ops.grouped_attention(q, pool, tables, torch.tensor(lens, dtype=torch.int32, device=DEV), records, v_heads=groups, maps=maps, vdim=vdim, v_first=v_first, scale=scale,
                          slices=slices, window=window, keep_first=keep)
    r = records.double()
    factor = torch.where(torch.isinf(r[..., 0]), 0.0, torch.exp2(r[..., 0] - r[..., 0].max(0).values))
    acc = torch.where(factor[..., None] > 0, r[..., 2:] * factor[..., None], 0.0).sum(0)
    got = acc / (torch.where(factor > 0, r[..., 1], 0.0) * factor).sum(0)[..., None]
    for t, n in enumerate(lens):
        p = torch.arange(n, device=DEV)
        if window:
            p = p[(p >= n - window) | (p < keep)]
        rows = pool[tables[t, p // 64].long(), p % 64].double()
        for h in range(heads):
            v = h // (heads // groups)
            k = v * maps + h % maps
            weights = torch.softmax(rows[:, k * dim:(k + 1) * dim] @ q[t, h].double() * scale, 0)
            want = weights @ rows[:, v_first + v * vdim:v_first + (v + 1) * vdim]
            # f32 scores and sums, weights as two bf16 parts (2^-17), exponentials within 2^-21: values of up to 5
            assert float((got[t, h] - want).abs().max()) <= 1e-4, (t, h)
