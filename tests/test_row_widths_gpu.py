"""The row operations at the widths where their kernels change over (words a thread keeps, element by element), against f64."""
import pytest
import torch

from tlaloc_b200 import ops

pytestmark = pytest.mark.gpu
DEV, F32, BF16, EPS = "cuda:0", torch.float32, torch.bfloat16, 1e-5
# f32: a norm's sum of n squares in another order moves it by n * 2^-24 at most (2^-11 for the widest), random signs far less; bf16 results: half a unit, 2^-9
TOL = {F32: 2e-5, BF16: 2.0 ** -8}


def randn(*shape, seed=0):
    return torch.randn(shape, generator=torch.Generator().manual_seed(seed)).to(DEV)


def rms(x):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + EPS)


def close(got, want, dtype):
    assert bool(((got.double() - want).abs() <= TOL[dtype] * (1 + want.abs())).all()), float((got.double() - want).abs().max())


@pytest.mark.parametrize("dtype", [F32, BF16])
@pytest.mark.parametrize("n", [4, 1024, 2048, 2052, 3072, 3076, 4096, 4100, 8192, 8196, 2050])
def test_norms(n, dtype):
    x, y, g, h = randn(3, n, seed=1), randn(3, n, seed=2), randn(n, seed=3), randn(n, seed=4)
    a, b = torch.empty((3, n), device=DEV, dtype=dtype), torch.empty((3, n), device=DEV, dtype=dtype)
    ops.rmsnorm_pair(x, g, a, EPS, h, b)
    close(a, rms(x.double()) * g.double(), dtype)
    close(b, rms(x.double()) * h.double(), dtype)
    want = x.double() + rms(y.double()) * g.double()
    ops.residual_norm(y, x, g, EPS, gain_next=h, out=a)
    close(x, want, F32)
    close(a, rms(want) * h.double(), dtype)


@pytest.mark.parametrize("dtype", [F32, BF16])
@pytest.mark.parametrize("vdim", [2, 62, 64, 66, 128, 130, 256, 258, 512, 514, 33])
def test_heads(vdim, dtype):
    rows, heads = 3, 2
    o, gate, maps = randn(rows, heads, vdim, seed=1), randn(rows, heads * vdim, seed=2), randn(rows, heads, 2, vdim, seed=3)
    out = torch.empty((rows, heads * vdim), device=DEV, dtype=dtype)
    ops.head_norm_gate(o, gate, out, EPS)
    z = gate.double()
    close(out, rms(o.double()).reshape(rows, -1) * z / (1 + torch.exp(-z)), dtype)
    ops.map_difference(maps, out, rows=rows, heads=heads, vdim=vdim, in_ld=vdim, lam=0.3, keep=0.7, eps=EPS)
    close(out, (rms(maps[:, :, 0].double() - 0.3 * maps[:, :, 1].double()) * 0.7).reshape(rows, -1), dtype)


@pytest.mark.parametrize("dtype", [F32, BF16])
@pytest.mark.parametrize("q_rank,kv_rank,rot,dims", [(2048, 1024, 64, 64), (2052, 64, 8, 4), (64, 1028, 8, 8), (0, 8, 4, 2), (1024, 512, 1024, 6), (6, 10, 2, 2), (1028, 4, 12, 10)])
def test_latent_rows(q_rank, kv_rank, rot, dims, dtype):
    T, row = 5, kv_rank + rot
    low, qg, kg = randn(T, q_rank + row, seed=1), randn(max(q_rank, 1), seed=2), randn(kv_rank, seed=3)
    cos, sin = randn(9, dims // 2, seed=4), randn(9, dims // 2, seed=5)
    positions, slots = torch.tensor([0, 3, 8, 1, 2], dtype=torch.int32, device=DEV), torch.tensor([7, -1, 0, 64, 3], dtype=torch.int32, device=DEV)
    pool, cq = torch.full((1, 64, row), 7.0, device=DEV, dtype=dtype), torch.empty((T, q_rank), device=DEV, dtype=dtype)
    ops.latent_kv_write(low, qg if q_rank else None, kg, EPS, positions, cos, sin, slots, cq if q_rank else None, pool, q_rank=q_rank, kv_rank=kv_rank, rot_dim=rot,
                        rot_dims=dims)
    d = low.double()
    if q_rank:
        close(cq, rms(d[:, :q_rank]) * qg.double(), dtype)
    turned = d[:, q_rank + kv_rank:].clone()
    c, s = cos.double()[positions.long()], sin.double()[positions.long()]
    u, v = turned[:, 0:dims:2].clone(), turned[:, 1:dims:2].clone()
    turned[:, 0:dims:2], turned[:, 1:dims:2] = u * c - v * s, v * c + u * s
    rows = torch.cat([rms(d[:, q_rank:q_rank + kv_rank]) * kg.double(), turned], 1)
    for t in (0, 2, 4):
        close(pool[0, slots[t]], rows[t], dtype)
    untouched = [i for i in range(64) if i not in (7, 0, 3)]
    assert bool((pool[0, untouched] == 7).all())


@pytest.mark.parametrize("dtype", [F32, BF16])
@pytest.mark.parametrize("width,dims,before", [(64, 64, 0), (64, 64, 128), (12, 8, 4), (12, 6, 4), (12, 4, 2), (7, 4, 1), (10, 10, 2)])
def test_interleaved_rotation(width, dims, before, dtype):
    T, heads = 5, 3
    x = randn(T, heads, before + width, seed=1).to(dtype)
    cos, sin = randn(9, dims // 2, seed=4), randn(9, dims // 2, seed=5)
    positions = torch.tensor([0, 3, 8, 1, 2], dtype=torch.int32, device=DEV)
    want = x.double()
    c, s = cos.double()[positions.long()][:, None], sin.double()[positions.long()][:, None]
    u, v = want[:, :, before:before + dims:2].clone(), want[:, :, before + 1:before + dims:2].clone()
    want[:, :, before:before + dims:2], want[:, :, before + 1:before + dims:2] = u * c - v * s, v * c + u * s
    out = torch.zeros_like(x)
    ops.rope_interleaved(x[:, :, before:], out[:, :, before:], positions, cos, sin, rot_dims=dims)
    close(out[:, :, before:], want[:, :, before:], dtype)
    ops.rope_interleaved(x[:, :, before:], x[:, :, before:], positions, cos, sin, rot_dims=dims)  # in place
    close(x, want, dtype)
