"""The f32 projection on the tensor cores against f64: edges of its tiles, chunks and slices, its distance from f64 beside the plain kernel's, operands
that its parts cannot hold (needs a B200)."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.fixture(autouse=True)
def no_wait_runs_out():
    yield
    from tlaloc_b200 import _native

    torch.cuda.synchronize()
    assert _native.lib().tlaloc_b200_device_status() == 0


def ops():
    from tlaloc_b200 import ops as o

    return o


def rand(*shape, seed=0):
    g = torch.Generator(device=DEV)
    g.manual_seed(seed + sum(shape))
    return torch.randn(shape, device=DEV, generator=g)


def in_order(x, w):
    """The product by the plain kernel: f32 FMAs in k order."""
    y = torch.empty((x.shape[0], w.shape[0]), device=DEV)
    before = ops().set_order_faithful(True)
    try:
        ops().dense_gemm(ops().dense(x, w, y))
    finally:
        ops().set_order_faithful(before)
    return y


def bound(x, w):
    """Every addition loses at most 2^-23 of what it holds: k / 32 rounded ones of chunks, and 16 inside a chunk, whose size is at most the
    sum of magnitudes."""
    k = x.shape[-1]
    return (k / 32 + 16) * 2.0 ** -23 * (x.double().abs() @ w.double().abs().transpose(-1, -2)) + 2.0 ** -148


# rows: one tile of 16 .. 208, then equal parts; n, k: remainders of 128 columns and of chunks of 32 and 64, two chunks and fewer
@pytest.mark.parametrize("m", [1, 15, 17, 32, 33, 64, 65, 127, 129, 193, 208, 209, 500])
@pytest.mark.parametrize("n,k", [(1, 4), (128, 64), (200, 100), (1344, 192), (130, 1028)])
def test_tiles_and_chunks(m, n, k):
    x, w, b, r = rand(m, k), rand(n, k, seed=1), rand(n, seed=2), rand(m, n, seed=3)
    y = torch.full((m + 1, n), 7.0, device=DEV)
    ops().dense_gemm(ops().dense(x, w, y[:m]))
    want = x.double() @ w.double().T
    assert bool(((y[:m].double() - want).abs() <= bound(x, w)).all()) and bool((y[m] == 7).all())
    want = (want + b.double()).clamp_min(0) ** 2 + r.double()
    tol = bound(x, w) * (2 * want.abs().sqrt() + 1) + 2.0 ** -20 * (want.abs() + 1)
    ops().dense_gemm(ops().dense(x, w, r, bias=b, act=1, residual=r), weights_const=True)
    assert bool(((r.double() - want).abs() <= tol).all())


@pytest.mark.parametrize("m", [3, 40, 100, 203])
@pytest.mark.parametrize("k", [2048, 10304])
def test_no_further_from_f64_than_plain_sums(m, k):
    x, w = rand(m, k), rand(256, k, seed=1)
    want = x.double() @ w.double().T
    y = torch.empty((m, 256), device=DEV)
    ops().dense_gemm(ops().dense(x, w, y))
    assert float((y - want).norm()) <= float((in_order(x, w) - want).norm())


@pytest.mark.parametrize("m", [4, 200])
@pytest.mark.parametrize("k", [4, 16, 28, 32, 36, 64, 128, 512])
@pytest.mark.parametrize("signs", ["both", "one", "near one"])
def test_no_further_from_f64_at_few_k(m, k, signs):
    x, w = rand(m, k), rand(512, k, seed=1)
    if signs != "both":
        x, w = (torch.sigmoid(a) if signs == "one" else 1 + 1e-3 * torch.sigmoid(a) for a in (x, w))
    y, want = torch.empty((m, 512), device=DEV), x.double() @ w.double().T
    ops().dense_gemm(ops().dense(x, w, y))
    assert float((y - want).norm()) <= float((in_order(x, w) - want).norm())


# k 2048: slices of k; n 19000: none
@pytest.mark.parametrize("m,n,k", [(9, 200, 2048), (200, 200, 2048), (9, 19000, 96), (200, 19000, 96)])
@pytest.mark.parametrize("large", [1.0, 1e10, 1e20, 1e30, 1e38])
def test_small_operands(m, n, k, large):
    """Rows from 1e-41 (subnormal) to 1e-33, alone and beside a row of one, against weights of `large`: each row as near to f64 as plain FMAs are, and not
    zero where those are not."""
    x, w = rand(m, k), rand(n, k, seed=1).clamp(-3, 3) * large
    x *= torch.tensor([10.0 ** (r - 41) if r < 9 else 1e-37 for r in range(m)], device=DEV, dtype=torch.float64)[:, None].float()
    x[4, ::2], x[-1] = 0.0, 0.0
    y = torch.empty((m, n), device=DEV)
    ops().dense_gemm(ops().dense(x, w, y))
    want, plain = x.double() @ w.double().T, in_order(x, w)
    assert bool(((y - want).norm(dim=1) <= (plain - want).norm(dim=1) + 2.0 ** -149 * n ** 0.5).all())
    assert bool((y[-1] == 0).all()) and torch.equal(y == 0, want.float() == 0)


@pytest.mark.parametrize("m,n,k", [(5, 140, 96), (150, 140, 96), (40, 200, 1024)])
@pytest.mark.parametrize("size", [1e12, 1e15, 1e19, 1e31, 1e38])
def test_large_sums(m, n, k, size):
    """Above what the parts' sums hold the outputs are the plain kernel's, infinities and NaN among them."""
    x, w = rand(m, k).clamp(-3, 3) * size, rand(n, k, seed=1).clamp(-3, 3) * min(size, 1e19)  # finite: 3e38 is below f32's largest number
    x[1] *= 1e-30 / size
    y = torch.empty((m, n), device=DEV)
    ops().dense_gemm(ops().dense(x, w, y))
    plain, want = in_order(x, w), x[1:2].double() @ w.double().T
    large = plain.isnan() | (plain.abs() > 2.0 ** 81)
    assert torch.equal(y[large].nan_to_num(7.0), plain[large].nan_to_num(7.0)) and torch.equal(y.isnan(), plain.isnan())
    assert bool(((y[1:2].double() - want).abs() <= bound(x[1:2], w)).all())


@pytest.mark.parametrize("m", [5, 150])
def test_what_the_parts_cannot_hold(m):
    """Infinities, NaN, f32's largest numbers and subnormal ones give what f32 gives, in their rows and columns alone."""
    x, w = rand(m, 96), rand(140, 96, seed=1)
    x[0, 3], x[1, 5], x[2, 7], x[3] = float("inf"), float("nan"), 3.4e38, x[3] * 1e-36
    w[:, 7] *= 0.1
    w[17, 9], w[18] = -float("inf"), 0.0
    y = torch.empty((m, 140), device=DEV)
    ops().dense_gemm(ops().dense(x, w, y))
    want = x.double() @ w.double().T
    assert torch.equal(y.isnan(), want.isnan()) and torch.equal(y.isinf(), want.isinf()) and torch.equal(y[y.isinf()].double(), want[want.isinf()])
    fine = want.isfinite()
    assert bool(((y.double() - want).abs() <= bound(x, w).nan_to_num(0, 0, 0))[fine].all())


# 235 tiles of 148 CTAs; and a gated one, whose pairs are computed again together
@pytest.mark.parametrize("m,n,k,act", [(208, 30000, 4096, 0), (40, 30016, 1028, 2)])
def test_tiles_of_infinities_before_finite_ones(m, n, k, act):
    """A CTA's first tile is infinite throughout: its outputs are the plain kernel's, and no wait of the next tile runs out meanwhile."""
    x, w = rand(m, k), rand(n, k, seed=1)
    w[:148 * 128, k - 1] = float("inf")
    y = torch.empty((m, n // 2 if act else n), device=DEV)
    ops().dense_gemm(ops().dense(x, w, y, act=act))
    if act:
        u = (x @ w.T).view(m, -1, 2, 16)
        want = (u[:, :, 0].double() / (1 + torch.exp(-u[:, :, 0].double())) * u[:, :, 1]).reshape(m, -1)
        fine = 148 * 64
        assert torch.equal(y[:, :fine].isnan(), want[:, :fine].isnan()) and torch.equal(y[:, :fine].isinf(), want[:, :fine].isinf())
        z = x.double() @ w[2 * fine:].double().T
        z = z.view(m, -1, 2, 16)
        want = (z[:, :, 0] * torch.sigmoid(z[:, :, 0]) * z[:, :, 1]).reshape(m, -1)
        assert float((y[:, fine:].double() - want).norm() / want.norm()) < 1e-6
    else:
        plain = x[:, k - 1:].sign() * float("inf")
        assert torch.equal(y[:, :148 * 128], plain.expand(m, 148 * 128))
        want = x.double() @ w[148 * 128:].double().T
        assert bool(((y[:, 148 * 128:].double() - want).abs() <= bound(x, w[148 * 128:])).all())


@pytest.mark.parametrize("batch_x,batch_w", [(0, None), (None, 0), (None, 4), (4, None), (0, 0), (100 * 64, 0)])
def test_batches_that_share_or_overlap(batch_x, batch_w):
    """Strides between batch entries that a tensor map may not have: the same rows or weights for all of them, or each four values further on."""
    b, m, n, k = 5, 40, 96, 64
    x, w, y = rand(b * 100 * k), rand(b * n * k, seed=1), torch.empty((b, m, n), device=DEV)
    p = ops().dense(x[:b * m * k].view(b, m, k), w.view(b, n, k), y)
    p.batch_x = p.batch_x if batch_x is None else batch_x
    p.batch_w = p.batch_w if batch_w is None else batch_w
    ops().dense_gemm(p)
    xs, ws = x.as_strided((b, m, k), (p.batch_x, k, 1)), w.as_strided((b, n, k), (p.batch_w, k, 1))
    assert bool(((y.double() - xs.double() @ ws.double().transpose(1, 2)).abs() <= bound(xs, ws)).all())


def test_a_row_stride_beyond_tensor_maps():
    x, w, y = rand(1, 64), rand(96, 64, seed=1), torch.empty((1, 96), device=DEV)
    p = ops().dense(x, w, y)
    p.ld_x = 1 << 38  # of one row: never used
    ops().dense_gemm(p)
    assert bool(((y.double() - x.double() @ w.double().T).abs() <= bound(x, w)).all())


@pytest.mark.parametrize("sizes", [[0, 3, 40, 0, 70, 1], [5] * 64, [300, 0]])
@pytest.mark.parametrize("act", [0, 2])
def test_groups(sizes, act):
    o, n, k = ops(), 192, 160
    rows = sum(sizes)
    x, w = rand(rows, k), rand(len(sizes), n, k, seed=1)
    offsets = torch.tensor([0] + sizes, device=DEV).cumsum(0).int()
    y = torch.full((rows + 1, n // 2 if act else n), 7.0, device=DEV)
    o.dense_gemm(o.grouped_dense(x, w, y[:rows], offsets, act=act))
    z = torch.cat([x[a:b].double() @ w[e].double().T for e, (a, b) in enumerate(zip(offsets[:-1].tolist(), offsets[1:].tolist()))])
    if act:
        z = z.view(rows, -1, 2, 16)
        z = (z[:, :, 0] * torch.sigmoid(z[:, :, 0]) * z[:, :, 1]).reshape(rows, -1)
    assert float((y[:rows].double() - z).norm() / z.norm()) < 1e-6 and bool((y[rows] == 7).all())
