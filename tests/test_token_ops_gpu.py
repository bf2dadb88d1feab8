"""The ends of a step at the sizes where their splits change, against the CPU oracle (needs a B200)."""
import numpy as np
import pytest
import torch

import oracle

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def ops():
    from tlaloc_b200 import ops as o

    return o


# one CTA a row up to 8191 columns, then clusters of 2, 4 and 8; multiples of four take 16-byte loads
@pytest.mark.parametrize("n", [1, 3, 4, 2047, 8191, 8192, 8195, 16384, 32767, 32768, 40004, 128256])
@pytest.mark.parametrize("rows", [1, 7])
def test_argmax_takes_the_first_maximum(n, rows):
    rng = np.random.default_rng(n)
    x = rng.standard_normal((rows, n)).astype(np.float32)
    for r in range(rows):  # ties at any two places
        i, j = sorted(rng.integers(0, n, size=2))
        x[r, i] = x[r, j] = 9.0
    got = ops().argmax(torch.from_numpy(x).to(DEV)).cpu().numpy()
    assert np.array_equal(got, x.argmax(1)) and np.array_equal(got, oracle.argmax(x))


@pytest.mark.parametrize("n", [5, 8192, 32768])
def test_argmax_of_rows_without_a_largest_number(n):
    x = torch.full((4, n), float("nan"), device=DEV)
    x[1, n - 2] = -1e30         # the only number
    x[2] = -float("inf")        # all equal: the first
    x[3, n // 2:] = -float("inf")
    assert ops().argmax(x).tolist() == [0, n - 2, 0, n // 2]
    odd = torch.zeros((3 * n + 1,), device=DEV)[1:].view(3, n)  # rows off 16 bytes
    odd[:, n - 1] = 1.0
    assert ops().argmax(odd).tolist() == [n - 1] * 3


@pytest.mark.parametrize("dim", [1, 7, 8, 96, 1020, 1024, 1032, 8192])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("offset", [0, 1])
def test_embedding_rows(dim, dtype, offset):
    table = torch.randn((9 * dim + offset,), device=DEV).to(dtype)[offset:].view(9, dim)
    ids = torch.tensor([3, -2, 8, 0, 99, 3], dtype=torch.int32, device=DEV)  # ids outside are clamped
    assert torch.equal(ops().embedding(table, ids), table[ids.long().clamp(0, 8)].float())
