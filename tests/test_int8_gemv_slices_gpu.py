"""The row-vector int8 projection over every number of slices of k: one to eight CTAs of a cluster share a column tile, some of them without rows of their own."""
import numpy as np
import pytest
import torch

from tlaloc_b200 import ops

pytestmark = pytest.mark.gpu

# (k, n): shapes whose tiles of 128 columns fill the SMs with 1, 2, 3, 4, 5, 6 and 8 slices; ragged ends of k and n; slices that would have no rows (2560, 8192), that would be too
# short beyond two CTAs an SM (520, 640, 2048), and a second wave of short ones (4096, 11008: eight up to 8 rows, five from 9 on); two and three stages on either side of their lines
SHAPES = [(128, 28672), (264, 37888), (1536, 28656), (520, 14208), (640, 14336), (776, 9472), (1032, 8064), (1032, 7088), (16, 16), (2048, 144),
          (2048, 8192), (2560, 8192), (2568, 8192), (4096, 11008), (4104, 6144), (4096, 28656), (4104, 32752)]


@pytest.mark.parametrize("rows", [1, 8, 9, 16])
@pytest.mark.parametrize("k,n", SHAPES)
def test_every_slice_count(k, n, rows):
    """Whole activations: every sum stays below 2^24 (4104 x 8 x 128 = 2^22), so f32 sums in any order are exact."""
    rng = np.random.default_rng(k + n + rows)
    x = rng.integers(-8, 9, size=(rows, k)).astype(np.float32)
    codes = rng.integers(-128, 128, size=(k, n), dtype=np.int8)
    residual = rng.integers(-100, 101, size=(rows, n)).astype(np.float32)
    scales = (0.25 * 2.0 ** rng.integers(0, 3, size=n)).astype(np.float32)
    t = lambda a: torch.from_numpy(a).cuda()
    want = torch.from_numpy((x.astype(np.float64) @ codes.astype(np.float64)) * scales + residual).float()
    for const in (False, True):
        got = ops.int8_gemm(t(x).bfloat16(), t(codes), t(scales), residual=t(residual), weights_const=const)
        assert torch.equal(got.cpu(), want)
