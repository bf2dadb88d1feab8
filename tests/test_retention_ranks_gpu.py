"""One token of a recurrence whose heads' columns are shared by the CTAs of a cluster (few rows, large states), against the same rows among many (one CTA a head)."""
import pytest
import torch

from tlaloc_b200 import ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("heads,dim,vdim", [(1, 256, 512), (3, 128, 256), (2, 129, 258), (1, 512, 1021), (1, 256, 135), (5, 300, 130), (2, 70, 1024)])
def test_ranks_agree_with_one_cta(heads, dim, vdim, dtype):
    g = torch.Generator(device="cuda").manual_seed(1)
    r = lambda *s: torch.randn(s, generator=g, device="cuda")
    many, vp, dims = 260 // heads, -(-vdim // 4) * 4, dim // 4 * 2
    state, x = r(many + 1, heads, dim, vp), r(many, 2 * heads * (dim + vdim))
    positions = torch.randint(0, 3, (many,), generator=g, device="cuda", dtype=torch.int32)
    cos, sin, decay = r(3, dims // 2), r(3, dims // 2), torch.rand(heads, generator=g, device="cuda")
    slots = torch.randperm(many, generator=g, device="cuda").to(torch.int32) + 1

    def step(rows, state):
        out = torch.empty((rows, heads * vdim), device="cuda", dtype=dtype)
        ops.retention_step(x[:rows], positions[:rows], cos, sin, decay, slots[:rows], state, out, heads=heads, dim=dim, vdim=vdim, rot_dims=dims, k_scale=0.1, eps=1e-5)
        return out

    whole = state.clone()
    want = step(many, whole).double()
    for rows in (1, 2, 7):
        few = state.clone()
        got = step(rows, few).double()
        for t in range(rows):
            assert torch.equal(few[slots[t]], whole[slots[t]])  # a state's values do not depend on how they are shared out
        touched = set(slots[:rows].tolist())
        assert all(torch.equal(few[s], state[s]) for s in range(many + 1) if s not in touched)
        # sums of dim products in another order: dim * 2^-24 of the largest partial sum, twice over the norm; then the result's own rounding
        scale = want[:rows].abs().max()
        assert float((got - want[:rows]).abs().max() / scale) <= (dim * 2.0 ** -23 if dtype == torch.float32 else 2.0 ** -7)
