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


@pytest.mark.parametrize("offset", [0, 1])
def test_embedding_rows_longer_than_a_grid(offset):
    dim = 65535 * 512 + 516
    table = torch.arange(2 * dim + offset, dtype=torch.int32, device=DEV).float()[offset:].view(2, dim)
    assert torch.equal(ops().embedding(table, torch.tensor([1], dtype=torch.int32, device=DEV)), table[1:])


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


@pytest.mark.parametrize("sizes", [[1], [5, 0, 300, 1], [256, 256], [1] * 16])
def test_unpacking_of_a_steps_inputs(sizes):
    packed = torch.randint(-9, 9, (sum(sizes) + 3,), dtype=torch.int32, device=DEV)
    outs = [torch.full((n + 1,), 77, dtype=torch.int32, device=DEV) for n in sizes]
    ops().unpack_i32(packed, [o[:n] for o, n in zip(outs, sizes)])
    at = 0
    for o, n in zip(outs, sizes):
        assert torch.equal(o[:n], packed[at:at + n]) and int(o[n]) == 77
        at += n


def test_inputs_of_steps_in_flight_do_not_mix():
    """More steps than there are pinned buffers, queued behind a busy stream: each finds its own inputs."""
    from tlaloc_b200.step_model import StepModel

    m = StepModel(50, 50, 8, 30, 16, 100, DEV)
    seen, sent = [], []
    a = torch.randn((4096, 4096), device=DEV)
    for step in range(5):
        for _ in range(3):
            a = a @ a * 1e-4
        rng = np.random.default_rng(step)
        sent.append([rng.integers(0, 99, size=shape) for shape in ((50,), (50,), (50, 30), (50,), (50,))])
        m.set_inputs(*sent[-1])
        seen.append([t.clone() for t in (m.token_ids, m.positions, m.block_tables, m.seq_lens, m.slot_mapping)])
    for got, want in zip(seen, sent):
        assert all(np.array_equal(g.cpu().numpy(), w) for g, w in zip(got, want))
    with pytest.raises(RuntimeError):
        m.set_inputs(sent[0][0][:7], None, None, None, None)


@pytest.mark.parametrize("as_array", [False, True])
def test_page_locked_inputs_are_read_in_stream_order(as_array):
    """A copy from the device into the inputs is still on its way when they are handed over."""
    from tlaloc_b200.step_model import StepModel

    m = StepModel(50, 50, 8, 30, 16, 100, DEV)
    pinned = [torch.zeros(s, dtype=torch.int32).pin_memory() for s in ((50,), (50,), (50, 30), (50,), (50,))]
    coming = [torch.randint(0, 99, tuple(p.shape), dtype=torch.int32, device=DEV) for p in pinned]
    a = torch.randn((8192, 8192), device=DEV)
    torch.cuda.synchronize()
    for _ in range(10):
        a = a @ a * 1e-4
    for p, c in zip(pinned, coming):
        p.copy_(c, non_blocking=True)
    m.set_inputs(*([p.numpy() for p in pinned] if as_array else pinned))
    torch.cuda.synchronize()
    for got, want in zip((m.token_ids, m.positions, m.block_tables, m.seq_lens, m.slot_mapping), coming):
        assert torch.equal(got, want)


def test_the_first_step_locks_no_pages():
    from tlaloc_b200.step_model import StepModel

    m = StepModel(50, 50, 8, 30, 16, 100, DEV)
    before = torch.cuda.host_memory_stats()["num_host_alloc"]
    m.set_inputs(*(np.zeros(s, np.int32) for s in ((50,), (50,), (50, 30), (50,), (50,))))
    assert torch.cuda.host_memory_stats()["num_host_alloc"] == before
