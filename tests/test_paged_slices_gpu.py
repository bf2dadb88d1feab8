"""Paged attention where the number and the length of its slices change over: windows that reach few slices of a wide table, small batches, short contexts, against f64."""
import pytest
import torch

from tlaloc_b200 import ops

pytestmark = pytest.mark.gpu
DEV, BF16, F8 = "cuda:0", torch.bfloat16, torch.float8_e4m3fn


def check(lens, *, heads, kv_heads, dim, pool, block=16, width=None, window=None, rows_per_table=1, query=torch.float32, seed=0, splits=None):
    """Rows of the given lengths (a table's rows one after the other) against f64; what no row may see is NaN in the pools."""
    g = torch.Generator(device=DEV).manual_seed(seed)
    R, T = len(lens), len(lens) // rows_per_table
    longest = [max(lens[t * rows_per_table:(t + 1) * rows_per_table]) for t in range(T)]
    need = [-(-max(n, 1) // block) for n in longest]
    width = width or max(need)
    tables = torch.zeros((T, width), dtype=torch.int32)
    pages = (1 + torch.randperm(sum(need), generator=torch.Generator().manual_seed(seed))).tolist()
    at = 0
    for t, n in enumerate(need):
        tables[t, :n] = torch.tensor(pages[at:at + n], dtype=torch.int32)
        at += n
    keys, values = (torch.randn((at + 1, block, kv_heads, dim), generator=g, device=DEV, dtype=BF16) for _ in range(2))
    for t, n in enumerate(longest):
        first = max(0, min(lens[t * rows_per_table:(t + 1) * rows_per_table]) - window) if window else 0
        for p in (keys, values):
            flat = p.view(-1, kv_heads, dim)
            rows = (tables[t, :need[t], None].long() * block + torch.arange(block)).view(-1).to(DEV)
            flat[rows[n:]] = float("nan")
            flat[rows[:first // 16 * 16]] = float("nan")
            flat[rows[first // 16 * 16:first]] = 300.0  # read with weight zero: the kernels go by groups of 16, of which the window's first is the sequence's own
    keys[0] = values[0] = float("nan")  # page 0 is where unused table entries point
    keys, values = keys.to(pool), values.to(pool)
    q = torch.randn((R, heads, dim), generator=g, device=DEV).to(query)
    tables, seq = tables.to(DEV), torch.tensor(lens, dtype=torch.int32, device=DEV)
    scratch = torch.full((splits or -(-width * block // 256), R, heads, dim + 2), float("nan"), device=DEV)
    got = ops.paged_attention(q, keys, values, tables, seq, scale=dim ** -0.5, sliding_window=window, scratch=scratch).double()
    group = heads // kv_heads
    for r, n in enumerate(lens):
        lo = max(0, n - window) if window else 0
        if n == 0:
            assert bool((got[r] == 0).all())
            continue
        p = torch.arange(lo, n, device=DEV)
        page = tables[r // rows_per_table, p // block].long()
        k, v = (x[page, p % block].double().repeat_interleave(group, 1) for x in (keys, values))
        w = torch.softmax(torch.einsum("hd,phd->hp", q[r].double(), k) * dim ** -0.5, -1)
        want = torch.einsum("hp,phd->hd", w, v)
        # f32 scores and sums, queries and weights as two 16-bit parts (2^-16 of values of up to 5); a bf16 result is rounded to 2^-9
        tol = 2e-4 + (2.0 ** -8 * want.abs() if query == BF16 else 0.0)
        assert bool(((got[r] - want).abs() <= tol).all()), (r, n, float((got[r] - want).abs().max()))


# around the slices' ends: a window that touches one slice more than its length says, rows shorter than it, empty rows
LENS = [0, 1, 16, 255, 256, 257, 511, 513, 999, 1000, 1001, 1023, 1024, 1025, 1255, 1256, 1257, 2047, 2049, 3000]


@pytest.mark.parametrize("pool", [BF16, F8, torch.float32])
@pytest.mark.parametrize("window", [1, 16, 257, 1000, 5000])
@pytest.mark.parametrize("wide", [1, 11])
@pytest.mark.parametrize("rows_per_table", [1, 2])
def test_a_window_in_tables_of_any_width(pool, window, wide, rows_per_table):
    check(LENS, heads=8, kv_heads=2, dim=64, pool=pool, width=wide * 188, window=window, rows_per_table=rows_per_table, seed=window)


@pytest.mark.parametrize("pool", [BF16, F8])
@pytest.mark.parametrize("rows,heads,kv_heads,dim", [(1, 8, 1, 128), (1, 32, 8, 128), (5, 20, 5, 64), (40, 24, 8, 128), (100, 20, 5, 64)])
@pytest.mark.parametrize("context", [255, 300, 511, 701, 1025, 2000])
def test_small_batches_and_short_contexts(rows, heads, kv_heads, dim, context, pool):
    check([context - (context * 7 // 8) * r // max(1, rows - 1) for r in range(rows)], heads=heads, kv_heads=kv_heads, dim=dim, pool=pool, query=BF16, seed=context)


@pytest.mark.parametrize("pool", [BF16, F8])
@pytest.mark.parametrize("context,splits", [(12288, None), (12289, None), (16000, None), (16000, 7), (16000, 2), (25000, None)])
def test_one_long_sequence(context, splits, pool):
    """Up to 48 slices, and more positions than those hold; scratch that holds fewer."""
    check([context], heads=8, kv_heads=2, dim=128, pool=pool, query=BF16, splits=splits)
    check([context], heads=8, kv_heads=2, dim=128, pool=pool, query=BF16, splits=splits, window=4096)
