"""The buffer for the streams of the longest rows: as large as the call's own rows need, on the first call of a context
too, none where no row needs it, and smaller where memory is short - with the same results."""
import numpy as np
import pytest

import cases
import oracle

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _case(name):
    ptr, ind, _, _, params = cases.build(name)
    order, table = oracle.csg(ptr, ind, False, with_table=True, **params)
    return torch.from_numpy(ptr).cuda(), torch.from_numpy(ind).cuda(), params, order, table


def _check(got, order, table):
    assert np.array_equal(got[1].cpu().numpy().view(np.uint64), table)
    assert np.array_equal(got[0].cpu().numpy(), order)


@pytest.mark.parametrize("ahead", [-1, 1])
@pytest.mark.parametrize("name", ["dense_ties", "dense_c4096", "dense_m256"])
def test_the_first_call_makes_the_room(name, ahead):
    import chunkedgreedy_b200 as sp
    ptr, ind, params, order, table = _case(name)
    ctx = sp.Context()
    ctx.set_ahead_threshold(ahead)
    held = []
    for _ in range(2):
        _check(sp.csg_table(ptr, ind, ctx=ctx, **params), order, table)
        held.append(ctx.workspace_bytes())
    assert held[0] == held[1]
    ctx.close()


def test_a_mesh_holds_no_room_for_streams():
    import chunkedgreedy_b200 as sp
    side = 400
    y, x = torch.meshgrid(torch.arange(side), torch.arange(side), indexing="ij")
    rows, cols = [], []
    for dy in (-1, 0, 1):
        for dx in (-1, 0, 1):
            ok = (y + dy >= 0) & (y + dy < side) & (x + dx >= 0) & (x + dx < side)
            rows.append((y * side + x)[ok])
            cols.append(((y + dy) * side + x + dx)[ok])
    n = side * side
    key = (torch.cat(rows) * n + torch.cat(cols)).sort()[0]
    ptr = torch.zeros(n + 1, dtype=torch.int64)
    ptr[1:] = torch.cumsum(torch.bincount(key // n, minlength=n), 0)
    ctx = sp.Context()
    sp.chunk_similarity_greedy(ptr.int().cuda(), (key % n).int().cuda(), ctx=ctx)
    # keys, payloads, groups and their places: 44 bytes a nonzero and some; lists and a table of 16 entries a row
    assert ctx.workspace_bytes() <= 1.13 * (46 * key.numel() + (24 + 8 * 16) * n) + (1 << 20)
    ctx.close()


def test_short_of_memory_fewer_rows_get_a_chain():
    # 300 rows of 89,700 candidates would take 215 MB: with 100 left the call makes do with less
    import chunkedgreedy_b200 as sp
    ptr, ind, params, order, table = _case("dense_ties")
    ctx = sp.Context()
    ctx.set_stream_limit(1)
    _check(sp.csg_table(ptr, ind, ctx=ctx, **params), order, table)  # (everything but the streams is there now)
    ctx.set_stream_limit(0)
    torch.cuda.empty_cache()
    free, _ = torch.cuda.mem_get_info()
    hog = torch.empty(free - (100 << 20), dtype=torch.uint8, device="cuda")
    try:
        got = sp.csg_table(ptr, ind, ctx=ctx, **params)
        held = ctx.workspace_bytes()
    finally:
        del hog
        torch.cuda.empty_cache()
    _check(got, order, table)
    _check(sp.csg_table(ptr, ind, ctx=ctx, **params), order, table)
    assert held < ctx.workspace_bytes()
    ctx.close()
