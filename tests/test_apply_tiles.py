"""Orders that stay in blocks of 1,024 are applied by tiles of 128 output entries, a run (the entries of a row in one
block of columns) at a time: bit-exact against numpy where runs end at the edges of tiles and change kind."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

RUNS = [1, 2, 31, 32, 33, 71, 72, 73, 127, 128, 129, 160, 161, 255, 256, 257, 700, 1023, 1024]


@pytest.mark.parametrize("values", [True, False])
@pytest.mark.parametrize("symmetric", [True, False])
@pytest.mark.parametrize("shift", [0, 1, 63, 127])
def test_runs_at_tile_edges(shift, symmetric, values):
    import chunkedgreedy_b200 as sp
    rng = np.random.default_rng(shift)
    n = 3 * 1024 + 77
    rows = [np.arange(shift)] if shift else [np.empty(0, int)]  # what lies in front of the first run
    for i, length in enumerate(RUNS * 3):
        cols = [1024 * (i % 3) + rng.choice(1024, length, replace=False)]
        if i % 2:  # a row of two or more runs
            cols.append(1024 * ((i + 1) % 3) + rng.choice(1024, RUNS[rng.integers(len(RUNS))], replace=False))
        if i % 5 == 0:
            cols.append(3 * 1024 + np.arange(rng.integers(0, 77)))
        rows.append(np.sort(np.concatenate(cols)))
        rows += [np.empty(0, int)] * (40 if i % 7 == 0 else i % 3)
    rows += [np.sort(rng.choice(n, rng.integers(0, 5), replace=False)) for _ in range(n - len(rows))]
    ptr = np.zeros(n + 1, np.int32)
    ptr[1:] = np.cumsum([r.size for r in rows])
    ind = np.concatenate(rows).astype(np.int32)
    val = rng.standard_normal(ind.size).astype(np.float32)
    order = np.concatenate([b + rng.permutation(min(1024, n - b)) for b in range(0, n, 1024)]).astype(np.int32)
    old2new = np.empty(n, np.int32)
    old2new[order] = np.arange(n)
    want_ptr = np.concatenate([[0], np.cumsum(np.diff(ptr)[order])])
    want_ind, want_val = [], []
    for r in order:
        c, v = ind[ptr[r]:ptr[r + 1]], val[ptr[r]:ptr[r + 1]]
        if symmetric:
            c = old2new[c]
            by = np.argsort(c)
            c, v = c[by], v[by]
        want_ind.append(c)
        want_val.append(v)
    got = sp.reorder(*(torch.from_numpy(x).cuda() for x in (ptr, ind, order)),
                     val=torch.from_numpy(val).cuda() if values else None, symmetric=symmetric)
    assert np.array_equal(got[0].cpu().numpy(), want_ptr)
    assert np.array_equal(got[1].cpu().numpy(), np.concatenate(want_ind))
    if values:
        assert np.array_equal(got[2].cpu().numpy(), np.concatenate(want_val))


def _apply_both_ways(lens, cols, order):
    """rows-only and symmetric apply of an order that stays in its blocks, against torch's sort of (row, column)"""
    import chunkedgreedy_b200 as sp
    n = lens.numel()
    ptr = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    ptr[1:] = torch.cumsum(lens, 0)
    old2new = torch.empty(n, dtype=torch.int64, device="cuda")
    old2new[order] = torch.arange(n, device="cuda")
    val = torch.arange(cols.numel(), device="cuda").float()  # (exact below 2^24: which entry went where)
    rows = old2new[torch.repeat_interleave(torch.arange(n, device="cuda"), lens)]
    want_ptr = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    want_ptr[1:] = torch.cumsum(lens[order], 0)
    for symmetric in (False, True):
        key = rows * n + (old2new[cols] if symmetric else cols)
        by = torch.argsort(key)
        got = sp.reorder(ptr.int(), cols.int(), order.int(), val=val, symmetric=symmetric)
        assert torch.equal(got[0].long(), want_ptr)
        assert torch.equal(got[1].long(), key[by] - rows[by] * n)
        assert torch.equal(got[2], val[by])


def _local_order(n, seed):
    rng = np.random.default_rng(seed)
    return torch.from_numpy(np.concatenate([b + rng.permutation(min(1024, n - b)) for b in range(0, n, 1024)])).cuda()


@pytest.mark.parametrize("length", [127, 128, 129, 255, 256, 257, 385, 8192, 1 << 20])
def test_tiles_of_a_long_row(length):
    # a row of one tile or several between rows of one entry: its further tiles are named by a warp
    n = 1 << 20
    lens = torch.ones(n, dtype=torch.int64, device="cuda")
    lens[1000] = length
    cols = torch.cat([torch.arange(1000), torch.arange(n - length, n), torch.arange(1001, n)]).cuda()
    _apply_both_ways(lens, cols, _local_order(n, length))


@pytest.mark.parametrize("gap", [1, 31, 32, 33, 1023, 1 << 21])
def test_empty_rows_inside_a_tile(gap):
    # rows without entries between those of one tile, in front of the first and behind the last one
    n = 128 * 1024 + 3 * gap
    lens = torch.zeros(n, dtype=torch.int64, device="cuda")
    filled = torch.cat([torch.arange(500), 500 + gap + torch.arange(0, 300, 3), n - gap - torch.arange(100, 0, -1)]).cuda()
    lens[filled] = 1 + torch.arange(filled.numel(), device="cuda") % 5
    rows = torch.repeat_interleave(torch.arange(n, device="cuda"), lens)
    nth = torch.arange(rows.numel(), device="cuda") - torch.repeat_interleave(torch.cumsum(lens, 0) - lens, lens)
    _apply_both_ways(lens, (rows * 7919 + nth * 400) % (n - 4000) % 1000 + nth * 1000, _local_order(n, gap))


@pytest.mark.parametrize("n", [1, 2047, 2048, 2049, 2048 * 2048, 2048 * 2048 + 1])
def test_blocks_of_rows(n):
    # rows counted in blocks of 2,048, whose sums are added up by each block or by a kernel of its own
    lens = (torch.arange(n, device="cuda") % 3 == 0).long()
    _apply_both_ways(lens, torch.arange(0, n, 3, device="cuda"), _local_order(n, n))


@pytest.mark.parametrize("tiles", [2, 16, 17, 18, 40])
def test_neighbouring_rows_of_several_tiles(tiles):
    # 70 rows of about so many tiles each: the first 16 further ones are named by the row's thread, the rest by its warp
    n = 1 << 13
    lens = torch.ones(n, dtype=torch.int64, device="cuda")
    lens[3000:3070] = tiles * 128 + torch.arange(70, device="cuda") * 61 % 131 - 65
    rows = torch.repeat_interleave(torch.arange(n, device="cuda"), lens)
    nth = torch.arange(rows.numel(), device="cuda") - torch.repeat_interleave(torch.cumsum(lens, 0) - lens, lens)
    cols = torch.sort(rows * n + (rows * 37 + nth) % n)[0] % n  # (ascending in every row)
    _apply_both_ways(lens, cols, _local_order(n, tiles))
