"""Chunks of more than 1,024 rows, sketches of 32 slots and the longest rows of a call take kernels of their own:
bit-exact tables and orders against the CPU oracle at the sizes where they change hands."""
import numpy as np
import pytest

import oracle

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _check(ptr, ind, limits=(0,), **params):
    import chunkedgreedy_b200 as sp
    order, table = oracle.csg(ptr, ind, False, with_table=True, **params)
    dp, di = torch.from_numpy(ptr).cuda(), torch.from_numpy(ind).cuda()
    ctx = sp.Context()
    for limit in limits:
        ctx.set_stream_limit(limit)
        got_order, got = sp.csg_table(dp, di, ctx=ctx, **params)
        assert np.array_equal(got.cpu().numpy().view(np.uint64), table)
        assert np.array_equal(got_order.cpu().numpy(), order)
    ctx.close()


def _csr(rows, n):
    rows = [np.unique(np.asarray(r, dtype=np.int32)) for r in rows]
    rows += [np.empty(0, dtype=np.int32)] * (n - len(rows))
    ptr = np.zeros(n + 1, dtype=np.int32)
    ptr[1:] = np.cumsum([r.size for r in rows])
    return ptr, np.concatenate(rows)


@pytest.mark.parametrize("chunk", [2048, 2049, 4095, 4096, 4097])
def test_tall_chunks_grouped_by_a_block_each(chunk):
    # enough chunks for a block each; among them a column that holds every row of its chunk, and one in all
    # rows but one (13 bits of a group's length), a chunk with more members of groups than the block has
    # places for, one with more nonzeros than it looks at, empty rows, and a last chunk of one row
    rng = np.random.default_rng(chunk)
    n = 40 * chunk + 1
    count = rng.integers(0, 4, n)
    count[3 * chunk:4 * chunk] = 6     # 16,384 members and more in groups
    count[4 * chunk:5 * chunk] = 8     # 28,672 nonzeros and more
    rows = [rng.integers(0, 9000, c) + 1 for c in count]
    for i in range(chunk):
        rows[chunk + i] = [0] + list(rows[chunk + i][:1])
        if i != 17:
            rows[2 * chunk + i] = [0, 1 + i % 3000]
    ptr, ind = _csr(rows, n)
    _check(ptr, ind, k=16, chunk_size=chunk)
    import chunkedgreedy_b200 as sp
    got = sp.count_pillars(torch.from_numpy(ptr).cuda(), torch.from_numpy(ind).cuda(), chunk)
    assert got == oracle.count_pillars(ptr, ind, chunk)


def _hubs(n, hubs, members, seed):
    """rows of two entries that lie in no hub or one or two, and eight that lie in all hubs"""
    rng = np.random.default_rng(seed)
    rows = [list(rng.integers(hubs, n, 2)) for _ in range(n)]
    for h in range(hubs):
        for r in rng.integers(0, n, members):
            rows[r].append(h)
    for r in range(0, n, n // 8):
        rows[r] += range(hubs)
    return _csr(rows, n)


@pytest.mark.parametrize("k", [1, 4, 8])
@pytest.mark.parametrize("n,hubs,members", [(1000, 120, 800), (9000, 40, 2000), (45_000, 32, 2300)])
def test_rows_of_32_slots_against_oracle(n, hubs, members, k):
    # the key table in shared memory and, for 45,000 rows, none; rows on either side of a warp each
    ptr, ind = _hubs(n, hubs, members, n)
    _check(ptr, ind, limits=(0, 1), k=k, chunk_size=n)


@pytest.mark.parametrize("k", [4, 8])
@pytest.mark.parametrize("chunk", [512, 1024, 2048, 4096])
def test_32_slots_one_chunk_ahead(chunk, k):
    # the chunk with the most nonzeros transposed first, its rows of 65,536 candidates and more on the second stream
    import chunkedgreedy_b200 as sp
    rng = np.random.default_rng(chunk + k)
    n = 4 * chunk + 100
    rows = [list(rng.integers(0, n, 4)) for _ in range(n)]
    for c in range(900):  # hubs of the second chunk
        for r in rng.choice(chunk, 150, replace=False):
            rows[chunk + r].append(c)
    for r in range(chunk + 10, chunk + 40):
        rows[r] += range(900)
    ptr, ind = _csr(rows, n)
    order, table = oracle.csg(ptr, ind, False, with_table=True, k=k, chunk_size=chunk)
    ctx = sp.Context()
    ctx.set_ahead_threshold(1)
    for limit in (0, 0, 300_000):
        ctx.set_stream_limit(limit)
        got = sp.csg_table(torch.from_numpy(ptr).cuda(), torch.from_numpy(ind).cuda(), ctx=ctx, k=k, chunk_size=chunk)
        assert np.array_equal(got[1].cpu().numpy().view(np.uint64), table)
        assert np.array_equal(got[0].cpu().numpy(), order)
    ctx.close()


@pytest.mark.parametrize("k", [8, 16, 40])
@pytest.mark.parametrize("chunk,skew", [(1024, 10), (1025, 10), (5000, 5), (40_000, 4)])
def test_rows_by_warp_before_the_lanes(chunk, skew, k):
    # streams from a few to tens of thousands of candidates: how many octaves below the longest
    # go to a warp each changes with the rows of a chunk
    rng = np.random.default_rng(chunk + k)
    n = 40_000
    rows = [list((n * rng.random(c) ** skew).astype(np.int64)) for c in 1 + rng.geometric(0.2, n) % 60]
    ptr, ind = _csr(rows, n)
    _check(ptr, ind, limits=(0, 3000), k=k, chunk_size=chunk)


@pytest.mark.parametrize("spread", [0, 30])
@pytest.mark.parametrize("k", [16, 24, 32])
@pytest.mark.parametrize("chunk", [1024, 1025, 66_000])
def test_windows_of_the_chains(chunk, k, spread):
    # 64, 96 and 128 slots; keys found by a word each, by hashed words, and without a table of slots.  Streams that end
    # at the edges of a window (32, 64), a staged segment (256) and the ring (1,024); columns of 40 rows drawn from few
    # (most candidates hit) and many; Dice terms all but equal (whole windows) and of rows with 1 to 30 more entries
    rng = np.random.default_rng(chunk + k + spread)
    lengths = [e + d for e in (32, 64, 256, 512, 768, 1024, 1280, 2048) for d in (-1, 0, 1, 33)] + [6000, 9001]
    rows = [[] for _ in range(chunk)]
    col = 0
    for i, length in enumerate(lengths):
        left = length
        while left > 0:
            take = min(left, 40)
            pool = 150 if i % 2 else chunk - 100
            for r in 100 + rng.choice(pool, take, replace=False):
                rows[r].append(col)
            rows[i].append(col)
            left -= take
            col += 1
    for r in range(100, chunk):  # (columns of its own: they bring no candidates)
        extra = rng.integers(0, spread + 1)
        rows[r] += range(col, col + extra)
        col += extra
    ptr, ind = _csr(rows, max(col, chunk))
    _check(ptr, ind, k=k, chunk_size=chunk)


@pytest.mark.parametrize("k", [12, 24, 32])
def test_many_rows_with_a_chain_each(k):
    # 5,000 rows of some 2,500 candidates and fewer: more rows than one block scans at a time, more than the list of
    # chains takes, and, with little room for their streams, only the first of them
    rng = np.random.default_rng(k)
    rows = [[] for _ in range(5000)]
    for c in range(9000):
        base = c % 5 * 1000
        for r in base + (1000 * rng.random(33) ** 2).astype(np.int64):
            rows[r].append(c)
    ptr, ind = _csr(rows, 9000)
    _check(ptr, ind, limits=(0, 200_000, 0), k=k, chunk_size=1000)
