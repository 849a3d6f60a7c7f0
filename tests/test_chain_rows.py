"""The kernel of the longest candidate streams, with the rows that go to it named by the caller: bit-exact tables and
orders against the CPU oracle, and the number of rows it took."""
import numpy as np
import pytest

import oracle

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

LEAST = 64  # candidates of the shortest row it takes


def _csr(rows):
    rows = [np.unique(np.asarray(r, dtype=np.int32)) for r in rows]
    ptr = np.zeros(len(rows) + 1, dtype=np.int32)
    ptr[1:] = np.cumsum([r.size for r in rows])
    return ptr, np.concatenate(rows)


def _candidates(ptr, ind, chunk):
    row = np.repeat(np.arange(ptr.size - 1), np.diff(ptr))
    _, at, count = np.unique(row // chunk * (1 << 32) + ind, return_inverse=True, return_counts=True)
    return np.bincount(row, weights=count[at] - 1, minlength=ptr.size - 1)


def _check(ptr, ind, limits, k, chunk):
    """csg with the chain kernel's rows forced, per limit on their streams; returns how many there were each time"""
    import chunkedgreedy_b200 as sp
    order, table = oracle.csg(ptr, ind, False, with_table=True, k=k, chunk_size=chunk)
    dp, di = torch.from_numpy(ptr).cuda(), torch.from_numpy(ind).cuda()
    ctx = sp.Context()
    ctx.set_chain_threshold(LEAST)
    took = []
    for limit in limits:
        ctx.set_stream_limit(limit)
        got_order, got = sp.csg_table(dp, di, ctx=ctx, k=k, chunk_size=chunk)
        assert np.array_equal(got.cpu().numpy().view(np.uint64), table)
        assert np.array_equal(got_order.cpu().numpy(), order)
        took.append(ctx.chain_rows())
    ctx.close()
    return took


@pytest.mark.parametrize("spread", [0, 30])
@pytest.mark.parametrize("k", [8, 16, 24, 32, 40])
@pytest.mark.parametrize("chunk", [1024, 1025, 66_000])
def test_streams_at_the_edges_of_a_window(chunk, k, spread):
    # 32 to 128 slots in rounds and 160 without; keys found by a word each, by hashed words, and without a table of
    # slots.  Streams that end at the edges of a window, a staged segment (256) and the ring (1,024)
    rng = np.random.default_rng(chunk + k + spread)
    lengths = [e + d for e in (64, 96, 128, 256, 512, 768, 1024, 1280, 2048) for d in (-1, 0, 1, 33)] + [6000]
    rows = [[] for _ in range(chunk)]
    col = 0
    for i, length in enumerate(lengths):
        for left in range(length, 0, -40):
            for r in 100 + rng.choice(150 if i % 2 else chunk - 100, min(left, 40), replace=False):
                rows[r].append(col)
            rows[i].append(col)
            col += 1
    for r in range(100, chunk):  # (columns of its own: they bring no candidates)
        extra = rng.integers(0, spread + 1)
        rows[r] += range(col, col + extra)
        col += extra
    ptr, ind = _csr(rows + [[] for _ in range(col - chunk)])
    long_enough = int((_candidates(ptr, ind, chunk) >= LEAST).sum())
    assert long_enough >= len(lengths) - 1
    assert _check(ptr, ind, (0,), k, chunk) == [long_enough]


def _random(columns, members, skew):
    """5,000 rows in five chunks of 1,000"""
    rng = np.random.default_rng(columns)
    rows = [[] for _ in range(5000)]
    for c in range(columns):
        for r in c % 5 * 1000 + (1000 * rng.random(members) ** skew).astype(np.int64):
            rows[r].append(c)
    return _csr(rows + [[]] * max(columns - 5000, 0))


@pytest.mark.parametrize("k", [8, 12, 24, 32])
def test_more_rows_than_a_block_scans(k):
    # all of them, and as many as fit into half the room: the cut lies behind the first 1,024
    ptr, ind = _random(9000, 33, 2)
    work = _candidates(ptr, ind, 1000)
    assert (np.sort(work)[::-1].cumsum() < work.sum() / 2).sum() > 1024
    all_rows = int((work >= LEAST).sum())
    took = _check(ptr, ind, (0, int(work.sum() / 2), 0), k, 1000)
    assert took[0] == took[2] == all_rows
    assert 1024 < took[1] < all_rows


@pytest.mark.parametrize("k", [8, 12, 24, 32])
def test_more_rows_than_a_limited_buffer_lists(k):
    # 4,096 rows and one for every 65,536 elements: here it is their number that is cut, not what they take
    ptr, ind = _random(9000, 10, 1)
    work = _candidates(ptr, ind, 1000)
    room = int(work.sum()) + 1000
    most = room // 65536 + 1 + 4096
    assert (work >= LEAST).sum() > most
    assert _check(ptr, ind, (room,), k, 1000) == [most]


@pytest.mark.parametrize("scale", [14, 15])
@pytest.mark.parametrize("k", [8, 20])
def test_no_more_rows_than_the_costs_hold_for(scale, k):
    # the whole matrix as one chunk and long streams throughout: the rule by costs ends at 4,096 rows and one for every
    # 65,536 candidates of those it takes
    import chunkedgreedy_b200 as sp
    from chunkedgreedy_b200 import synth
    ptr, ind, _ = synth.rmat_gcn(scale, 8)
    work = _candidates(ptr, ind, ptr.size)
    ctx = sp.Context()
    sp.similarity_graph(torch.from_numpy(ptr).cuda(), torch.from_numpy(ind).cuda(), k=k, ctx=ctx)
    took = ctx.chain_rows()
    ctx.close()
    assert 0 < took <= 4096 + int(np.sort(work)[::-1][:took].sum()) // 65536
