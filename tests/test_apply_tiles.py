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
