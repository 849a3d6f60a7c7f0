"""The SpMM's choice of shape: the host-side rules on the CPU, the kernels they choose on the GPU."""
import ctypes
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SMS = 148

SHIM = r"""
#include "chunkedgreedy_b200/csrc/spmm_plan.h"
using namespace csg;
extern "C" void plan(int n, int nnz, int w, int align, int sms, int cap, long long *out) {
  const SpmmPlan p = spmm_plan(n, nnz, w, align, sms, cap);
  const SpmmShape s = p.shape;
  bool known = false;
#define CSG_KNOWN(G, V, P, M, W, E, B) known = known || s == SpmmShape{G, V, P, M, W, E, B};
  CSG_SPMM_SHAPES(CSG_KNOWN)
  const long long v[] = {s.lanes, s.vec, s.panels, s.masked, s.whole, s.even, s.blocks, p.rows_grid, p.long_grid,
                         p.unit, p.split, p.piece, known, batch_rows(s.lanes, s.vec),
                         batch_pairs(s.lanes, s.vec, s.panels, s.blocks), ROW_COST, M_WARPS, UNIT_MIN};
  for (unsigned i = 0; i < sizeof v / sizeof v[0]; ++i) out[i] = v[i];
}
"""
FIELDS = ("lanes vec panels masked whole even blocks rows_grid long_grid unit split piece known batch_rows "
          "batch_pairs row_cost warps unit_min").split()


@pytest.fixture(scope="module")
def plan(tmp_path_factory):
    d = tmp_path_factory.mktemp("spmm_plan")
    src, lib = d / "shim.cpp", d / "shim.so"
    src.write_text(SHIM)
    subprocess.check_call(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-I", ROOT, str(src), "-o", str(lib)])
    fn = ctypes.CDLL(str(lib)).plan

    def call(n, nnz, w, align=16):
        out = (ctypes.c_longlong * len(FIELDS))()
        fn(n, nnz, w, align, SMS, nnz // 128 + 1, out)
        return dict(zip(FIELDS, out))
    return call


def test_every_width_has_a_kernel_that_covers_it(plan):
    for n, nnz in ((1, 0), (10_000, 33_000), (1 << 20, 9 << 20), (1 << 20, 31 << 20), (1 << 22, 65_000_000)):
        for w in list(range(1, 700)) + [1024, 4096]:
            for align in (16, 8, 4):
                p = plan(n, nnz, w, align)
                what = (n, nnz, w, align, p)
                assert p["known"], what
                assert w % p["vec"] == 0 and align >= 4 * p["vec"], what
                if not p["masked"]:
                    assert w % (p["lanes"] * p["vec"] * p["panels"]) == 0, what
                if p["even"] != p["lanes"]:
                    assert w % (p["even"] * p["vec"]) == 0, what
                if p["lanes"] < 32 and w > 1:  # these walk one panel; groups of less than the row would walk it in turn
                    assert p["lanes"] * p["vec"] >= w, what
                assert p["unit_min"] <= p["unit"] <= p["batch_rows"] * p["row_cost"], what
                assert p["batch_pairs"] >= 16, what  # a row of a short unit fits
                shared = p["warps"] * (4 * (p["batch_rows"] + 1) + 8 * p["batch_pairs"])
                assert shared <= 48 << 10 and p["blocks"] * (shared + 1024) <= 228 << 10, what
                assert 1 <= p["rows_grid"] <= SMS * p["blocks"] and p["piece"] >= 1, what


@pytest.mark.parametrize("degree", [9.0, 3.3])
@pytest.mark.parametrize("w", [96, 128, 192, 256])
def test_short_rows_at_whole_warp_widths(plan, w, degree):
    # Matrices of short rows where a warp takes a row: lane groups fill the width without a rest,
    # and the units are as many as the warps of the grid that is launched draw in full rounds.
    for n in (10_000, 40_000, 150_000, 400_000, 1 << 20):
        nnz = int(n * degree)
        p = plan(n, nnz, w)
        assert p["lanes"] == 32 and w % (p["even"] * p["vec"]) == 0
        total = p["row_cost"] * n + nnz
        units, warps = total // p["unit"] + 1, p["rows_grid"] * p["warps"]
        if p["unit"] > p["unit_min"] and p["unit"] < p["batch_rows"] * p["row_cost"]:
            assert units <= -(-units // warps) * warps and units > 0.95 * (-(-units // warps)) * warps
        else:
            assert units <= warps or p["unit"] == p["batch_rows"] * p["row_cost"]


torch = pytest.importorskip("torch")


def _rows(kind, n):
    """Row lengths: `even` 9 for all; `mixed` 1 to 16, no two neighbours alike; `edge` 16 and 17 (the longest short
    row and one more); `late` short rows with one of 300 in the middle; `mild` 1 to 31, `over` 32 and 33."""
    if kind == "even":
        length = torch.full((n,), 9, device="cuda")
    elif kind == "mixed":
        length = torch.arange(n, device="cuda") * 7 % 16 + 1
    elif kind == "edge":
        length = 16 + (torch.arange(n, device="cuda") % 40 == 39).long()
    elif kind == "mild":
        length = torch.arange(n, device="cuda") * 7 % 31 + 1
    elif kind == "over":
        length = 32 + (torch.arange(n, device="cuda") % 40 == 39).long()
    else:
        length = torch.full((n,), 6, device="cuda")
        length[n // 2] = 300
    return length


def _check(length, w, g):
    import chunkedgreedy_b200 as sp
    n = length.numel()
    ptr = torch.zeros(n + 1, dtype=torch.int32, device="cuda")
    ptr[1:] = torch.cumsum(length, 0)
    nnz = int(ptr[-1])
    ind = torch.randint(0, n, (nnz,), generator=g, device="cuda", dtype=torch.int32)
    val = torch.randn(nnz, generator=g, device="cuda")
    B = torch.randn((n, w), generator=g, device="cuda")
    C = torch.full((n, w), float("nan"), device="cuda")
    sp.spmm(ptr, ind, val, B, out=C)
    rows = torch.repeat_interleave(torch.arange(n, device="cuda"), length)
    for c0 in range(0, w, 16):  # (in 16 columns at a time: the products of all nonzeros in 64 bits)
        part = B[:, c0:c0 + 16].double()[ind.long()] * val.double()[:, None]
        want = torch.zeros((n, part.shape[1]), dtype=torch.float64, device="cuda").index_add_(0, rows, part)
        size = torch.zeros_like(want).index_add_(0, rows, part.abs())
        # a sum of m terms in fp32, in any order: m + 1 roundings of 2^-24 each at most
        bound = (length[:, None].double() + 1) * 2.0 ** -24 * size
        assert torch.all((C[:, c0:c0 + 16].double() - want).abs() <= bound), (w, c0)


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["even", "mixed", "edge", "late"])
@pytest.mark.parametrize("n", [1, 9, 257, 30_011])
@pytest.mark.parametrize("w", [68, 80, 96, 124, 128, 144, 160, 176, 192, 256, 320, 384])
def test_units_of_short_rows(kind, n, w):
    g = torch.Generator(device="cuda").manual_seed(n + w)
    _check(_rows(kind, n), w, g)


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["even", "mixed", "late"])
@pytest.mark.parametrize("n,w", [(700_001, 48), (400_001, 128), (160_001, 160), (140_001, 192), (200_001, 256),
                                 (180_001, 144)])
def test_shapes_of_large_products(kind, n, w):
    # B beyond the lines where four blocks per SM (or, at 48, groups of four lanes) take over
    g = torch.Generator(device="cuda").manual_seed(w)
    _check(_rows(kind, n), w, g)


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["even", "mixed", "edge", "mild", "over", "late"])
@pytest.mark.parametrize("n", [1, 33, 30_011, 300_007])
def test_32_columns(kind, n):
    g = torch.Generator(device="cuda").manual_seed(n)
    _check(_rows(kind, n), 32, g)


def _best_of(ptr, ind, val, widths):
    import chunkedgreedy_b200 as sp
    n, best = ptr.numel() - 1, {}
    for w in widths:
        B, C = torch.randn((n, w), device="cuda"), torch.empty((n, w), device="cuda")
        times = []
        for _ in range(12):
            e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            e0.record()
            for _ in range(5):
                sp.spmm(ptr, ind, val, B, out=C, sync=False)
            e1.record()
            e1.synchronize()
            times.append(e0.elapsed_time(e1))
        best[w] = min(times)
    return best


@pytest.mark.gpu
def test_rows_of_24_at_32_columns_cost_half_of_64():
    # 24 nonzeros anywhere in each of 2^20 rows: half the bytes of 64 columns.  With a warp to a row of 32 columns
    # the ratio was 0.81, by lane groups it is 0.41.
    n = 1 << 20
    ptr = torch.arange(0, 24 * n + 1, 24, device="cuda", dtype=torch.int32)
    ind = torch.randint(0, n, (24 * n,), device="cuda", dtype=torch.int32)
    best = _best_of(ptr, ind, torch.randn(24 * n, device="cuda"), (32, 64))
    assert best[32] <= 0.65 * best[64], best


@pytest.mark.gpu
def test_a_mesh_costs_no_more_per_column_at_a_wide_width():
    # 9-point mesh in grid order, 2^20 rows: the gathers of 96 columns are 1.5 times those of 64.
    # With a warp to a row and a quarter of its lanes idle the ratio was 2.4, by lane groups it is 1.4.
    a = 1024
    v = torch.arange(a * a, device="cuda")
    y, x = v // a, v % a
    ok, cols = [], []
    for dy in (-1, 0, 1):
        for dx in (-1, 0, 1):
            ok.append((y + dy >= 0) & (y + dy < a) & (x + dx >= 0) & (x + dx < a))
            cols.append(v + dy * a + dx)
    ok, cols = torch.stack(ok, 1), torch.stack(cols, 1)
    ptr = torch.zeros(a * a + 1, dtype=torch.int32, device="cuda")
    ptr[1:] = torch.cumsum(ok.sum(1), 0)
    ind = cols[ok].int()
    val = torch.randn(ind.numel(), device="cuda")
    best = _best_of(ptr, ind, val, (64, 96))
    assert best[96] <= 1.9 * best[64], best
