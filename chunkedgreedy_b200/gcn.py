"""Two-layer GCN on the library's SpMM, and the reorder-then-train experiment.

Mirrors the reference's end-to-end script (experiments/e2e_gcn.py): the propagation
operator is ``op(x) = D^-1/2 A D^-1/2 x`` on a symmetric pattern with unit values, the
autograd function uses the same ``op`` for the backward pass (valid because the operator
is symmetric, e2e_gcn.py:50-58), the model is ``Linear(in, hidden) -> op -> ReLU ->
Linear(hidden, classes) -> op -> log_softmax`` with the mean negative log-likelihood as
loss (:126-137), three warm-up epochs precede the timed ones (:139-146), and the total is
``reorder + permute + epochs`` (:1-4).  torch is used for the dense layers, autograd and
the optimiser only; every sparse product is ``sporder_spmm``.

The reference trains with Adam(lr=0.01) (:128); the benchmark definition this repository
follows asks for full-batch SGD, so ``optimizer`` selects either and both arms of a
comparison use the same one.
"""
from __future__ import annotations

import time

import torch
import torch.nn.functional as F

from . import _ctx, _enter, _lib, chunk_similarity_greedy, reorder, spmm

__all__ = ["SpMMFn", "GraphOperator", "GCN", "train", "reorder_and_train", "breakeven_epochs"]


class SpMMFn(torch.autograd.Function):
    """y = op(x) with dy/dx applied through the same (symmetric) operator."""

    @staticmethod
    def forward(ctx, x, op):
        ctx.op = op
        return op(x.contiguous())

    @staticmethod
    def backward(ctx, g):
        return ctx.op(g.contiguous()), None


class GraphOperator:
    """x -> A x for a CSR matrix held on the GPU (values already normalised), counting
    the time spent in SpMM with CUDA events when ``timed`` is set."""

    def __init__(self, ptr, ind, val, ctx=None, timed=False):
        self.ptr, self.ind, self.val, self.ctx, self.timed = ptr, ind, val, ctx, timed
        self.spmm_ms = 0.0
        self._pending = []

    def __call__(self, x):
        if not self.timed:
            return spmm(self.ptr, self.ind, self.val, x, ctx=self.ctx, sync=False)
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record()
        out = spmm(self.ptr, self.ind, self.val, x, ctx=self.ctx, sync=False)
        e1.record()
        self._pending.append((e0, e1))
        return out

    def row_sums(self):
        """A 1, one float per row."""
        out = torch.empty(self.ptr.numel() - 1, dtype=torch.float32, device=self.ptr.device)
        ctx = _ctx(self.ctx, self.ptr)
        with torch.cuda.device(self.ptr.device):
            _enter(ctx, self.ptr)
            if _lib.load().sporder_row_sums(ctx.handle, out.numel(), self.val.numel(), self.ptr.data_ptr(),
                                            self.val.data_ptr(), out.data_ptr()) != 0:
                _lib.check()
        return out

    def collect(self):
        torch.cuda.synchronize()
        self.spmm_ms += sum(a.elapsed_time(b) for a, b in self._pending)
        self._pending.clear()
        return self.spmm_ms


def moved_columns(width):
    """Full width that a sparse product of ``width`` columns costs as much as, or more: a power of two up
    to 32, a multiple of four beyond."""
    return max(4, 1 << (width - 1).bit_length()) if width <= 32 else (width + 3) // 4 * 4


def padded_columns(width):
    """Columns to take a sparse product of ``width`` at where the caller may choose.  Symmetrised R-MAT scale 20, us: 3
    columns 480 and 4 425, 7 651 and 8 416, 13 1,014 and 16 479, 20 850, 30 1,058 and 32 634.  An odd width from 17 on
    has a lane per column (17 628, 47 880 and 48 832), beyond 32 the rest is small."""
    return width if width > 32 or (width > 16 and width % 2) else moved_columns(width)


def step_widths(rows, in_dim, hidden, classes, fused):
    """Widths of a training step's four sparse products, (first layer forward, second forward, second
    backward, first backward).  The second operator goes behind the second linear layer (op(h) W2^T =
    op(h W2^T)) where that moves no more columns, on the fused route, which saves besides; on torch's where the
    columns saved are worth a bias and a padding of their own (300 inputs, 64 hidden units, 10 classes: 4,096 rows 0.67 ms
    as it stands and 0.70 behind, 1.05 M rows 6.7 and 6.1).  Logits are padded from 131,072 rows on: below, a step
    is its launches (4,096 rows 0.58 ms, 0.60 padded; 60,000 rows 0.62 and 0.65).  The first layer keeps its order: hidden units within a rounding
    of zero decide by their sign, and op(x) W1^T rounds differently.  Backward, the fused route takes op(x)
    or op(D), whichever moves fewer columns (128 inputs, 64 hidden units, 16 classes, 1.05 M rows: 4.8 and 4.2 ms)."""
    saved = hidden - moved_columns(classes)
    behind = saved >= 0 if fused else rows * saved >= 1 << 22
    second = hidden if not behind else padded_columns(classes) if rows >= 1 << 17 else classes
    first = in_dim if fused and moved_columns(in_dim) <= moved_columns(hidden) else hidden
    return hidden, second, second, first


def _call(fn, *args):
    if fn(*args) != 0:
        _lib.check()


class LayersFn(torch.autograd.Function):
    """relu(op(x W1^T + b1)) W2^T for features that want no gradient, in ``out`` columns, those
    behind the classes zero.  The backward pass needs the first layer's gradient D^T op(x) = op(D)^T x (op
    is symmetric): one sparse product over whichever is narrower, and everything dense in one or two kernels."""

    @staticmethod
    def forward(ctx, x, op, w1, b1, w2, out, first):
        n, hidden, classes = x.shape[0], w1.shape[0], w2.shape[0]
        x, w1, b1, w2 = x.contiguous(), w1.contiguous(), b1.contiguous(), w2.contiguous()
        y = torch.empty((n, hidden), dtype=torch.float32, device=x.device)
        u = torch.empty((n, out), dtype=torch.float32, device=x.device)
        ctx.lib_ctx = _ctx(getattr(op, "ctx", None), x)
        lib, handle = _lib.load(), ctx.lib_ctx.handle
        with torch.cuda.device(x.device):
            _enter(ctx.lib_ctx, x)
            _call(lib.sporder_linear, handle, n, x.shape[1], hidden, x.data_ptr(), w1.data_ptr(), b1.data_ptr(),
                  y.data_ptr())
            z = op(y)
            _enter(ctx.lib_ctx, x)
            _call(lib.sporder_gcn_forward_padded, handle, n, hidden, classes, out, z.data_ptr(), w2.data_ptr(),
                  u.data_ptr())
        ctx.op, ctx.first = op, first
        ctx.save_for_backward(x, z, w2)
        return u

    @staticmethod
    @torch.autograd.function.once_differentiable
    def backward(ctx, g):
        x, z, w2 = ctx.saved_tensors
        op = ctx.op
        n, in_dim, hidden, classes, out = x.shape[0], x.shape[1], z.shape[1], w2.shape[0], g.shape[1]
        g = g.contiguous()
        dw1 = torch.empty((hidden, in_dim), dtype=torch.float32, device=x.device)
        db1 = torch.empty(hidden, dtype=torch.float32, device=x.device)
        dw2 = torch.empty((classes, hidden), dtype=torch.float32, device=x.device)
        lib, handle = _lib.load(), ctx.lib_ctx.handle
        with torch.cuda.device(x.device):
            if ctx.first == in_dim:
                p = op(x)
                s = op.row_sums() if hasattr(op, "row_sums") else op(torch.ones_like(x[:, :1]))[:, 0].contiguous()
                _enter(ctx.lib_ctx, x)
                _call(lib.sporder_gcn_backward_padded, handle, n, in_dim, hidden, classes, out, g.data_ptr(),
                      z.data_ptr(), p.data_ptr(), s.data_ptr(), w2.data_ptr(), dw1.data_ptr(), db1.data_ptr(),
                      dw2.data_ptr())
            else:
                d = torch.empty_like(z)
                _enter(ctx.lib_ctx, x)
                _call(lib.sporder_gcn_hidden_gradient, handle, n, hidden, classes, out, g.data_ptr(), z.data_ptr(),
                      w2.data_ptr(), d.data_ptr(), dw2.data_ptr())
                e = op(d)
                _enter(ctx.lib_ctx, x)
                _call(lib.sporder_gcn_input_gradients, handle, n, in_dim, hidden, e.data_ptr(), x.data_ptr(),
                      dw1.data_ptr(), db1.data_ptr())
        return None, None, dw1, db1, dw2, None, None


def _pad_columns(g, width, ctx):
    if not (g.is_cuda and g.dtype == torch.float32):
        return F.pad(g, (0, width - g.shape[1]))
    g = g.contiguous()
    padded = torch.empty((g.shape[0], width), dtype=torch.float32, device=g.device)
    ctx = _ctx(ctx, g)
    with torch.cuda.device(g.device):
        _enter(ctx, g)
        _call(_lib.load().sporder_pad_columns, ctx.handle, g.shape[0], g.shape[1], width, g.data_ptr(),
              padded.data_ptr())
    return padded


class LogitsFn(torch.autograd.Function):
    """op(u) + b over the first ``classes`` columns of u."""

    @staticmethod
    def forward(ctx, u, op, b, classes):
        ctx.op, ctx.width, ctx.biased = op, u.shape[1], b is not None
        z = op(u.contiguous())[:, :classes]
        return z + b if ctx.biased else z.contiguous()

    @staticmethod
    def backward(ctx, g):
        db = g.sum(0) if ctx.biased else None
        g = _pad_columns(g, ctx.width, getattr(ctx.op, "ctx", None))
        return ctx.op(g.contiguous()), None, db, None


def _logits(u, op, b, classes):
    if u.shape[1] != classes:
        return LogitsFn.apply(u, op, b, classes)
    z = SpMMFn.apply(u, op)  # (the bias by torch's own autograd: a small step is its host work)
    return z if b is None else z + b


def _plain(layer):
    """A linear layer that is its weight and bias and nothing else: no hooks (which recompute a normalised weight, count
    calls, ...), no other module in its place."""
    return type(layer) is torch.nn.Linear and not (layer._forward_hooks or layer._forward_pre_hooks
                                                   or layer._backward_hooks or layer._backward_pre_hooks)


class GCN(torch.nn.Module):
    """Linear -> op -> ReLU -> op -> Linear; `step_widths` says where the operators go."""

    def __init__(self, in_dim, hidden, classes):
        super().__init__()
        self.w1 = torch.nn.Linear(in_dim, hidden)
        self.w2 = torch.nn.Linear(hidden, classes)

    def forward(self, x, op):
        # (a small step is its host work, and a module's attributes are looked up one by one)
        l1, l2 = self.w1, self.w2
        if not (_plain(l1) and _plain(l2)):
            return l2(SpMMFn.apply(F.relu(SpMMFn.apply(l1(x), op)), op))
        w1, b1, w2, b2 = l1.weight, l1.bias, l2.weight, l2.bias
        (hidden, in_dim), classes = w1.shape, w2.shape[0]
        # limits of the fused kernels; others, and features that want a gradient, by torch
        fused = (not x.requires_grad and in_dim % 4 == 0 and in_dim <= 128 and hidden % 4 == 0 and hidden <= 128
                 and classes <= 48 and moved_columns(classes) <= hidden and b1 is not None
                 and x.data_ptr() % 16 == 0
                 and all(t.is_cuda and t.dtype == torch.float32 for t in (x, w1, w2)))
        _, out, _, first = step_widths(x.shape[0], in_dim, hidden, classes, fused)
        if fused:
            return _logits(LayersFn.apply(x, op, w1, b1, w2, out, first), op, b2, classes)
        h = F.relu(SpMMFn.apply(l1(x), op))
        if out == hidden:
            return l2(SpMMFn.apply(h, op))
        return _logits(F.linear(h, w2 if out == classes else F.pad(w2, (0, 0, 0, out - classes))), op, b2, classes)


def normalised_values(ptr, ind):
    """D^-1/2 A D^-1/2 values for a unit-valued pattern, D = clamp_min(row sums, 1)
    (experiments/e2e_gcn.py:116-123)."""
    n = ptr.numel() - 1
    deg = (ptr[1:] - ptr[:-1]).to(torch.float32).clamp_min(1.0)
    dinv = deg.rsqrt()
    rows = torch.repeat_interleave(torch.arange(n, device=ptr.device), (ptr[1:] - ptr[:-1]).long())
    return (dinv[rows] * dinv[ind.long()]).contiguous()


def train(ptr, ind, val, x, y, *, hidden=128, classes=16, epochs=200, warmup=3, lr=0.01,
          optimizer="sgd", seed=0, ctx=None):
    """Full-batch training; returns dict(train_ms, epoch_ms, spmm_ms_per_epoch, final_loss)."""
    torch.manual_seed(seed)
    model = GCN(x.shape[1], hidden, classes).to(x.device)
    opt = (torch.optim.SGD(model.parameters(), lr=lr) if optimizer == "sgd"
           else torch.optim.Adam(model.parameters(), lr=lr))
    op = GraphOperator(ptr, ind, val, ctx=ctx, timed=True)

    def epoch():
        opt.zero_grad()
        z = model(x, op)
        loss = -F.log_softmax(z, 1).gather(1, y[:, None]).mean()
        loss.backward()
        opt.step()
        return loss

    for _ in range(warmup):
        epoch()
    op.collect()
    op.spmm_ms = 0.0
    torch.cuda.synchronize()
    t0 = time.perf_counter()
    for _ in range(epochs):
        loss = epoch()
    torch.cuda.synchronize()
    train_ms = (time.perf_counter() - t0) * 1e3
    spmm_ms = op.collect()
    return dict(train_ms=train_ms, epoch_ms=train_ms / max(epochs, 1),
                spmm_ms_per_epoch=spmm_ms / max(epochs, 1), final_loss=float(loss))


def breakeven_epochs(reorder_ms, perm_ms, epoch_ms_original, epoch_ms_reordered):
    """Epochs after which reordering has paid for itself: (reorder + permute) over the time
    one epoch saves, infinite when an epoch did not get faster (analysis/e2e.py:32-33)."""
    gain = float(epoch_ms_original) - float(epoch_ms_reordered)
    return (float(reorder_ms) + float(perm_ms)) / gain if gain > 0 else float("inf")


def reorder_and_train(ptr, ind, val, x, y, *, ctx=None, **kw):
    """The amortisation experiment: train on the matrix as given, then reorder once with
    csg, apply P A P^T to the matrix and P to features and labels, and train again.
    Returns both results plus reorder_ms, perm_ms and the end-to-end totals."""
    base = train(ptr, ind, val, x, y, ctx=ctx, **kw)
    torch.cuda.synchronize()
    t0 = time.perf_counter()
    order, timing = chunk_similarity_greedy(ptr, ind, is_symmetric=True, with_timing=True, ctx=ctx)
    reorder_ms = timing["wall_ms"]
    torch.cuda.synchronize()
    t0 = time.perf_counter()
    p2, i2, v2 = reorder(ptr, ind, order, val=val, symmetric=True, ctx=ctx)
    x2, y2 = x[order.long()].contiguous(), y[order.long()].contiguous()
    torch.cuda.synchronize()
    perm_ms = (time.perf_counter() - t0) * 1e3
    re = train(p2, i2, v2, x2, y2, ctx=ctx, **kw)
    total_re = reorder_ms + perm_ms + re["train_ms"]
    return dict(original=base, reordered=re, reorder_ms=reorder_ms, perm_ms=perm_ms,
                total_original_ms=base["train_ms"], total_reordered_ms=total_re,
                epoch_speedup=base["epoch_ms"] / re["epoch_ms"],
                spmm_speedup=(base["spmm_ms_per_epoch"] / re["spmm_ms_per_epoch"]
                              if re["spmm_ms_per_epoch"] > 0 else float("nan")),
                breakeven_epochs=breakeven_epochs(reorder_ms, perm_ms, base["epoch_ms"], re["epoch_ms"]),
                end_to_end_speedup=base["train_ms"] / total_re, order=order)
