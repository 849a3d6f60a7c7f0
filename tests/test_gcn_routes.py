"""Where a GCN training step takes its sparse products: the rule on the CPU, the fused kernels of each
route on the GPU."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from chunkedgreedy_b200 import gcn  # noqa: E402

ROWS = [1, 4096, 65_536, 131_071, 131_072, 1 << 20]


@pytest.mark.parametrize("in_dim", [4, 16, 64, 100, 128])
@pytest.mark.parametrize("hidden", [4, 16, 32, 64, 96, 128])
def test_no_route_moves_more_columns_than_the_plain_step(in_dim, hidden):
    # the plain step takes all four products at the hidden width
    for rows in ROWS:
        for classes in range(1, 129):
            for fused in (False, True):
                if fused and (classes > 48 or gcn.moved_columns(classes) > hidden):
                    continue
                widths = gcn.step_widths(rows, in_dim, hidden, classes, fused)
                assert all(gcn.moved_columns(w) <= gcn.moved_columns(hidden) for w in widths), (rows, classes, widths)
                assert widths[1] == widths[2] and (widths[1] >= classes or widths[1] == hidden)
                assert widths[3] in (in_dim, hidden)


def test_columns():
    for width in range(1, 300):
        assert width <= gcn.padded_columns(width) <= gcn.moved_columns(width)
    assert [gcn.padded_columns(w) for w in (1, 3, 7, 10, 16, 17, 18, 28, 30, 31, 32, 33, 47)] == [
        4, 4, 8, 16, 16, 17, 32, 32, 32, 31, 32, 33, 47]


def test_layers_with_hooks_and_other_layers_are_called():
    # a pre-hook that sets the weight (as weight normalisation does), a hook that sees the output, a layer
    # of another kind; sizes at which plain layers would have their weights taken out of them
    n = 1 << 17
    x = torch.randn((n, 4), generator=torch.Generator().manual_seed(0))
    op = lambda t: 0.5 * t  # noqa: E731 (stands for the sparse product)
    model = gcn.GCN(4, 64, 3)
    with torch.no_grad():
        want = op(torch.relu(op(model.w1(x)))) @ (2.0 * model.w2.weight).t() + model.w2.bias
        assert torch.allclose(model(x, op), op(torch.relu(op(model.w1(x)))) @ model.w2.weight.t() + model.w2.bias, atol=1e-5)
        weight, seen = model.w2.weight.clone(), []

        def set_weight(layer, value):
            layer.weight.copy_(value)

        pre = model.w2.register_forward_pre_hook(lambda m, _: set_weight(m, 2.0 * weight))
        post = model.w2.register_forward_hook(lambda m, i, o: seen.append(o.shape))
        assert torch.allclose(model(x, op), want, atol=1e-5) and seen == [(n, 3)]
        pre.remove()
        post.remove()
        model.w2 = torch.nn.Sequential(torch.nn.Linear(64, 8), torch.nn.ReLU(), torch.nn.Linear(8, 3))
        assert torch.allclose(model(x, op), model.w2(op(torch.relu(op(model.w1(x))))), atol=1e-5)


def test_logits_without_a_bias():
    model = gcn.GCN(4, 64, 3)
    model.w2.bias = None
    x = torch.randn((1 << 17, 4))
    z = model(x, lambda t: 0.5 * t)
    assert torch.allclose(z, 0.5 * torch.relu(0.5 * model.w1(x)) @ model.w2.weight.t(), atol=1e-5)
    z.sum().backward()
    assert model.w2.weight.grad.shape == (3, 64)


def _signs(model, x, op):
    """Which hidden units the model takes as positive.  One within a rounding of zero may fall on the other side in
    64 bits, and its whole gradient with it, so the reference below takes the model's own decisions."""
    from chunkedgreedy_b200 import Context, _lib
    w, b = model.w1.weight.detach(), model.w1.bias.detach()
    x = x.detach()
    if x.shape[1] > 128 or w.shape[0] > 128:
        return op(torch.nn.functional.linear(x, w, b)) > 0
    y = torch.empty((x.shape[0], w.shape[0]), device="cuda")
    torch.cuda.synchronize()
    ctx = Context()
    assert _lib.load().sporder_linear(ctx.handle, x.shape[0], x.shape[1], w.shape[0], x.data_ptr(), w.data_ptr(),
                                      b.data_ptr(), y.data_ptr()) == 0, _lib.last_error()
    torch.cuda.synchronize()
    ctx.close()
    return op(y) > 0


def _model_against_fp64(n, sizes, want_x):
    from chunkedgreedy_b200 import synth
    in_dim, hidden, classes = sizes
    if n == 1:
        ptr, ind = np.array([0, 1], dtype=np.int32), np.zeros(1, dtype=np.int32)
    else:
        ptr, ind, _ = synth.random_sparse(n, 3, 5, symmetric=True, hub_cols=2, hub_frac=0.2)
    dp, di = torch.from_numpy(ptr).cuda(), torch.from_numpy(ind).cuda()
    op = gcn.GraphOperator(dp, di, gcn.normalised_values(dp, di))
    torch.manual_seed(3)
    model = gcn.GCN(in_dim, hidden, classes).cuda()
    x = torch.randn((n, in_dim), device="cuda", requires_grad=want_x)
    target = torch.randn((n, classes), device="cuda")
    z = model(x, op)
    assert z.shape == (n, classes) and z.is_contiguous()
    (z * target).sum().backward()
    a = torch.sparse_csr_tensor(dp.long(), di.long(), op.val.double(), size=(n, n))
    wide = [p.detach().double().requires_grad_(True) for p in model.parameters()]
    xr = x.detach().double().requires_grad_(want_x)
    w1, b1, w2, b2 = wide
    zr = a @ ((a @ (xr @ w1.t() + b1)) * _signs(model, x, op)) @ w2.t() + b2
    (zr * target.double()).sum().backward()
    pairs = [(z, zr)] + [(p.grad, q.grad) for p, q in zip(model.parameters(), wide)]
    if want_x:
        pairs.append((x.grad, xr.grad))
    for got, want in pairs:
        # (the bound of the fused kernels' other tests: sums of n terms that largely cancel)
        assert float((got.detach().double() - want).norm()) <= 2e-5 * float(want.norm()) + 1e-6


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 31, 32, 33, 40_001, 131_073])
@pytest.mark.parametrize("sizes", [(128, 32, 17), (128, 32, 30), (100, 36, 9), (128, 64, 3), (128, 64, 48), (128, 128, 30),
                                   (100, 64, 47), (12, 8, 5), (128, 16, 7), (68, 4, 2), (128, 124, 33)])
def test_fused_routes_against_fp64(n, sizes):
    # op(D) at the hidden width where it is narrower than the inputs, padded logits, 17 to 32 classes
    _model_against_fp64(n, sizes, False)


@pytest.mark.gpu
@pytest.mark.parametrize("n,sizes", [(131_072, (300, 64, 10)), (131_072, (36, 256, 30)), (4096, (300, 64, 10)),
                                     (100_000, (128, 64, 13))])
@pytest.mark.parametrize("want_x", [False, True])
def test_library_products_behind_and_in_front(n, sizes, want_x):
    _model_against_fp64(n, sizes, want_x)


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 100, 5000])
@pytest.mark.parametrize("narrow,wide", [(1, 1), (3, 4), (17, 32), (48, 48)])
def test_pad_columns(n, narrow, wide):
    g = torch.randn((n, narrow), device="cuda")
    assert torch.equal(gcn._pad_columns(g, wide, None), torch.nn.functional.pad(g, (0, wide - narrow)))
    assert torch.equal(gcn._pad_columns(g.t().contiguous().t(), wide, None), torch.nn.functional.pad(g, (0, wide - narrow)))
