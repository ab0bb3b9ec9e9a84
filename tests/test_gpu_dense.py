"""Dense products of the layers (yitu_linear_f32, yitu_gram_f32) on the GPU against 64-bit products, at the borders of every
tile, with strided and misaligned operands, and through the modules that use them."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _bound(terms, abs_product):
    """A float32 sum of `terms` products, in any order: each result carries at most `terms` + 1 roundings of 2^-24 (one per
    multiply-add, one more for the bias or a rounded partial sum), relative to the sum of the absolute products."""
    return (terms + 2) * 2.0 ** -24 * abs_product + 1e-37


def _strided(rows, cols, layout, gen):
    if layout == "plain":
        return torch.randn(rows, cols, device="cuda", generator=gen)
    pad, shift = {"padded": (4, 0), "odd": (3, 1)}[layout]
    flat = torch.randn(rows * (cols + pad) + 8, device="cuda", generator=gen)
    return flat[shift:shift + rows * (cols + pad)].view(rows, cols + pad)[:, :cols]


@pytest.mark.parametrize("layout", ["plain", "padded", "odd"])
@pytest.mark.parametrize("n,K,N", [(1, 1, 1), (5, 3, 7), (31, 16, 8), (33, 17, 9), (127, 64, 16), (129, 15, 17), (300, 100, 32), (257, 41, 33),
                                   (40001, 64, 64), (40001, 65, 65), (80003, 33, 4), (77001, 12, 15), (50021, 20, 31), (20011, 128, 129),
                                   (3001, 500, 16)])
def test_matmul_and_gram(n, K, N, layout):
    from yitu_b200 import ops
    gen = torch.Generator(device="cuda")
    gen.manual_seed(n + K * 7 + N)
    a, g = _strided(n, K, layout, gen), _strided(n, N, layout, gen)
    w, wt = _strided(N, K, layout, gen), _strided(K, N, layout, gen)
    bias = torch.randn(N, device="cuda", generator=gen)
    from yitu_b200._lib import check, lib

    def linear(b, b_t, bias):
        out = torch.full((n, N + 1), 7.0, device="cuda")
        check(lib().yitu_linear_f32(n, K, N, a.data_ptr(), a.stride(0), b.data_ptr(), b.stride(0), int(b_t),
                                    None if bias is None else bias.data_ptr(), out.data_ptr(), N + 1, ops._stream(a.device)))
        assert bool((out[:, N] == 7.0).all())
        return out[:, :N]

    ad = a.double()
    for b, b_t, got in ((w.t(), True, linear(w, True, bias)), (wt, False, linear(wt, False, None)),
                        (w.t(), True, ops.matmul(a, w, b_transposed=True, bias=bias)), (wt, False, ops.matmul(a, wt))):
        add = bias.double() if b_t else 0.0
        err = (got.double() - (ad @ b.double() + add)).abs()
        assert bool((err <= _bound(K, ad.abs() @ b.double().abs() + (bias.double().abs() if b_t else 0.0))).all())
    # the rows are split over the grid: no result is a chain of more than 512 additions at these sizes (rows of a split and
    # group, groups, splits), where a bound by the number of rows would let whole stages of rows go missing
    for x, y in ((g, a), (a, g)):
        c, s = ops.gram(x, y, sums=True)
        assert c.shape == (x.size(1), y.size(1))
        assert bool(((c.double() - x.double().t() @ y.double()).abs() <= _bound(min(n, 512), x.double().abs().t() @ y.double().abs())).all())
        assert bool(((s.double() - x.double().sum(0)).abs() <= _bound(min(n, 512), x.double().abs().sum(0))).all())
        c2, s2 = ops.gram(x, y, sums=True)
        assert torch.equal(c, c2) and torch.equal(s, s2), "the sums are formed in a fixed order"
        assert ops.gram(x, y)[1] is None


def test_empty_and_refused_operands():
    from yitu_b200 import ops
    w = torch.randn(8, 16, device="cuda")
    assert ops.matmul(torch.empty(0, 16, device="cuda"), w, b_transposed=True).shape == (0, 8)
    c, s = ops.gram(torch.empty(0, 4, device="cuda"), torch.empty(0, 8, device="cuda"), sums=True)
    assert c.shape == (4, 8) and float(c.abs().max()) == 0.0 and float(s.abs().max()) == 0.0
    with pytest.raises(RuntimeError):
        ops.matmul(torch.randn(4, 5, device="cuda"), w, b_transposed=True)
    # other types take the library's product and keep their type
    assert ops.matmul(torch.randn(4, 16, device="cuda").half(), w.half(), b_transposed=True).dtype == torch.float16
    # a program that allows TF32, by the older or the newer switch, keeps the library's product
    assert ops._dense_kernels_apply(w, w)
    for allow, back in ((lambda: torch.set_float32_matmul_precision("high"), lambda: torch.set_float32_matmul_precision("highest")),
                        (lambda: setattr(torch.backends.cuda.matmul, "fp32_precision", "tf32"),
                         lambda: setattr(torch.backends.cuda.matmul, "fp32_precision", "ieee"))):
        allow()
        try:
            assert not ops._dense_kernels_apply(w, w)
            assert ops.matmul(torch.randn(4, 16, device="cuda"), w, b_transposed=True).shape == (4, 8)
        finally:
            back()
    assert ops._dense_kernels_apply(w, w)
    # what autograd records stays recorded
    wr = w.clone().requires_grad_(True)
    assert ops.matmul(torch.randn(4, 16, device="cuda"), wr, b_transposed=True).requires_grad


@pytest.mark.parametrize("layout", ["plain", "odd", "expanded"])
def test_linear_module_gradients(layout):
    """nn.Linear's results, gradients and gradients of gradients, with inputs and output gradients of any stride."""
    from yitu_b200.nn.layers import Linear
    gen = torch.Generator(device="cuda")
    gen.manual_seed(3)
    n, K, N = 2053, 36, 20
    lin = Linear(K, N).cuda()
    x = (torch.randn(1, K, device="cuda", generator=gen).expand(n, K) if layout == "expanded" else _strided(n, K, layout, gen))
    x = x.detach().requires_grad_(True)
    g = _strided(n, N, "odd" if layout == "odd" else "plain", gen)
    if layout == "expanded":
        g = torch.ones(1, 1, device="cuda").expand(n, N)
    params = [x, lin.weight, lin.bias]
    out = lin(x)
    grads = torch.autograd.grad(out, params, g)
    ref_in = [p.detach().double().requires_grad_(True) for p in params]
    ref_out = torch.nn.functional.linear(*ref_in)
    refs = torch.autograd.grad(ref_out, ref_in, g.double())
    for got, ref, terms in zip([out, *grads], [ref_out, *refs], (K, N, n, n)):
        scale = float(ref.detach().abs().max()) + 1.0
        assert float((got.double() - ref).abs().max()) <= (terms + 2) * 2.0 ** -24 * 8 * scale
    # a gradient of a gradient: d/dW of sum(dx) is the column sums of g, for every input feature
    if layout == "plain":
        dx, = torch.autograd.grad(lin(x), [x], g, create_graph=True)
        dw, = torch.autograd.grad(dx.sum(), [lin.weight])
        ref = g.double().sum(0)[:, None].expand(N, K)
        assert float((dw.double() - ref).abs().max()) <= (n + 2) * 2.0 ** -24 * float(g.abs().sum(0).max())
    assert lin(torch.randn(3, 4, K, device="cuda")).shape == (3, 4, N)
    with torch.autocast("cuda", dtype=torch.bfloat16):
        assert lin(x.detach()).dtype == torch.bfloat16


def test_first_layer_skips_the_input_gradient():
    """GCNConv / GINConv: the weight gradient does not depend on whether the input gradient is asked for."""
    from types import SimpleNamespace
    from yitu_b200 import graphs
    from yitu_b200.nn import GCNConv, GINConv
    n = 600
    src, dst = graphs.rmat_edges(3, n, n, 5000, device="cuda")
    indptr, indices = graphs.csr_by_destination(src, dst, n, n, self_loops=True)
    one = torch.zeros(1, dtype=torch.int32, device="cuda")
    info = SimpleNamespace(row_pointers=indptr, column_index=indices, degrees=graphs.in_degrees(indptr).clamp(min=1).rsqrt(), partPtr=one,
                           part2Node=one, partSize=32, dimWorker=32, warpPerBlock=4)
    for conv in (GCNConv(24, 12).cuda(), GINConv(24, 12).cuda()):
        x = torch.randn(n, 24, device="cuda")
        gw, = torch.autograd.grad(conv(x, info).square().sum(), [conv.weights])
        xr = x.clone().requires_grad_(True)
        gx, gw2 = torch.autograd.grad(conv(xr, info).square().sum(), [xr, conv.weights])
        assert torch.equal(gw, gw2) and gx.shape == x.shape and float(gx.abs().max()) > 0
        conv.weights.requires_grad_(False)
        gx2, = torch.autograd.grad(conv(xr, info).square().sum(), [xr])
        assert torch.equal(gx, gx2)


@pytest.mark.parametrize("M,N", [(5, 12), (16, 64), (33, 40), (64, 64), (100, 128), (80, 9)])
def test_column_sums_with_infinite_values(M, N):
    """Infinite, overflowing and undefined columns end as they do in torch.sum; the others do not see them."""
    from yitu_b200 import ops
    gen = torch.Generator(device="cuda")
    gen.manual_seed(M)
    n = 20011
    g, x = torch.randn(n, M, device="cuda", generator=gen), torch.randn(n, N, device="cuda", generator=gen)
    clean = ops.gram(g, x, sums=True)[1]
    g[7000, 0] = float("inf")
    g[0, 1] = -float("inf")
    g[n - 1, 1] = float("inf")
    g[11, 2] = float("nan")
    g[:40, 3] = 3e38
    sums = ops.gram(g, x, sums=True)[1]
    assert float(sums[0]) == float("inf") and bool(torch.isnan(sums[1:3]).all()) and float(sums[3]) == float("inf")
    assert torch.equal(sums[4:], clean[4:])


def test_linear_saves_what_its_backward_reads():
    """As with torch's own product, a weight whose input needs no gradient may be updated before the backward pass, and so may
    the input of a frozen weight."""
    from yitu_b200.nn.layers import Linear
    lin, x, g = Linear(24, 12).cuda(), torch.randn(500, 24, device="cuda"), torch.randn(500, 12, device="cuda")
    want = g.t() @ x
    out = lin(x)
    with torch.no_grad():
        lin.weight.zero_()
    gw, gb = torch.autograd.grad(out, [lin.weight, lin.bias], g)
    assert float((gw - want).abs().max()) <= 1e-4 * float(want.abs().max())
    lin.weight.requires_grad_(False)
    with torch.no_grad():
        lin.weight.normal_()
    leaf = torch.randn(500, 24, device="cuda", requires_grad=True)
    x = leaf * 2
    out = lin(x)
    x.data.zero_()
    with torch.no_grad():
        x.add_(1.0)
    gx, gb = torch.autograd.grad(out, [leaf, lin.bias], g)
    assert float((gx - 2 * g @ lin.weight).abs().max()) <= 1e-4 * float(gx.abs().max())


def test_linear_is_seen_by_tracers_and_dispatch_modes():
    """A traced or counted Linear is nn.Linear's product, not a constant of the example input."""
    from torch.fx.experimental.proxy_tensor import make_fx
    from torch.utils.flop_counter import FlopCounterMode
    from yitu_b200.nn.layers import Linear
    lin = Linear(24, 12).cuda().requires_grad_(False)
    x, y = torch.randn(50, 24, device="cuda"), torch.randn(50, 24, device="cuda")
    want = torch.nn.functional.linear(y, lin.weight, lin.bias)
    compiled = torch.compile(lin, backend="eager", fullgraph=True)
    for f in (make_fx(lin)(x), torch.jit.trace(lin, x), compiled):
        assert float((f(y) - want).abs().max()) <= 1e-5 * float(want.abs().max())
    with FlopCounterMode(display=False) as counter:
        lin(x)
    assert counter.get_total_flops() == 2 * 50 * 24 * 12


@pytest.mark.parametrize("M,N", [(4, 64), (8, 64), (16, 16), (64, 12), (40, 64)])
def test_column_sums_are_rounded_once_per_split(M, N):
    """Columns that cancel.  Rounded are the splits' sums and the result, each by 2^-24 * 0.58 of its size (rms), and the sizes
    are those of random walks of n steps in all: 2^-24 * 0.58 * sqrt(2 n), where a chain over a split's 128 threads adds four
    times that."""
    from yitu_b200 import ops
    n, err = 100003, []
    for seed in range(8):
        gen = torch.Generator(device="cuda")
        gen.manual_seed(seed)
        g, x = torch.randn(n, M, device="cuda", generator=gen), torch.randn(n, N, device="cuda", generator=gen)
        err.append(ops.gram(g, x, sums=True)[1].double() - g.double().sum(0))
    assert float(torch.stack(err).square().mean().sqrt()) <= 1.5 * 2.0 ** -24 * 0.58 * (2 * n) ** 0.5


@pytest.mark.parametrize("layout", ["plain", "odd"])
@pytest.mark.parametrize("n,M,N", [(1, 3, 5), (63, 8, 64), (64, 9, 64), (65, 16, 65), (257, 33, 41), (4096, 64, 64), (4099, 64, 65), (18943, 12, 300),
                                   (20011, 128, 129), (40001, 64, 64), (40031, 65, 7), (80003, 4, 33), (75777, 32, 96), (151553, 8, 16)])
def test_gram_counts_every_row_once(n, M, N, layout):
    """Whole numbers whose sums stay below 2^24: the result is exact, so a row left out or counted twice at the border of a
    stage, a group or a split shows."""
    from yitu_b200 import ops
    gen = torch.Generator(device="cuda")
    gen.manual_seed(n)
    a, b = (_strided(n, w, layout, gen) for w in (M, N))
    for t in (a, b):
        t.copy_(torch.randint(-3, 4, t.shape, device="cuda", generator=gen))
    for x, y in ((a, b), (b, a)):
        c, s = ops.gram(x, y, sums=True)
        assert torch.equal(c.double(), x.double().t() @ y.double()) and torch.equal(s.double(), x.double().sum(0))


@pytest.mark.parametrize("n", [100, 511, 512, 1499, 1500, 2048, 4096, 4097])
@pytest.mark.parametrize("K,N", [(32, 64), (33, 64), (64, 17), (65, 64), (128, 64), (128, 128), (129, 16), (129, 17), (256, 128), (256, 129),
                                 (257, 16), (512, 16), (513, 8), (1024, 16), (1025, 8), (1433, 41), (64, 65), (8, 4096)])
def test_products_at_the_borders_of_the_dispatch(n, K, N):
    """Own kernel or library, with and without a bias: the same product within the rounding of a sum of its length."""
    from yitu_b200 import ops
    gen = torch.Generator(device="cuda")
    gen.manual_seed(n + K + N)
    a, w, bias = (torch.randn(*s, device="cuda", generator=gen) for s in ((n, K), (N, K), (N,)))
    exact, size = a.double() @ w.double().t(), a.double().abs() @ w.double().abs().t()
    for got, add in ((ops.matmul(a, w, b_transposed=True, bias=bias), bias), (ops.matmul(a, w, b_transposed=True), None),
                     (ops.matmul(a, w.t().contiguous()), None)):
        ref, scale = (exact, size) if add is None else (exact + add.double(), size + add.double().abs())
        assert bool(((got.double() - ref).abs() <= _bound(K, scale)).all())
    g = torch.randn(n, N, device="cuda", generator=gen)
    for sums in (False, True):
        c, s = ops.gram(g, a, sums=sums)
        assert bool(((c.double() - g.double().t() @ a.double()).abs() <= _bound(n, g.double().abs().t() @ a.double().abs())).all())
        assert s is None if not sums else bool(((s.double() - g.double().sum(0)).abs() <= _bound(n, g.double().abs().sum(0))).all())
