"""The dense layers' kernels (bias and ReLU, gradients of weight, bias and ReLU) against 64-bit products, and the
conditions under which a Linear is called as a module instead."""
import pytest
import torch
from torch import nn

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("n,n_in,n_out", [(1, 1, 1), (15, 3, 5), (64, 64, 64), (65, 192, 64), (1000, 128, 128), (4097, 130, 70),
                                          (20011, 64, 10), (3000, 68, 132), (777, 260, 12), (40000, 32, 128)])
@pytest.mark.parametrize("relu", [False, True])
@pytest.mark.parametrize("offset", [0, 1])
def test_dense_layer_against_64_bits(monkeypatch, n, n_in, n_out, relu, offset):
    """Sizes around the tiles of 64 and 128, one row, column counts that do not divide by four, operands off 16-byte
    alignment (offset)."""
    from fastgraphcompute_b200 import dense
    monkeypatch.setattr(dense, "min_rows", 1)
    torch.manual_seed(n + n_in)
    lin = nn.Linear(n_in, n_out).to(DEV)
    x = torch.randn(n * n_in + offset, device=DEV)[offset:].view(n, n_in).requires_grad_(True)
    g = torch.randn(n * n_out + offset, device=DEV)[offset:].view(n, n_out)
    out = dense.linear_relu(lin, nn.ReLU(), x) if relu else dense.linear(lin, x)
    assert type(out.grad_fn).__name__ == "_LinearBackward"
    grads = torch.autograd.grad(out, [x, lin.weight, lin.bias], g)
    again = torch.autograd.grad(dense.linear_relu(lin, nn.ReLU(), x) if relu else dense.linear(lin, x), [x, lin.weight, lin.bias], g)
    assert all(torch.equal(a, b) for a, b in zip(grads, again))          # fixed order of all sums
    xd, wd, bd, gd = x.detach().double(), lin.weight.detach().double(), lin.bias.detach().double(), g.double()
    y = xd @ wd.T + bd
    if relu:
        gd = torch.where(out.detach() <= 0, 0.0, gd)
        y = y.relu()
    # a sum of m products in fp32: every term is rounded at most m times, in practice a random walk
    eps = 2.0 ** -24

    def close(a, ref, mag, m):
        assert (a.double() - ref).abs().max() <= 4 * eps * (m ** 0.5 + 4) * mag.max() + 1e-30
    close(out.detach(), y, xd.abs() @ wd.abs().T + bd.abs(), n_in)
    close(grads[0], gd @ wd, gd.abs() @ wd.abs(), n_out)
    close(grads[1], gd.T @ xd, gd.abs().T @ xd.abs(), n)
    close(grads[2], gd.sum(0), gd.abs().sum(0), n)


def test_dense_layer_special_values_and_plain_calls(monkeypatch):
    from fastgraphcompute_b200 import dense
    lin = nn.Linear(8, 4).to(DEV)
    assert not dense.fused_ok(lin, torch.zeros((dense.min_rows - 1, 8), device=DEV))
    assert dense.fused_ok(lin, torch.zeros((dense.min_rows, 8), device=DEV))
    monkeypatch.setattr(dense, "min_rows", 1)
    relu = nn.ReLU()
    x = torch.randn((100, 8), device=DEV)
    x[3, 2], x[5, 1] = float("nan"), float("inf")
    xr = x.clone().requires_grad_(True)
    xm = x.clone().requires_grad_(True)
    out, ref = dense.linear_relu(lin, relu, xr), relu(lin(xm))
    torch.testing.assert_close(out, ref, rtol=1e-5, atol=1e-5, equal_nan=True)
    g = torch.randn_like(out)
    for a, b in zip(torch.autograd.grad(out, [xr, lin.weight], g), torch.autograd.grad(ref, [xm, lin.weight], g)):
        torch.testing.assert_close(a, b, rtol=1e-5, atol=1e-5, equal_nan=True)
    # a second derivative exists, as with the modules
    xs = torch.randn((50, 8), device=DEV, requires_grad=True)
    d, = torch.autograd.grad((dense.linear_relu(lin, relu, xs) ** 2).sum(), xs, create_graph=True)
    e, = torch.autograd.grad((relu(lin(xs)) ** 2).sum(), xs, create_graph=True)
    for p, q in zip(torch.autograd.grad(d.sum(), [xs, lin.weight]), torch.autograd.grad(e.sum(), [xs, lin.weight])):
        torch.testing.assert_close(p, q, rtol=1e-4, atol=1e-4)
    # called as modules: hooks, other activations, no bias, other types, autocast, empty input
    seen = []
    stack = nn.Sequential(nn.Linear(8, 8), nn.ReLU(), nn.Linear(8, 4), nn.Tanh()).to(DEV)
    torch.testing.assert_close(dense.sequential(stack, xs), stack(xs), rtol=1e-5, atol=1e-5)
    stack[2].register_forward_hook(lambda m, i, o: seen.append(o.shape))
    dense.sequential(stack, xs)
    assert seen == [(50, 4)]
    assert not dense.fused_ok(nn.Linear(8, 4, bias=False).to(DEV), xs)
    assert not dense.fused_ok(nn.Linear(8, 4).to(DEV).double(), xs.double())
    assert not dense.fused_ok(lin, torch.empty((0, 8), device=DEV)) and not dense.fused_ok(lin, xs.cpu())
    with torch.autocast("cuda", dtype=torch.bfloat16):
        assert not dense.fused_ok(lin, xs)
    assert not torch.vmap(lambda v: torch.tensor(float(dense.fused_ok(lin, v))))(xs[:, None, :]).any()


@pytest.mark.parametrize("strided", ["x", "weight", "both"])
@pytest.mark.parametrize("relu", [False, True])
def test_second_derivatives_through_strided_operands(monkeypatch, strided, relu):
    """A slice of columns as input and a transposed weight: the derivatives of the first derivatives are those of the modules.  Sums of up
    to 60 x 8 products of fp32 numbers of size 10 or so, each rounded a few times: 1e-4 of the largest."""
    from fastgraphcompute_b200 import dense
    monkeypatch.setattr(dense, "min_rows", 1)
    monkeypatch.setattr(dense, "_pays", lambda *a: True)
    torch.manual_seed(7)
    lin, act = nn.Linear(12, 8).to(DEV), nn.ReLU()
    if strided != "x":
        lin.weight = nn.Parameter(torch.randn((12, 8), device=DEV).t())
        assert not lin.weight.is_contiguous()
    wide = torch.randn((60, 20), device=DEV, requires_grad=True)

    def second(layer):
        x = wide[:, 3:15] if strided != "weight" else wide[:, :12].clone()
        out = layer(x)
        dx, dw = torch.autograd.grad((out ** 2).sum(), [x, lin.weight], create_graph=True)
        return out, torch.autograd.grad((dw ** 2).sum() + (dx ** 2).sum(), [wide, lin.weight])
    out, got = second(lambda x: dense.linear_relu(lin, act, x) if relu else dense.linear(lin, x))
    assert type(out.grad_fn).__name__ == "_LinearBackward"
    for a, b in zip(got, second(lambda x: act(lin(x)) if relu else lin(x))[1]):
        assert (a - b).abs().max() <= 1e-4 * b.abs().max()


def test_forward_mode_derivatives_of_dense_layers(monkeypatch):
    """An input that carries a tangent goes through the modules, which have forward-mode derivatives: as one layer, and
    where the tangent starts at an inner layer's weight."""
    import torch.autograd.forward_ad as fwad
    from fastgraphcompute_b200 import dense
    monkeypatch.setattr(dense, "min_rows", 1)
    torch.manual_seed(0)
    stack = nn.Sequential(nn.Linear(8, 16), nn.ReLU(), nn.Linear(16, 4)).to(DEV)
    x, t = torch.randn((100, 8), device=DEV), torch.randn((100, 8), device=DEV)
    with fwad.dual_level():
        got = fwad.unpack_dual(dense.sequential(stack, fwad.make_dual(x, t))).tangent
        ref = fwad.unpack_dual(stack(fwad.make_dual(x, t))).tangent
        assert torch.equal(got, ref)
        w = stack[0].weight.detach()
        del stack[0]._parameters["weight"]
        stack[0].weight = fwad.make_dual(w, torch.ones_like(w))
        got = fwad.unpack_dual(dense.sequential(stack, x)).tangent
        ref = fwad.unpack_dual(stack(x)).tangent
        assert ref is not None and torch.equal(got, ref)


@pytest.mark.parametrize("n,n_out", [(1, 1), (1, 4), (255, 4), (257, 12), (1000, 7), (20011, 64), (3, 4100), (300000, 33)])
@pytest.mark.parametrize("relu", [False, True])
@pytest.mark.parametrize("offset", [0, 1])
def test_bias_and_relu_pass(n, n_out, relu, offset):
    """One addition and one comparison per entry: the same bits as torch, on and off 16-byte alignment."""
    from fastgraphcompute_b200 import _cabi
    torch.manual_seed(n)
    y = torch.randn(n * n_out + offset, device=DEV)[offset:].view(n, n_out)
    bias = torch.randn(n_out + offset, device=DEV)[offset:]
    ref = y + bias
    ref = ref.relu() if relu else ref
    assert _cabi.lib.fgc_bias_act(_cabi.ptr(y), _cabi.ptr(bias), n, n_out, int(relu), _cabi.current_stream(y.device)) == 0
    assert torch.equal(y, ref)


def test_dense_layer_is_fused_only_where_it_pays():
    """Small weights, few outputs, weights of many tiles and forwards without a large result stay modules."""
    from fastgraphcompute_b200 import dense
    rows = dense.min_rows

    def fused(n, n_in, n_out, grad=True):
        lin = nn.Linear(n_in, n_out).to(DEV).requires_grad_(grad)
        out = dense.linear(lin, torch.zeros((n, n_in), device=DEV))
        assert type(out.grad_fn).__name__ == ("_LinearBackward" if out.grad_fn is not None and dense._pays(
            lin, torch.empty((n, n_in), device=DEV)) else ("AddmmBackward0" if grad else "NoneType"))
        return dense._pays(lin, torch.empty((n, n_in), device=DEV))
    assert fused(rows, 128, 64) and fused(rows, 64, 24) and fused(2 * rows, 128, 10) and fused(rows, 256, 256)
    assert not fused(rows, 128, 10) and not fused(4 * rows, 32, 16) and not fused(4 * rows, 64, 4)
    assert not fused(rows, 384, 160) and not fused(rows, 512, 512)
    assert fused(4 * rows, 64, 64, grad=False) and not fused(rows, 128, 128, grad=False)


@pytest.mark.parametrize("n,n_in,n_out", [(127, 63, 16), (128, 64, 17), (129, 65, 80), (148 * 128 + 1, 128, 129), (5000, 191, 96), (641, 193, 144),
                                          (300, 512, 40), (300, 513, 40), (300, 40, 513), (63, 128, 8), (148 * 64 + 1, 8, 128)])
def test_tensor_core_tiles_against_64_bits(monkeypatch, n, n_in, n_out):
    """Rows, sums and columns around the tiles of 64 and 128, several shares of the columns, sums too long for the tensor cores.  The
    three parts of a number hold all its bits and three of nine products are left out, 2^-24 of the result each at most: the bound
    is that of a sum in fp32 (test_dense_layer_against_64_bits)."""
    from fastgraphcompute_b200 import dense
    monkeypatch.setattr(dense, "min_rows", 1)
    torch.manual_seed(n + n_in)
    lin = nn.Linear(n_in, n_out).to(DEV)
    x = torch.randn((n, n_in), device=DEV).requires_grad_(True)
    g = torch.randn((n, n_out), device=DEV)
    out = dense._Linear.apply(x, lin.weight, lin.bias, True)
    grads = torch.autograd.grad(out, [x, lin.weight, lin.bias], g)
    xd, wd, bd = x.detach().double(), lin.weight.detach().double(), lin.bias.detach().double()
    gd = torch.where(out.detach() <= 0, 0.0, g.double())
    eps = 2.0 ** -24
    for a, ref, mag, m in ((out.detach(), (xd @ wd.T + bd).relu(), xd.abs() @ wd.abs().T + bd.abs(), n_in),
                           (grads[0], gd @ wd, gd.abs() @ wd.abs(), n_out), (grads[1], gd.T @ xd, gd.abs().T @ xd.abs(), n),
                           (grads[2], gd.sum(0), gd.abs().sum(0), n)):
        assert (a.double() - ref).abs().max() <= 4 * eps * (m ** 0.5 + 4) * mag.max() + 1e-30


@pytest.mark.parametrize("where", ["x", "weight", "gradient"])
@pytest.mark.parametrize("value", [2.0 ** 60, 3e38, float("inf"), float("nan"), 1e-30])
def test_numbers_that_are_not_split(monkeypatch, where, value):
    """Numbers beyond 2^60, infinities and NaN give what plain products give, in their rows and columns only; tiny ones keep their bits."""
    from fastgraphcompute_b200 import dense
    monkeypatch.setattr(dense, "min_rows", 1)
    torch.manual_seed(3)
    n, n_in, n_out = 1500, 72, 24
    lin = nn.Linear(n_in, n_out).to(DEV)
    x, g = torch.randn((n, n_in), device=DEV), torch.randn((n, n_out), device=DEV)
    with torch.no_grad():
        if where == "x":
            x[700] = 0.0
            x[700, 5] = value
        elif where == "weight":
            lin.weight[3] = 0.0
            lin.weight[3, 7] = value
        else:
            g[900] = 0.0
            g[900, 2] = value
    xa, xb = x.clone().requires_grad_(True), x.clone().requires_grad_(True)
    out, ref = dense._Linear.apply(xa, lin.weight, lin.bias, False), torch.addmm(lin.bias, xb, lin.weight.t())
    # (sums that cancel are compared against their largest terms: 72 or 24 of them, or 1500, of fp32 rounding)
    for a, b in zip((out,) + torch.autograd.grad(out, [xa, lin.weight], g), (ref,) + torch.autograd.grad(ref, [xb, lin.weight], g)):
        a, b = a.detach(), b.detach()
        odd = ~(torch.isfinite(b) & (b.abs() < 1e15))
        torch.testing.assert_close(a[odd], b[odd], rtol=1e-5, atol=0.0, equal_nan=True)
        torch.testing.assert_close(a[~odd], b[~odd], rtol=1e-4, atol=1e-4)
    if value == 1e-30 and where == "x":
        bias_free = (x[700].double() @ lin.weight.detach().double().t())
        own = torch.empty((n, n_out), device=DEV)
        from fastgraphcompute_b200 import _cabi
        assert _cabi.lib.fgc_dense_forward(_cabi.ptr(x), _cabi.ptr(lin.weight.detach()), None, n, n_in, n_out, 0, _cabi.ptr(own),
                                           _cabi.current_stream(x.device)) == 0
        torch.testing.assert_close(own[700].double(), bias_free, rtol=1e-6, atol=0.0)


@pytest.mark.parametrize("exponent", [-108, -112, -118, -122, -126, -135, -149, 42])
@pytest.mark.parametrize("where", ["x", "weight"])
def test_operands_keep_all_their_bits(exponent, where):
    """Numbers from fp32's smallest on, all of one matrix of that size, the other of a size that is still split and keeps the results above
    fp32's subnormals.  The operands are exact in both, so that only sums are rounded: of 40 or 24 products, or of 64 rows and then of five such
    sums, sixteen at a time -- at most nine additions, by 2^-23 of the sum of the products' sizes each -- and products of 2^-24 are left out."""
    from fastgraphcompute_b200 import _cabi
    torch.manual_seed(5)
    n, n_in, n_out, other = 300, 40, 24, min(max(-exponent - 20, -40), 38)
    small = torch.randn((n, n_in) if where == "x" else (n_out, n_in), device=DEV) * 2.0 ** (exponent / 2) * 2.0 ** (exponent - exponent / 2)
    large = torch.randn((n_out, n_in) if where == "x" else (n, n_in), device=DEV) * 2.0 ** other
    x, weight = (small, large) if where == "x" else (large, small)
    assert small.abs().max() > 0 and torch.isfinite(large).all()
    stream, lib, ptr = _cabi.current_stream(x.device), _cabi.lib, _cabi.ptr

    def close(a, ref, mag):
        assert ((a.double() - ref).abs() <= 20 * 2.0 ** -24 * mag + 2.0 ** -149).all()
    out = torch.empty((n, n_out), device=DEV)
    assert lib.fgc_dense_forward(ptr(x), ptr(weight), None, n, n_in, n_out, 0, ptr(out), stream) == 0
    close(out, x.double() @ weight.double().t(), x.double().abs() @ weight.double().abs().t())
    # x as a gradient of n_in outputs: dx = x @ weight^T, and dw = x^T @ (large or small numbers)
    turned, dx = weight.t().contiguous(), torch.empty((n, n_out), device=DEV)
    assert lib.fgc_dense_input_gradient(ptr(x), None, ptr(turned), n, n_out, n_in, ptr(dx), stream) == 0
    close(dx, x.double() @ turned.double(), x.double().abs() @ turned.double().abs())
    y = (torch.randn((n, n_out), device=DEV) * 2.0 ** (other if where == "x" else exponent)).contiguous()
    nbytes = lib.fgc_dense_backward_bytes(n, n_in, n_out)
    dw, db, ws = torch.empty((n_out, n_in), device=DEV), torch.empty((n_out,), device=DEV), torch.empty(nbytes, dtype=torch.uint8, device=DEV)
    assert lib.fgc_dense_backward(ptr(x), ptr(y), None, n, n_in, n_out, None, ptr(dw), ptr(db), ptr(ws), nbytes, stream) == 0
    close(dw, y.double().t() @ x.double(), y.double().abs().t() @ x.double().abs())


@pytest.mark.parametrize("n_in,n_out", [(72, 70), (67, 129), (64, 24)])
def test_numbers_that_are_not_split_in_some_columns(n_in, n_out):
    """Infinities and NaN in the first, a middle and the last column of the weight, in the last row of x and in the gradient: elsewhere
    the results are those without them, bit for bit; there they are those of plain products."""
    from fastgraphcompute_b200 import dense
    torch.manual_seed(n_in)
    n, inf, nan = 1000, float("inf"), float("nan")
    x, w, g = torch.randn((n, n_in), device=DEV), torch.randn((n_out, n_in), device=DEV), torch.randn((n, n_out), device=DEV)
    bias = torch.randn((n_out,), device=DEV)

    def passes(x, w, g):
        x, w = x.clone().requires_grad_(True), w.clone().requires_grad_(True)
        out = dense._Linear.apply(x, w, bias, False)
        return (out.detach(),) + torch.autograd.grad(out, [x, w], g)
    clean = passes(x, w, g)
    xs, ws, gs = x.clone(), w.clone(), g.clone()
    ws[0, 3], ws[n_out // 2, n_in - 1], ws[n_out - 1, 0] = inf, nan, -inf
    xs[n - 1, 5], xs[3, 0] = 2.0 ** 50, nan
    gs[700, 1], gs[701, n_out - 1] = -inf, nan
    out, dx, dw = passes(xs, ws, gs)
    refs = (torch.addmm(bias.double(), xs.double(), ws.double().t()), gs.double() @ ws.double(), gs.double().t() @ xs.double())
    touched = [torch.zeros_like(a, dtype=torch.bool) for a in (out, dx, dw)]
    touched[0][:, [0, n_out // 2, n_out - 1]] = touched[0][[n - 1, 3]] = True
    touched[1][:, [3, n_in - 1, 0]] = touched[1][[700, 701]] = True
    touched[2][:, [5, 0]] = touched[2][[1, n_out - 1]] = True
    for got, ref, was, odd in zip((out, dx, dw), refs, clean, touched):
        # (tiles of scalar operations round in another order than the tensor core: 1000 products of size 1)
        torch.testing.assert_close(got[~odd], was[~odd], rtol=1e-4, atol=1e-4)
        torch.testing.assert_close(got[odd].double(), ref[odd], rtol=1e-4, atol=1e-4, equal_nan=True)


@pytest.mark.parametrize("value", [float("nan"), float("inf")])
@pytest.mark.parametrize("where", ["weight", "x"])
def test_a_diverged_run_is_not_much_slower(value, where):
    """One such number in the weight, or such numbers everywhere in x: forward and backward take at most 25 times as long as without: NaN once,
    an infinity in the weight four times, infinities everywhere ten times measured, 65 to 110 times when every result was summed on its own."""
    from fastgraphcompute_b200 import dense
    n, n_in, n_out = 100000, 128, 128
    lin, x = nn.Linear(n_in, n_out).to(DEV), torch.randn((n, n_in), device=DEV, requires_grad=True)
    g = torch.randn((n, n_out), device=DEV)

    def time():
        best = float("inf")
        for _ in range(4):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            out = dense._Linear.apply(x, lin.weight, lin.bias, True)
            torch.autograd.grad(out, [x, lin.weight, lin.bias], g)
            b.record()
            b.synchronize()
            best = min(best, a.elapsed_time(b))
        return best
    plain = time()
    with torch.no_grad():
        if where == "x":
            x.fill_(value)
        else:
            lin.weight[3, 4] = value
    assert time() <= 25 * plain


@pytest.mark.parametrize("n_in,n_out", [(128, 128), (64, 64), (72, 40), (96, 200), (200, 24), (130, 70)])
@pytest.mark.parametrize("relu", [False, True])
def test_every_part_of_a_product_counts(n_in, n_out, relu):
    """One product per result, over several steps of many CTAs: nothing averages out.  Of the nine products of parts the three left out are below
    2^-25, 2^-25 and 2^-33 of the result, and what is added is rounded by 2^-24 a few times; a third part that is lost, or left from the step
    before, is 2^-17 and more."""
    from fastgraphcompute_b200 import _cabi
    lib, ptr, n = _cabi.lib, _cabi.ptr, 148 * 64 * 5 + 17
    gen = torch.Generator(device=DEV).manual_seed(n_in)
    stream, rnd = _cabi.current_stream(torch.device(DEV)), lambda *size: torch.randn(size, generator=gen, device=DEV)
    weight, rows = rnd(n_out, n_in), torch.arange(n, device=DEV)
    y = torch.where(rnd(n, n_out) < 0, 0.0, 1.0) if relu else None

    def close(got, ref):
        assert ((got.double() - ref).abs() <= 4 * 2.0 ** -24 * ref.abs()).all()
    # forward: one number a row of x
    x, col, v = torch.zeros((n, n_in), device=DEV), torch.randint(0, n_in, (n,), generator=gen, device=DEV), rnd(n)
    x[rows, col] = v
    out = torch.empty((n, n_out), device=DEV)
    assert lib.fgc_dense_forward(ptr(x), ptr(weight), None, n, n_in, n_out, int(relu), ptr(out), stream) == 0
    ref = v.double()[:, None] * weight.t()[col].double()
    close(out, ref.relu() if relu else ref)
    # input gradient: one number a row of dy
    dy, col = torch.zeros((n, n_out), device=DEV), torch.randint(0, n_out, (n,), generator=gen, device=DEV)
    dy[rows, col] = v
    passes = torch.ones(n, device=DEV) if y is None else y[rows, col]
    dx = torch.empty((n, n_in), device=DEV)
    assert lib.fgc_dense_input_gradient(ptr(dy), ptr(y), ptr(weight), n, n_in, n_out, ptr(dx), stream) == 0
    close(dx, (v * passes).double()[:, None] * weight[col].double())
    # weight gradient: a dense x, one row of dy for every output
    x = rnd(n, n_in)
    nbytes = lib.fgc_dense_backward_bytes(n, n_in, n_out)
    dw, db, ws = torch.empty((n_out, n_in), device=DEV), torch.empty((n_out,), device=DEV), torch.empty(nbytes, dtype=torch.uint8, device=DEV)
    for _ in range(6):
        row, outputs, g = torch.randperm(n, generator=gen, device=DEV)[:n_out], torch.arange(n_out, device=DEV), rnd(n_out)
        dy.zero_()
        dy[row, outputs] = g
        passes = torch.ones(n_out, device=DEV) if y is None else y[row, outputs]
        assert lib.fgc_dense_backward(ptr(x), ptr(dy), ptr(y), n, n_in, n_out, None, ptr(dw), ptr(db), ptr(ws), nbytes, stream) == 0
        close(dw, (g * passes).double()[:, None] * x[row].double())
        assert torch.equal(db, g * passes)
