"""torch.nn.Linear (and a ReLU behind it) with this library's kernels.

The modules stay what they are -- parameters, names, hooks, activation -- and are called as
usual wherever the plain form is not given: see ``_plain_linear`` and ``fused_ok``.
"""
import torch
from torch import nn
from torch.autograd import forward_ad

from . import _cabi

# Fewer rows: launches outweigh most of what is saved.  Forward and backward with ReLU, modules / own kernels, us: 32 768 rows, 64 to 64 171 / 134, 128 to
# 128 247 / 133, 64 to 24 154 / 133; 16 384 rows 164 / 146, 141 / 133 and 137 / 133, but 256 to 256 259 / 137.  (Drawn with scalar kernels; these
# are ahead on both sides of it.)
min_rows = 32768

# Sums over more columns (FGC_DENSE_MAX_SUM) stay with the library.
max_sum = 512

# Products from the library: results of this many entries or more get bias and ReLU in a pass of their own: the library's product with the bias in
# it is then slower than the plain product and the pass (forward alone, module / pass, us: 200 000 rows, 64 to 128
# without ReLU 230 / 160, with it 264 / 161; 131 072 rows, 128 to 64 98 / 95 and 106 / 96).  Below, the pass and its
# launch cost more than they save (200 000 rows, 128 to 10 85 / 91; 32 768 rows, 128 to 128 59 / 64).
pass_from = 1 << 23
# Forward alone, module with ReLU / own kernel, us: 66 000 rows, 128 to 64 71 / 45; 64 to 128 92 / 46; 100 000 rows, 128 to 64 91 / 52; several
# shares of the columns, 200 000 rows: 256 to 256 789 / 246, 512 to 128 636 / 461, 512 to 512 2381 / 1825; 16 384 rows, 512 to 512 217 / 168.
# (Ahead below it too, 32 768 rows, 128 to 128 50 / 21: not measured to its edge.)
forward_from = (1 << 22) + 1


class _Linear(torch.autograd.Function):
    """act(x @ weight^T + bias) on the tensor cores at fp32 accuracy, forward and gradients (csrc/dense.cu); products that sum over
    more than max_sum columns from the library, with bias and ReLU in one pass over a large result."""

    @staticmethod
    def forward(ctx, x, weight, bias, relu):
        if max_sum >= x.shape[1]:
            # (a copy is the kernel's alone: what is saved below are the inputs, which second derivatives go through)
            rows, columns = x.contiguous(), weight.contiguous()
            y = torch.empty((x.shape[0], weight.shape[0]), dtype=torch.float32, device=x.device)
            with _cabi.on_device(x.device):
                _cabi.check(_cabi.lib.fgc_dense_forward(
                    _cabi.ptr(rows), _cabi.ptr(columns), _cabi.ptr(bias.contiguous()), x.shape[0], x.shape[1], weight.shape[0], int(relu),
                    _cabi.ptr(y), _cabi.current_stream(x.device)), "fgc_dense_forward")
        elif x.shape[0] * weight.shape[0] < pass_from:
            y = torch.addmm(bias, x, weight.t())
            if relu:
                y.relu_()
        else:
            y = torch.mm(x, weight.t())
            with _cabi.on_device(x.device):
                _cabi.check(_cabi.lib.fgc_bias_act(_cabi.ptr(y), _cabi.ptr(bias.contiguous()), y.shape[0], y.shape[1],
                                                   int(relu), _cabi.current_stream(x.device)), "fgc_bias_act")
        ctx.save_for_backward(x, weight, y if relu else None)
        return y

    @staticmethod
    def backward(ctx, dy):
        x, weight, y = ctx.saved_tensors
        need_x, need_w, need_b, _ = ctx.needs_input_grad
        if torch.is_grad_enabled() or not (need_w or need_b):
            # differentiable again (create_graph), or nothing but the input gradient wanted
            if y is not None:
                dy = torch.where(y <= 0, 0.0, dy)
            return (dy @ weight if need_x else None, dy.t() @ x if need_w else None, dy.sum(0) if need_b else None, None)
        x, dy = x.contiguous(), dy.contiguous()
        n, n_in = x.shape
        n_out = dy.shape[1]
        own = need_x and n_out <= max_sum                        # (else the library's product, of the masked gradient)
        masked = torch.empty_like(dy) if y is not None and need_x and not own else None
        dw = torch.empty((n_out, n_in), dtype=torch.float32, device=x.device)
        db = torch.empty((n_out,), dtype=torch.float32, device=x.device)
        nbytes = _cabi.lib.fgc_dense_backward_bytes(n, n_in, n_out)
        ws = torch.empty(nbytes, dtype=torch.uint8, device=x.device)
        with _cabi.on_device(x.device):
            _cabi.check(_cabi.lib.fgc_dense_backward(
                _cabi.ptr(x), _cabi.ptr(dy), _cabi.ptr(y), n, n_in, n_out, _cabi.ptr(masked), _cabi.ptr(dw), _cabi.ptr(db),
                _cabi.ptr(ws), nbytes, _cabi.current_stream(x.device)), "fgc_dense_backward")
        dx = None
        if own:
            dx = torch.empty_like(x)
            weight = weight.contiguous()
            with _cabi.on_device(x.device):
                _cabi.check(_cabi.lib.fgc_dense_input_gradient(
                    _cabi.ptr(dy), _cabi.ptr(y), _cabi.ptr(weight), n, n_in, n_out, _cabi.ptr(dx), _cabi.current_stream(x.device)),
                    "fgc_dense_input_gradient")
        elif need_x:
            dx = torch.mm(dy if masked is None else masked, weight)
        return dx, dw if need_w else None, db if need_b else None, None


def _no_hooks(m: nn.Module) -> bool:
    return not (m._forward_hooks or m._forward_pre_hooks or m._backward_hooks or m._backward_pre_hooks)


def _plain_linear(m) -> bool:
    return (type(m) is nn.Linear and _no_hooks(m) and "forward" not in m.__dict__ and type(m.weight) is nn.Parameter
            and type(m.bias) is nn.Parameter)


def _full_precision() -> bool:
    try:
        return torch.get_float32_matmul_precision() == "highest"
    except RuntimeError:        # set through the per-backend switches: leave it to the library
        return False


def _traced() -> bool:
    """Asked before any look at a shape: a tracer would record the comparison of the row count with a threshold as a
    condition on a dynamic size (an export then fails, a compiled module gets a second graph)."""
    return torch.jit.is_tracing() or torch.compiler.is_compiling() or torch._C._are_functorch_transforms_active()


def fused_ok(linear, x) -> bool:
    """Whether ``linear(x)`` may take the fused form: plain fp32 matrices on one GPU, fp32 arithmetic asked
    for, no hooks and no tracing that would have to see the module called."""
    if _traced() or type(x) is not torch.Tensor or x.dim() != 2 or x.shape[0] < min_rows:
        return False
    if nn.modules.module._has_any_global_hook() or not _plain_linear(linear):
        return False
    if forward_ad.unpack_dual(x).tangent is not None:        # forward-mode derivatives: the modules have them
        return False
    w = linear.weight
    return (x.is_cuda and x.shape[0] > 0 and x.dtype == torch.float32 and w.dtype == torch.float32
            and linear.bias.dtype == torch.float32 and w.device == x.device and linear.bias.device == x.device
            and x.shape[1] == w.shape[1] and max(w.shape) <= 65535 and min(w.shape) > 0
            and not torch.is_autocast_enabled("cuda") and _full_precision())


def _pays(linear, x) -> bool:
    """Whether the fused form is the faster one of those that ``fused_ok`` allows (B200, forward and backward, modules /
    fused, us)."""
    if _traced() or type(linear) is not nn.Linear or x.dim() != 2 or x.shape[0] < min_rows:
        return False
    n, n_in, n_out = x.shape[0], linear.in_features, linear.out_features
    if not (torch.is_grad_enabled() and (x.requires_grad or linear.weight.requires_grad)):
        return n * n_out >= (forward_from if n_in <= max_sum else pass_from)           # nothing but the forward to gain
    # A small weight: the library's product for its gradient is a good one, and little is gained: 200 000 rows, 32 to 16 158 / 134, 65 536
    # rows 137 / 133, but 32 to 32 657 / 134.
    if n_in * n_out < min_rows // 32:
        return False
    # Few outputs fill a part of a tile, which takes twice the rows to gain from: 128 to 10 at 32 768 rows 133 / 132, at
    # 65 536 156 / 133; 64 to 24 at 32 768 154 / 133.
    if n_out < 24 and (n + 1) // 2 < min_rows:
        return False
    # Many tiles of a weight read x and the gradient again and again, and gain less: 200 000 rows, 256 to 256 2106 / 840, 512 to 128 2026 /
    # 1004, 384 to 160 2155 / 1034, 512 to 512 6550 / 4909.  (Drawn with scalar kernels, which lost on the last two.)
    return _padded(n_in) * _padded(n_out) <= 65536


def _padded(columns: int) -> int:
    return 64 if columns <= 64 else -(-columns // 128) * 128


def linear_relu(linear: nn.Module, relu: nn.Module, x: torch.Tensor) -> torch.Tensor:
    """relu(linear(x))."""
    if type(relu) is nn.ReLU and _no_hooks(relu) and "forward" not in relu.__dict__ and _pays(linear, x) \
            and fused_ok(linear, x):
        return _Linear.apply(x, linear.weight, linear.bias, True)
    return relu(linear(x))


def linear(module: nn.Module, x: torch.Tensor) -> torch.Tensor:
    """module(x)."""
    if _pays(module, x) and fused_ok(module, x):
        return _Linear.apply(x, module.weight, module.bias, False)
    return module(x)


def sequential(stack: nn.Module, x: torch.Tensor) -> torch.Tensor:
    """stack(x), every plain Linear (with the ReLU behind it, if there is one) in the fused form."""
    if type(stack) is not nn.Sequential or not _no_hooks(stack) or "forward" in stack.__dict__:
        return stack(x)
    modules = list(stack)
    i = 0
    while i < len(modules):
        m = modules[i]
        if type(m) is nn.Linear and i + 1 < len(modules) and type(modules[i + 1]) is nn.ReLU:
            x = linear_relu(m, modules[i + 1], x)
            i += 2
        else:
            x = linear(m, x) if type(m) is nn.Linear else m(x)
            i += 1
    return x
