"""The library calls are torch.library custom operators: their fake implementations must give
the shapes and dtypes the real ones produce, so that torch.compile can trace through them
without a GPU in sight."""
import pytest
import torch
from torch._subclasses.fake_tensor import FakeTensorMode

from gemq_b200 import kernels as K

E, D, Fd, A = 8, 4096, 14336, 2


def fake_inputs():
    h, i32, i64 = torch.float16, torch.int32, torch.int64
    x = torch.empty(1, D, dtype=h)
    wq = torch.empty(256, Fd, dtype=i32)
    sz = torch.empty(32, Fd, dtype=h)
    meta = torch.empty(E, dtype=i32)
    idx = torch.empty(A, dtype=i64)
    return x, wq, sz, meta, idx


def test_every_op_is_registered():
    for name in ("dequant_gemv_rows", "dequant_splitk_gemv", "dequant_sel_splitk_gemv", "fused_dequant_up_proj",
                 "fused_dequant_down_proj", "dequant_gemm", "dequant_group_gemm", "moe_route", "moe_decode",
                 "moe_prefill", "moe_prefill_routed"):
        assert hasattr(torch.ops.gemq_b200, name), name


def test_fake_shapes_and_dtypes():
    with FakeTensorMode():
        x, wq, sz, meta, idx = fake_inputs()
        y = K.dequant_splitk_gemv(x, wq, sz, sz, 2, 128)
        assert y.shape == (1, Fd) and y.dtype == torch.float16
        y = K.dequant_sel_splitk_gemv(x, idx[:1], wq, sz, sz, meta, meta, 128)
        assert y.shape == (1, Fd)
        x1, x3 = K.fused_dequant_up_proj(x, idx, wq, wq, sz, sz, sz, sz, meta, meta, 128)
        assert x1.shape == x3.shape == (1, A * Fd) and x1.dtype == torch.float16
        w2 = torch.empty(Fd // 16, D, dtype=torch.int32)
        s2 = torch.empty(Fd // 128, D, dtype=torch.float16)
        x2 = K.fused_dequant_down_proj(x1, x3, idx, w2, s2, s2, meta, meta, 128)
        assert x2.shape == (1, A * D)
        for M, dt, want in ((7, torch.float16, torch.float16), (200, torch.float16, torch.float16),
                            (200, torch.bfloat16, torch.bfloat16)):
            y = K.dequant_gemm(torch.empty(M, D, dtype=dt), wq, sz, sz, 2, 128)
            assert y.shape == (M, Fd) and y.dtype == want
        y = K.dequant_group_gemm(torch.empty(50, D, dtype=torch.float16), idx, wq, sz, sz, meta, meta, meta, meta)
        assert y.shape == (A, 50, Fd) and y.dtype == torch.float16
        from gemq_b200.inference.moe_block import route_tokens
        w, i, logits = route_tokens(torch.empty(5, D, dtype=torch.bfloat16), torch.empty(E, D, dtype=torch.bfloat16), A, 1, True)
        assert w.shape == (5, A) and w.dtype == torch.bfloat16 and i.dtype == torch.int64 and logits.shape == (5, E)


def _scale_op():
    from gemq_b200.kernels._ops import library_op
    if not hasattr(_scale_op, "op"):
        @library_op("test_scale", lambda x, k: torch.empty_like(x))
        def test_scale(x: torch.Tensor, k: float) -> torch.Tensor:
            return x * k
        _scale_op.op = test_scale
    return _scale_op.op, torch.ops.gemq_b200.test_scale.default


@pytest.mark.parametrize("native", [True, False])
def test_direct_calls_leave_the_operator_what_is_its_own(native, monkeypatch):
    """Where someone looks at the call (autograd, a tracer, a function mode, forward-mode duals, function transforms)
    the call is the operator, with its refusals; under a default device and without gradients it is the function."""
    import torch.autograd.forward_ad as fw
    from torch.overrides import TorchFunctionMode
    from gemq_b200 import _capi
    from gemq_b200.kernels._ops import plain_call
    if not native:
        monkeypatch.setattr(_capi, "host", _capi._NoHost)
    else:
        assert _capi.host.plain(torch.ones(1), None, 3) is True
    call, op = _scale_op()
    x = torch.ones(3, 4)
    v = x.clone().requires_grad_()
    assert plain_call(x, 2.0, None) and not plain_call(v) and not plain_call(x, v)
    with torch.no_grad():
        assert plain_call(v) and not call(v, 2.0).requires_grad
    for f in (call, op):
        y = f(v, 2.0)
        with pytest.raises(RuntimeError, match="no autograd formula"):
            y.sum().backward()
        with pytest.raises(RuntimeError):
            torch.func.grad(lambda a: f(a, 2.0).sum())(x)
        assert "test_scale" in str(torch.jit.trace(lambda a: f(a, 2.0), x).graph)
        with fw.dual_level():
            assert fw.unpack_dual(f(fw.make_dual(x, torch.ones_like(x)), 2.0)).tangent is None
        assert torch.equal(torch.vmap(lambda a: f(a, 2.0))(x), 2 * x)
        seen = []

        class Watch(TorchFunctionMode):
            def __torch_function__(self, func, types, args=(), kwargs=None):
                seen.append(str(func))
                return func(*args, **(kwargs or {}))

        with Watch():
            f(x, 2.0)
        assert any("test_scale" in s for s in seen)
    with torch.device("cpu"):
        assert plain_call(x)


def test_quant_linear_keeps_the_gradient_of_its_bias(monkeypatch):
    """The bias is added outside the operator when it asks for a gradient, as in the plain expression."""
    from gemq_b200.inference import quant_linear as Q
    lin = Q.QuantLinear.__new__(Q.QuantLinear)
    torch.nn.Module.__init__(lin)
    lin.in_features, lin.out_features, lin.W_nbits, lin.group_size = 128, 32, 2, 128
    lin.W_q, lin.scales, lin.zeros = torch.zeros(8, 32, dtype=torch.int32), torch.zeros(1, 32), torch.zeros(1, 32)
    lin.bias = torch.nn.Parameter(torch.zeros(32))
    monkeypatch.setattr(Q, "host_linear", lambda *a: None)
    monkeypatch.setattr(Q, "quant_linear", lambda x, w, s, z, b, g, bias: x[:, :32] if bias is None else x[:, :32] + bias.detach())
    y = lin(torch.ones(2, 3, 128))
    y.sum().backward()
    assert torch.equal(lin.bias.grad, torch.full((32,), 6.0))
    with torch.no_grad():
        assert torch.equal(lin(torch.ones(2, 3, 128)), y)
