"""Which calls of the prefill model take the fused norm and norm + rotary kernels: those that give what the torch expressions
give, and no others (tensors or norms that something watches, replaces or transforms stay with torch)."""
import pytest
import torch
from torch import nn
from torch.autograd import forward_ad

GPU = pytest.mark.gpu


def _norm(K, device, eps=1e-6):
    from fp8_inference_toolkit_b200.qwen3 import RMSNorm

    m = RMSNorm(K, eps, device)
    m.weight.data.copy_(torch.linspace(0.5, 1.5, K))
    return m


def _expression(x, weight, eps):
    xf = x.float()
    return (xf * torch.rsqrt(xf.pow(2).mean(-1, keepdim=True) + eps)).to(x.dtype) * weight


def _close(a, b):
    # one bf16 step of either rounding (2^-8 each), the sum of squares being added in another order
    return ((a.float() - b.float()).abs() <= 2.0 ** -7 * b.float().abs()).all()


def _x(*shape):
    return torch.randn(*shape, device="cuda", generator=torch.Generator(device="cuda").manual_seed(3)).to(torch.bfloat16)


@pytest.fixture
def calls(monkeypatch):
    """Counts the calls of the two kernels."""
    from fp8_inference_toolkit_b200 import ops

    n = {"rmsnorm": 0, "qk_norm_rope_": 0}

    def counted(name, op):
        def call(*a):
            n[name] += 1
            return op(*a)
        return call

    for name in n:
        monkeypatch.setattr(ops, name, counted(name, getattr(ops, name)))
    return n


@GPU
@pytest.mark.parametrize("K", [1024, 16384])
def test_plain_rows_take_the_kernel(K, calls):
    x, m = _x(3, 5, K), _norm(K, "cuda")
    assert _close(m(x), _expression(x, m.weight, m.eps)) and calls["rmsnorm"] == 1
    with torch.device("cuda"):      # a default device is no reason to leave it
        m(x)
    assert calls["rmsnorm"] == 2


@GPU
@pytest.mark.parametrize("case", ["strided", "short", "long", "half", "misaligned input", "misaligned weight", "broadcast weight",
                                  "negative view", "scalar"])
def test_other_tensors_keep_the_expression(case, calls):
    K = {"short": 1016, "long": 16392, "scalar": 1}.get(case, 1024)
    x, m = _x(4, K), _norm(K, "cuda")
    if case == "strided":
        x = _x(K, 4).t()
    elif case == "half":
        x, m = x.half(), m.half()
    elif case == "misaligned input":
        x = _x(4 * K + 4)[4:].view(4, K)
    elif case == "misaligned weight":
        flat = torch.zeros(K + 4, dtype=torch.bfloat16, device="cuda")
        flat[4:] = m.weight.data
        m.weight.data = flat[4:]
        assert m.weight.data_ptr() % 16 == 8
    elif case == "broadcast weight":
        m.weight = nn.Parameter(m.weight.data[:1], requires_grad=False)
    elif case == "negative view":
        x = torch._neg_view(x)
    elif case == "scalar":
        x = x[0, 0]
    assert torch.equal(m(x), _expression(x, m.weight, m.eps)) and calls["rmsnorm"] == 0


@GPU
def test_transformed_tensors_keep_the_expression(calls):
    from torch._subclasses.fake_tensor import FakeTensorMode
    from torch.fx.experimental.proxy_tensor import make_fx
    from torch.utils.flop_counter import FlopCounterMode

    K = 1024
    x, t, m = _x(4, K), _x(4, K) * 0.5, _norm(K, "cuda")
    ref = _expression(x, m.weight, m.eps)
    # forward mode, alone and under a functional transform
    with forward_ad.dual_level():
        want = forward_ad.unpack_dual(_expression(forward_ad.make_dual(x, t), m.weight, m.eps)).tangent
        got = forward_ad.unpack_dual(m(forward_ad.make_dual(x, t))).tangent
    assert got is not None and torch.equal(got, want)
    with torch.no_grad():
        assert torch.equal(torch.func.jvp(m, (x,), (t,))[1], want)
    # reverse mode
    xr = x.clone().requires_grad_()
    m(xr).float().sum().backward()
    assert xr.grad is not None and xr.grad.abs().sum() > 0
    assert torch.equal(torch.func.vmap(m)(x), ref)
    # tracers and modes that watch the torch ops
    traced = make_fx(m)(x)
    assert any("rsqrt" in str(n.target) for n in traced.graph.nodes) and torch.equal(traced(x), ref)
    jitted = torch.jit.trace(m, x, check_trace=False)     # (the check runs the module untraced)
    assert _close(jitted(2 * x), _expression(2 * x, m.weight, m.eps))
    with FakeTensorMode(allow_non_fake_inputs=True) as mode:
        assert m(mode.from_tensor(x)).shape == x.shape
    with FlopCounterMode(display=False):
        assert torch.equal(m(x), ref)
    assert calls["rmsnorm"] == 0
