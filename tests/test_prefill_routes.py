"""Which calls of the prefill model take the fused norm and norm + rotary kernels: those that give what the torch expressions
give, and no others (tensors or norms that something watches, replaces or transforms stay with torch)."""
import pytest
import torch
import torch.nn.functional as F
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


def _block(q_heads, kv_heads, device):
    """A layer's attention without its linears (which need a GPU)."""
    from fp8_inference_toolkit_b200.qwen3 import Block, Qwen3Config

    blk = Block.__new__(Block)
    nn.Module.__init__(blk)
    blk.cfg = Qwen3Config(hidden=256, q_heads=q_heads, kv_heads=kv_heads, head_dim=128)
    blk.q_norm, blk.k_norm = _norm(128, device), _norm(128, device)
    return blk


def _inputs(blk, B, S, device):
    from fp8_inference_toolkit_b200.qwen3 import rope_tables

    width = (blk.cfg.q_heads + 2 * blk.cfg.kv_heads) * 128
    qkv = torch.randn(B, S, width, generator=torch.Generator().manual_seed(5)).to(torch.bfloat16).to(device)
    return qkv, *rope_tables(S, 128, 1e4, device)


def _attention(blk, qkv, B, S, cos, sin):
    """The layer's attention as torch ops, through its norm modules."""
    from fp8_inference_toolkit_b200.qwen3 import apply_rope

    hq, hk = blk.cfg.q_heads, blk.cfg.kv_heads
    q, k, v = (t.view(B, S, -1, 128) for t in qkv.split([hq * 128, hk * 128, hk * 128], -1))
    q, k, v = blk.q_norm(q).transpose(1, 2), blk.k_norm(k).transpose(1, 2), v.transpose(1, 2)
    q, k = apply_rope(q, cos, sin), apply_rope(k, cos, sin)
    return F.scaled_dot_product_attention(q, k, v, is_causal=True, enable_gqa=True).transpose(1, 2).reshape(B, S, -1)


def test_attention_on_the_cpu_stays_with_torch():
    blk = _block(4, 2, "cpu")
    args = _inputs(blk, 2, 9, "cpu")
    assert torch.equal(blk._attention(args[0], 2, 9, *args[1:]), _attention(blk, args[0], 2, 9, *args[1:]))


@GPU
@pytest.mark.parametrize("case", ["plain", "eps", "hook", "global hook", "pre-hook", "replaced", "patched", "unequal eps",
                                  "float tables", "strided tables", "half", "shared weight", "grad"])
def test_attention_goes_through_norms_that_someone_changed(case, calls):
    B, S = 2, 9
    blk = _block(4, 2, "cuda")
    qkv, cos, sin = _inputs(blk, B, S, "cuda")
    seen, handles = [], []
    if case == "eps":           # the norms' own, not the configuration's
        blk.q_norm.eps = blk.k_norm.eps = 3.0
    elif case == "unequal eps":
        blk.k_norm.eps = 3.0
    elif case == "hook":
        handles.append(blk.q_norm.register_forward_hook(lambda m, i, o: seen.append(1) or 2 * o))
    elif case == "pre-hook":
        handles.append(blk.k_norm.register_forward_pre_hook(lambda m, i: seen.append(1)))
    elif case == "global hook":
        handles.append(nn.modules.module.register_module_forward_hook(lambda m, i, o: seen.append(1)))
    elif case == "replaced":
        blk.k_norm = nn.Identity()
    elif case == "patched":
        blk.q_norm.forward = lambda x: x * 0.5
    elif case == "float tables":
        sin = sin.float().to(torch.bfloat16).float()
        cos = cos.float()
        # (fp32 tables promote q and k, so the values have to follow)
        qkv, blk = qkv.float(), blk.float()
    elif case == "strided tables":
        cos, sin = cos.t().contiguous().t(), sin.t().contiguous().t()
    elif case == "half":
        qkv, cos, sin, blk = qkv.half(), cos.half(), sin.half(), blk.half()
    elif case == "shared weight":
        blk.q_norm.weight = nn.Parameter(blk.q_norm.weight.data[:1], requires_grad=False)
    elif case == "grad":
        blk.q_norm.weight.requires_grad_()
    ref = _attention(blk, qkv.clone(), B, S, cos, sin)
    fired = len(seen)
    got = blk._attention(qkv.clone(), B, S, cos, sin)
    for h in handles:
        h.remove()
    if case in ("plain", "eps"):
        assert calls["qk_norm_rope_"] == 1
        # norm and rotary round to bf16 as torch does; a score moves by a few bf16 steps of its terms at most
        err = (got.float() - ref.float()).norm() / ref.float().norm()
        assert err < 2e-2, err
    else:
        assert calls["qk_norm_rope_"] == 0 and torch.equal(got, ref)
        assert len(seen) == 2 * fired
    if case == "grad":
        got.float().sum().backward()
        assert blk.q_norm.weight.grad is not None


@GPU
def test_wide_prefill_takes_both_kernels(calls):
    """A model of the real head size and of a hidden size that the norm kernel takes, against its torch path."""
    from fp8_inference_toolkit_b200 import ops
    from fp8_inference_toolkit_b200.qwen3 import Qwen3Config, Qwen3Prefill

    cfg = Qwen3Config(hidden=1024, layers=2, q_heads=8, kv_heads=2, head_dim=128, inter=1536, vocab=1000)
    m = Qwen3Prefill(cfg, "cuda")
    ids = torch.randint(0, cfg.vocab, (3, 70), device="cuda", generator=torch.Generator(device="cuda").manual_seed(1))
    y = m(ids)
    ops.check_status()
    assert calls == {"rmsnorm": 1, "qk_norm_rope_": cfg.layers}     # the final norm; one attention per layer
    assert torch.equal(y, m(ids))
    ids2 = ids.clone()
    ids2[:, -1] = (ids2[:, -1] + 1) % cfg.vocab
    assert torch.equal(m(ids2)[:, :-1], y[:, :-1])                  # causal
    plain = Qwen3Prefill(cfg, "cuda", fused=False)
    plain.embed.load_state_dict(m.embed.state_dict())               # the linears are seeded, the embedding table is not
    before = calls["qk_norm_rope_"]
    y_plain = plain(ids)
    assert calls["qk_norm_rope_"] == before
    assert F.cosine_similarity(y.float().flatten(), y_plain.float().flatten(), dim=0).item() > 0.995
