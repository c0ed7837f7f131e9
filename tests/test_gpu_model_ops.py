"""GPU: RMSNorm and the fused per-head norm + rotary embedding against the same ops in torch (which round to bf16 at the
same places; only the order of the sum of squares differs, so an element may move by one bf16 step: 2^-7 of it, or of the
two products it is the sum of)."""
import pytest
import torch

from tests.helpers import device_us

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,K", [(1, 8), (3, 264), (65, 2048), (7, 4096), (2, 16384)])
def test_rmsnorm(rows, K):
    from fp8_inference_toolkit_b200 import ops

    gen = torch.Generator(device="cuda").manual_seed(K)
    x = (torch.randn(rows, K, device="cuda", generator=gen) * 3).to(torch.bfloat16)
    w = torch.randn(K, device="cuda", generator=gen).to(torch.bfloat16)
    xf = x.double()
    ref = (xf * torch.rsqrt(xf.pow(2).mean(-1, keepdim=True) + 1e-6)).to(torch.bfloat16) * w
    out = ops.rmsnorm(x, w, 1e-6)
    assert ((out.float() - ref.float()).abs() <= 2.0 ** -7 * ref.float().abs()).all()
    assert (out != ref).float().mean() < 0.01


@pytest.mark.parametrize("B,S,q_heads,kv_heads", [(1, 1, 1, 1), (2, 5, 3, 1), (3, 70, 32, 8)])
def test_qk_norm_rope(B, S, q_heads, kv_heads):
    from fp8_inference_toolkit_b200 import ops
    from fp8_inference_toolkit_b200.qwen3 import apply_rope, rope_tables

    gen = torch.Generator(device="cuda").manual_seed(S)
    width = (q_heads + 2 * kv_heads) * 128
    qkv = torch.randn(B * S, width, device="cuda", generator=gen).to(torch.bfloat16)
    wq, wk = (torch.rand(128, device="cuda", generator=gen).add(0.5).to(torch.bfloat16) for _ in range(2))
    cos, sin = rope_tables(S, 128, 1e6, "cuda")
    before = qkv.clone()
    ops.qk_norm_rope_(qkv, wq, wk, cos, sin, q_heads, kv_heads, S, 1e-6)
    n = q_heads + kv_heads
    assert torch.equal(qkv[:, n * 128:], before[:, n * 128:])          # values stay
    x = before[:, : n * 128].view(B, S, n, 128)
    xf = x.double()
    y = (xf * torch.rsqrt(xf.pow(2).mean(-1, keepdim=True) + 1e-6)).to(torch.bfloat16)
    y = torch.cat([y[:, :, :q_heads] * wq, y[:, :, q_heads:] * wk], 2)
    ref = apply_rope(y.transpose(1, 2), cos, sin).transpose(1, 2).reshape(B * S, -1).float()
    mag = y.abs().float()
    bound = 2.0 ** -7 * (mag + mag.roll(64, -1)).view(B * S, -1)
    out = qkv[:, : n * 128].float()
    assert ((out - ref).abs() <= bound).all()
    assert (out != ref).float().mean() < 0.01


@pytest.mark.parametrize("q_heads,kv_heads", [(1, 0), (1, 1), (2, 1), (4, 1), (32, 8), (64, 8)])
def test_qk_norm_rope_splits_the_same_work(q_heads, kv_heads):
    """However tokens and heads are shared out over warps and blocks, and with operands aligned to 8 bytes only, every bit is the same:
    100 tokens at once against the same tokens in smaller calls and off a 16-byte boundary."""
    from fp8_inference_toolkit_b200 import ops
    from fp8_inference_toolkit_b200.qwen3 import rope_tables

    T, width = 100, (q_heads + 2 * kv_heads) * 128
    gen = torch.Generator(device="cuda").manual_seed(q_heads)
    qkv = torch.randn(T, width, device="cuda", generator=gen).to(torch.bfloat16)
    wq, wk = (torch.rand(128, device="cuda", generator=gen).add(0.5).to(torch.bfloat16) for _ in range(2))
    cos, sin = rope_tables(T, 128, 1e6, "cuda")

    def run(offset, *bounds):
        x = torch.empty(T * width + offset, dtype=torch.bfloat16, device="cuda")[offset:].view(T, width).copy_(qkv)
        for a, b in zip((0,) + bounds, bounds + (T,)):
            ops.qk_norm_rope_(x[a:b], wq, wk, cos[a:b].contiguous(), sin[a:b].contiguous(), q_heads, kv_heads, b - a, 1e-6)
        return x

    want = run(0)
    assert torch.equal(run(0, 1, 4, 20, 35), want)      # calls of 1, 3, 16, 15 and 65 tokens
    assert torch.equal(run(4), want) and torch.equal(run(4, 36), want)


def test_qk_norm_rope_uses_the_device():
    """One token's 72 heads run side by side (in one block they took twice as long as eight heads), and one head's tokens do not leave most
    warps of a block idle (they took 0.8 of the time of five heads)."""
    from fp8_inference_toolkit_b200 import ops
    from fp8_inference_toolkit_b200.qwen3 import rope_tables

    def us(T, q_heads, kv_heads):
        x = torch.randn(T, (q_heads + 2 * kv_heads) * 128, device="cuda").to(torch.bfloat16)
        w = torch.ones(128, device="cuda", dtype=torch.bfloat16)
        cos, sin = rope_tables(T, 128, 1e6, "cuda")
        return device_us(lambda: ops.qk_norm_rope_(x, w, w, cos, sin, q_heads, kv_heads, T, 1e-6))

    assert us(1, 64, 8) < 1.5 * us(1, 7, 1)
    assert us(16384, 1, 0) < 0.7 * us(16384, 4, 1)
