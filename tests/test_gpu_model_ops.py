"""GPU: RMSNorm and the fused per-head norm + rotary embedding against the same ops in torch (which round to bf16 at the
same places; only the order of the sum of squares differs, so an element may move by one bf16 step: 2^-7 of it, or of the
two products it is the sum of)."""
import pytest
import torch

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
