"""GPU: SwiGLU in front of the quantiser rounds to bf16 as its definition does, for every bf16 gate value.  A group that holds a
single product other than zero shows it in its scale, absmax / 7; the up values are so large that no scale meets its floor."""
import numpy as np
import pytest
import torch

from oracle import w4a4_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("slot", [0, 5])
def test_every_gate_value(slot):
    from fp8_inference_toolkit_b200 import moe

    gate = torch.arange(0, 65536, dtype=torch.int32).to(torch.int16).view(torch.bfloat16)
    gate = gate[gate.isfinite()]
    gen = torch.Generator().manual_seed(slot)
    reps = 8
    n = gate.numel()
    up = (torch.rand(reps, n, generator=gen) + 1.0) * 2.0 ** 50 * (torch.randint(0, 2, (reps, n), generator=gen) * 2 - 1)
    g = torch.randn(reps * n, 128, generator=gen).to(torch.bfloat16)    # gates beside it, with up values of zero
    u = torch.zeros(reps * n, 128, dtype=torch.bfloat16)
    at = 8 * 3 + slot
    g[:, at] = gate.repeat(reps)
    u[:, at] = up.view(-1).to(torch.bfloat16)
    h = torch.cat([g, u], 1)
    _, s = moe.moe_silu_mul_quant(h.cuda())
    y = O.silu_mul(torch.stack([g[:, at], u[:, at]], 1)).float().view(-1).numpy()
    want = np.maximum(np.abs(y) / np.float32(7), np.float32(1.0) / np.float32(7.0 * 512.0)).astype(np.float32)
    got = s.cpu().numpy().reshape(-1)
    bad = np.nonzero(got != want)[0]
    assert bad.size == 0, (bad.size, g[bad[:4], at], u[bad[:4], at], got[bad[:4]], want[bad[:4]])


@pytest.mark.parametrize("values", [[float("inf")], [float("nan")], [-float("inf"), 40.0], [33.0, -33.0, 32.0, -32.0]])
def test_extreme_gates_leave_their_neighbours_alone(values):
    """Two elements share a reciprocal and eight a decision: whatever one of them holds, the others come out the same."""
    from fp8_inference_toolkit_b200 import moe

    gen = torch.Generator().manual_seed(3)
    g = torch.randn(8, 128, generator=gen).to(torch.bfloat16)
    u = torch.zeros(8, 128, dtype=torch.bfloat16)
    for row in range(8):                       # the element that shows is beside the extreme ones
        g[row, 16 : 16 + 8] = torch.tensor((values * 8)[:8]).to(torch.bfloat16)
        g[row, 16 + row] = torch.tensor(0.75 + row / 8).to(torch.bfloat16)
        u[row, 16 + row] = 2.0 ** 20
    finite = torch.where(torch.isfinite(g), g, torch.zeros_like(g))   # (inf * 0 and nan * 0 are not numbers and count for nothing)
    _, s = moe.moe_silu_mul_quant(torch.cat([finite, u], 1).cuda())
    _, e = moe.moe_silu_mul_quant(torch.cat([g, u], 1).cuda())
    assert torch.equal(s, e)
