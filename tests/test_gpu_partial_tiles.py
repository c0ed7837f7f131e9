"""GPU: row tiles that are mostly padding (a few tokens per expert) give the oracle's bits, whatever part of a warp's rows
exists; and the one-call linear equals its separate ops and refuses what they refuse."""
import numpy as np
import pytest
import torch

from oracle import w4a4_oracle as O
from tests.helpers import dev_f32, dev_packed, rand_codes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N", [128, 256, 264])
def test_experts_of_every_fill(N):
    from fp8_inference_toolkit_b200 import moe, ops

    counts = [0, 1, 15, 16, 17, 32, 33, 48, 49, 0, 100, 128, 129, 144, 145, 3]
    G, E, P = 3, len(counts), sum(counts)
    rng = np.random.RandomState(N)
    a, b = rand_codes(rng, (G, P, 128)), rand_codes(rng, (E, G, N, 128))
    sa = (rng.rand(G, P).astype(np.float32) + 0.01) * 0.1
    sb = (rng.rand(E, G, N).astype(np.float32) + 0.01) * 0.01
    offsets = np.concatenate([[0], np.cumsum(counts)]).astype(np.int32)
    out = torch.full((P, N), float("nan"), dtype=torch.bfloat16, device="cuda")
    moe.moe_w4a4_grouped_gemm(dev_packed(a), dev_f32(sa), dev_packed(b), dev_f32(sb), torch.from_numpy(offsets).cuda(), out, N, G, E)
    ops.check_status()
    for e in range(E):
        r0, r1 = offsets[e], offsets[e + 1]
        if r1 > r0:
            ref = O.linear_grouped(np.ascontiguousarray(a[:, r0:r1]), b[e], np.ascontiguousarray(sa[:, r0:r1]), sb[e])
            assert torch.equal(out[r0:r1].cpu(), ref), (e, counts[e])


@pytest.mark.parametrize("per_channel", [False, True])
@pytest.mark.parametrize("M", [1, 2, 17, 100, 129, 600])
def test_one_call_linear_equals_the_ops(M, per_channel):
    from fp8_inference_toolkit_b200 import ops

    K, N = 2048, 1000
    gen = torch.Generator(device="cuda").manual_seed(M)
    wide = torch.randn(M, K + 8, device="cuda", generator=gen).to(torch.bfloat16)
    w = torch.randn(N, K, device="cuda", generator=gen).to(torch.bfloat16)
    wp, ws = ops.static_int4_weight_quant(w) if per_channel else ops.static_int4_weight_quant_grouped(w, 128)
    inputs = [wide[:, :K].contiguous(), wide[:, 8:], wide[:, :K].half(), wide[:, :K].float()]
    if M > 1:   # (one misaligned row counts as contiguous and is refused by the quantisers)
        inputs.append(wide[:, 3:K + 3])
    for x in inputs:
        ref = torch.empty(M, N, dtype=torch.bfloat16, device="cuda")
        if per_channel:
            xp, xs = ops.dynamic_int4_quant(x)
            ops.cutlass_int4_scaled_mm(xp, wp, xs, ws, ref, M, N, K)
        else:
            xp, xs = ops.dynamic_int4_quant_grouped(x, 128)
            ops.cutlass_int4_fused_grouped_gemm(xp, wp, xs, ws, ref, M, N, 128, K // 128)
        assert torch.equal(ops.linear(x, wp, ws, N, per_channel), ref)
    ops.check_status()


@pytest.mark.parametrize("per_channel", [False, True])
def test_one_call_linear_refuses_what_the_ops_refuse(per_channel):
    from fp8_inference_toolkit_b200 import ops

    M, K, N, G = 4, 256, 24, 1 if per_channel else 2
    x = torch.zeros(M, K, dtype=torch.bfloat16, device="cuda")
    w = torch.zeros(N * K // 2, dtype=torch.uint8, device="cuda")
    s = torch.ones(G * N, device="cuda")
    assert not ops.linear(x, w, s, N, per_channel).any()
    odd = K - 32     # neither whole groups nor whole 32-byte rows of codes
    for args in [(x.cpu(), w, s), (x[0], w, s), (x.int(), w, s), (x[:, :odd].contiguous(), w[: N * odd // 2], s),
                 (x, w[:-1], s), (x, w.view(torch.int8), s), (x, torch.zeros(N * K, dtype=torch.uint8, device="cuda")[::2], s),
                 (x, w.cpu(), s), (x, w, s[:-1]), (x, w, s.double()), (x, w, s.cpu()), (x, w, torch.ones(2 * G * N, device="cuda")[::2])]:
        with pytest.raises(RuntimeError):
            ops.linear(*args, N, per_channel)
    with pytest.raises(RuntimeError):
        ops.linear(x, w, s, N + 1, per_channel)
    assert ops.linear(x[:0], w, s, N, per_channel).shape == (0, N)
