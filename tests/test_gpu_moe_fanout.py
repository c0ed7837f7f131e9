"""GPU: quantising each token straight into its expert-sorted rows gives the rows of quantise-then-copy; the one-chunk sort; and
layers one after the other, whose kernels start under the end of their predecessors, on inputs that change every call."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T,K,top_k", [(1, 128, 1), (7, 384, 3), (65, 1152, 8), (130, 2048, 40)])
def test_same_rows_as_the_copy(T, K, top_k):
    from fp8_inference_toolkit_b200 import moe, ops

    gen = torch.Generator(device="cuda").manual_seed(T)
    x = torch.randn(T, K, device="cuda", generator=gen).to(torch.bfloat16)
    ids = torch.randint(-1, 9, (T, top_k), device="cuda", generator=gen).to(torch.int32)     # -1 and 8: left out
    sp, inv, off = moe.moe_sort_tokens(ids, 8)
    n = int(off[-1])
    p, s = moe.moe_quant_gather(x, sp, top_k)
    p2, s2 = moe.moe_quant_fanout(x, inv, top_k)
    assert torch.equal(p[:, :n], p2[:, :n]) and torch.equal(s[:, :n], s2[:, :n])
    ops.check_status()


def test_rows_past_the_destination_are_not_written():
    from fp8_inference_toolkit_b200 import moe, ops

    T, K, R = 5, 256, 7
    x = torch.randn(T, K, device="cuda").to(torch.bfloat16)
    inv = torch.tensor([0, 2, 4, 7, 2 ** 31 - 1, -1, -(2 ** 31), 1, 3, 6], dtype=torch.int32, device="cuda")
    p = torch.full((K // 128, R, 64), 0x5A, dtype=torch.uint8, device="cuda")
    s = torch.full((K // 128, R), -1.0, device="cuda")
    ops.check(ops.lib.i4tc_moe_quant_fanout(x.data_ptr(), T, K, K, inv.data_ptr(), 2, R, p.data_ptr(), s.data_ptr(), 0,
                                            torch.cuda.current_stream().cuda_stream), "moe_quant_fanout")
    want_p, want_s = ops.dynamic_int4_quant_grouped(x, 128)
    rows = {0: 0, 2: 0, 4: 1, 1: 3, 3: 4, 6: 4}
    for r in range(R):
        if r in rows:
            assert torch.equal(p[:, r], want_p[:, rows[r]]) and torch.equal(s[:, r], want_s[:, rows[r]])
        else:
            assert (p[:, r] == 0x5A).all() and (s[:, r] == -1.0).all()


def _stage_by_stage(x, ids, wt, w):
    """The layer with nothing beside anything: every kernel ends before the next is launched, the rows by quantise and copy."""
    from fp8_inference_toolkit_b200 import moe

    def done(result):
        torch.cuda.synchronize()
        return result

    T, k = ids.shape
    sp, inv, off = done(moe.moe_sort_tokens(ids, w.num_experts))
    a, sa = done(moe.moe_gather_quant(x, sp, k))
    h = torch.empty(T * k, 2 * w.inter, dtype=torch.bfloat16, device="cuda")
    done(moe.moe_w4a4_grouped_gemm(a, sa, w.gate_up_packed, w.gate_up_scale, off, h, 2 * w.inter, w.hidden // 128, w.num_experts))
    b, sb = done(moe.moe_silu_mul_quant(h))
    y = torch.empty(T * k, w.hidden, dtype=torch.bfloat16, device="cuda")
    done(moe.moe_w4a4_grouped_gemm(b, sb, w.down_packed, w.down_scale, off, y, w.hidden, w.inter // 128, w.num_experts))
    return done(moe.moe_combine(y, inv, wt.contiguous(), T, k))


@pytest.mark.parametrize("T", [3, 64, 300, 700])
def test_layers_back_to_back(T):
    """300 and 700 tokens: the register-fed and the tile kernel."""
    from fp8_inference_toolkit_b200 import moe, ops

    E, H, I, k = 16, 512, 256, 2
    gen = torch.Generator(device="cuda").manual_seed(T)
    w = moe.MoEWeights.quantize((torch.randn(E, 2 * I, H, device="cuda", generator=gen) * 0.02).to(torch.bfloat16),
                                (torch.randn(E, H, I, device="cuda", generator=gen) * 0.02).to(torch.bfloat16))
    xs = [torch.randn(T, H, device="cuda", generator=gen).mul_(2.0 ** i).to(torch.bfloat16) for i in range(4)]
    routes = [moe.moe_route(torch.randn(T, E, device="cuda", generator=gen), k) for _ in range(4)]
    want = [_stage_by_stage(x, ids, wt, w) for x, (ids, wt) in zip(xs, routes)]
    got = [moe.moe_layer(xs[i % 4], *routes[i % 4], w) for i in range(24)]
    for i, out in enumerate(got):
        assert torch.equal(out, want[i % 4])
    ops.check_status()
