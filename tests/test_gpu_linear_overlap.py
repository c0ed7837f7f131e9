"""GPU: the one-call linear, whose GEMM starts under the end of its quantiser, gives what the separate calls give on every route it
can take -- back to back with other inputs and buffers that come round again, and captured in a graph."""
import pytest
import torch

pytestmark = pytest.mark.gpu

# M: CUDA-core kernel, register-fed kernel (tokens staged or not, row-major), split-K tiles, expanded operands on SM pairs, one wave and many
SHAPES = [(1, 1024, 96), (2, 4096, 1000), (8, 4096, 2048), (16, 4096, 9600), (32, 8192, 512), (40, 2048, 1000), (100, 4096, 1024),
          (129, 8192, 1000), (300, 4096, 4096), (1000, 2048, 3001)]


def _separate(x, lin, per_channel):
    from fp8_inference_toolkit_b200 import ops

    M, K = x.shape
    N = lin.out_features
    out = torch.empty(M, N, dtype=torch.bfloat16, device="cuda")
    if per_channel:
        p, s = ops.dynamic_int4_quant(x)
        torch.cuda.synchronize()
        ops.cutlass_int4_scaled_mm(p, lin.weight_int4, s, lin.weight_scale, out, M, N, K)
    else:
        p, s = ops.dynamic_int4_quant_grouped(x, 128)
        torch.cuda.synchronize()
        ops.cutlass_int4_fused_grouped_gemm(p, lin.weight_int4, s, lin.weight_scale, out, M, N, 128, K // 128)
    return out


def _linear(K, N, per_channel, gen):
    from fp8_inference_toolkit_b200.linear import W4A4Linear

    lin = W4A4Linear(K, N, per_channel=per_channel, device="cuda")
    lin.weight.data.copy_((torch.randn(N, K, device="cuda", generator=gen) * 0.02).to(torch.bfloat16))
    return lin.quantize_()


@pytest.mark.parametrize("per_channel", [False, True])
@pytest.mark.parametrize("M,K,N", SHAPES)
def test_back_to_back(M, K, N, per_channel):
    from fp8_inference_toolkit_b200 import ops

    gen = torch.Generator(device="cuda").manual_seed(M + N)
    lins = [_linear(K, N, per_channel, gen) for _ in range(3)]
    xs = [torch.randn(M, K, device="cuda", generator=gen).mul_(10.0 ** (i - 2)).to(torch.bfloat16) for i in range(5)]
    want = [[_separate(x, lin, per_channel) for x in xs] for lin in lins]
    torch.cuda.synchronize()
    got = [(i % 3, i % 5, lins[i % 3](xs[i % 5])) for i in range(30)]   # no synchronisation between; scratch is reused at once
    for a, b, out in got:
        assert torch.equal(out, want[a][b])
    # weights quantised right in front of the call that reads them
    fresh = _linear(K, N, per_channel, gen)
    first = fresh(xs[0])
    assert torch.equal(first, _separate(xs[0], fresh, per_channel))
    ops.check_status()


@pytest.mark.parametrize("per_channel", [False, True])
@pytest.mark.parametrize("M,K,N", SHAPES)
def test_in_a_graph(M, K, N, per_channel):
    from fp8_inference_toolkit_b200 import ops

    gen = torch.Generator(device="cuda").manual_seed(M + K)
    lin = _linear(K, N, per_channel, gen)
    x = torch.randn(M, K, device="cuda", generator=gen).to(torch.bfloat16)
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        lin(x)      # (the split-K workspace of the stream)
    torch.cuda.current_stream().wait_stream(side)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=side):
        y = lin(lin(x)[:, :1].expand(M, K).contiguous())   # two in a row, the second on the first one's output
    for i in range(3):
        x.copy_(torch.randn(M, K, device="cuda", generator=gen).mul_(3.0 ** i).to(torch.bfloat16))
        graph.replay()
        z = _separate(x, lin, per_channel)[:, :1].expand(M, K).contiguous()
        assert torch.equal(y, _separate(z, lin, per_channel))
    ops.check_status()


@pytest.mark.parametrize("smooth", [False, True])
@pytest.mark.parametrize("M,K,N", [(1, 1024, 96), (40, 2048, 1000), (300, 4096, 4096), (1000, 2048, 3001)])
def test_asymmetric_back_to_back(M, K, N, smooth):
    from fp8_inference_toolkit_b200 import ops

    gen = torch.Generator(device="cuda").manual_seed(M)
    w = (torch.randn(N, K, device="cuda", generator=gen) * 0.02).to(torch.bfloat16)
    wp, ws = ops.static_int4_weight_quant_grouped(w, 128)
    cs = ops.int4_weight_group_sums(wp)
    sm = (torch.rand(K, device="cuda", generator=gen) + 0.5).to(torch.bfloat16) if smooth else None
    xs = [(torch.randn(M, K, device="cuda", generator=gen) + 0.75 * i).to(torch.bfloat16) for i in range(4)]
    want = []
    for x in xs:
        out = torch.empty(M, N, dtype=torch.bfloat16, device="cuda")
        p, s, z = ops.dynamic_int4_quant_asymmetric_clipped_grouped(x, 128, 0.95, sm)
        torch.cuda.synchronize()
        ops.cutlass_int4_fused_grouped_gemm_azp(p, wp, s, ws, out, z, cs, M, N, 128, K // 128)
        want.append(out)
    torch.cuda.synchronize()
    got = [ops.linear_asymmetric(xs[i % 4], wp, ws, cs, N, 0.95, sm) for i in range(20)]
    for i, out in enumerate(got):
        assert torch.equal(out, want[i % 4])
    ops.check_status()


@pytest.mark.parametrize("M,K,N", [(40, 2048, 1000), (100, 4096, 1024), (300, 4096, 4096), (1000, 2048, 3001)])
def test_weights_written_in_front(M, K, N):
    """The GEMM entry points start under the kernel in front of them as well, which may have written the weights."""
    from fp8_inference_toolkit_b200 import ops

    gen = torch.Generator(device="cuda").manual_seed(N)
    x = torch.randn(M, K, device="cuda", generator=gen).to(torch.bfloat16)
    ws = [(torch.randn(N, K, device="cuda", generator=gen) * 0.02).to(torch.bfloat16) for _ in range(3)]
    xp, xs = ops.dynamic_int4_quant_grouped(x, 128)
    x8, x8s = ops.dynamic_int8_quant(x)

    def grouped(w, between=lambda: None):
        out = torch.empty(M, N, dtype=torch.bfloat16, device="cuda")
        p, s = ops.static_int4_weight_quant_grouped(w, 128)
        between()
        ops.cutlass_int4_fused_grouped_gemm(xp, p, xs, s, out, M, N, 128, K // 128)
        return out

    def int8(w, between=lambda: None):   # (the int8 rows of the weight stand for the unpacked codes)
        out = torch.empty(M, N, dtype=torch.bfloat16, device="cuda")
        q, s = ops.dynamic_int8_quant(w)
        between()
        ops.cutlass_w4a8_scaled_mm(x8, q, x8s, s, out, M, N, K)
        return out

    for run in (grouped, int8):
        want = []
        for w in ws:
            want.append(run(w, torch.cuda.synchronize))   # the weights are complete before the GEMM is launched
            torch.cuda.synchronize()
        got = [run(ws[i % 3]) for i in range(12)]   # the packed weights of a call take the memory of the ones before
        for i, out in enumerate(got):
            assert torch.equal(out, want[i % 3])
    ops.check_status()
