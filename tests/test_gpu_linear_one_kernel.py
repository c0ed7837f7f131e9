"""GPU: one or two bf16 tokens, quantised inside the CUDA-core GEMM, give the codes, scales and outputs of the two separate kernels."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _rows(M, K, kind, gen):
    x = torch.randn(M, K, device="cuda", generator=gen)
    if kind == "halves":          # x / s exactly on k + 0.5, and next to it
        step = torch.randint(-14, 15, (M, K), device="cuda", generator=gen).float() / 14
        top = torch.randint(128, 256, (M, K // 128, 1), device="cuda", generator=gen).float()
        x = (step.view(M, -1, 128) * top).view(M, K)
        x[:, ::128] = top.view(M, -1)
    elif kind == "edges":         # zero, tiny, huge, infinite groups and numbers that are none
        x.view(M, -1, 128)[:, 0::6] = 0.0
        x.view(M, -1, 128)[:, 1::6] *= 1e-38
        x.view(M, -1, 128)[:, 2::6] *= 1e37
        x.view(M, -1, 128)[:, 3::6, 5] = float("inf")
        x.view(M, -1, 128)[:, 4::6, 7] = float("nan")
    return x.to(torch.bfloat16)


@pytest.mark.parametrize("kind", ["normal", "halves", "edges"])
@pytest.mark.parametrize("M", [1, 2])
@pytest.mark.parametrize("K,N,pad", [(128, 1, 0), (384, 33, 8), (4096, 6144, 0), (1920, 1000, 128), (12288, 4096, 0), (65408, 96, 0), (4096, 24576, 16)])
def test_same_as_two_kernels(M, K, N, pad, kind):
    from fp8_inference_toolkit_b200 import ops

    gen = torch.Generator(device="cuda").manual_seed(K + N + M)
    w = (torch.randn(N, K, device="cuda", generator=gen) * 0.02).to(torch.bfloat16)
    wp, ws = ops.static_int4_weight_quant_grouped(w, 128)
    base = torch.zeros(M, K + pad, dtype=torch.bfloat16, device="cuda")
    x = base[:, :K]
    x.copy_(_rows(M, K, kind, gen))
    p, s = ops.dynamic_int4_quant_grouped(x, 128)
    want = torch.empty(M, N, dtype=torch.bfloat16, device="cuda")
    ops.cutlass_int4_fused_grouped_gemm(p, wp, s, ws, want, M, N, 128, K // 128)
    q, t, out = torch.full_like(p, 0x55), torch.full_like(s, -1.0), torch.full_like(want, 7.0)
    args = (wp.data_ptr(), ws.data_ptr(), 0, q.data_ptr(), t.data_ptr(), out.data_ptr(), N, None, 0, 0, torch.cuda.current_stream().cuda_stream)
    ops.check(ops.lib.i4tc_linear(x.data_ptr(), ops._DTYPES[x.dtype], M, K, x.stride(0), *args), "linear")
    assert torch.equal(q, p)
    assert torch.equal(t.view(torch.int32), s.view(torch.int32))
    assert torch.equal(out.view(torch.int16), want.view(torch.int16))
    got = ops.linear(x, wp, ws, N, False)
    assert torch.equal(got.view(torch.int16), want.view(torch.int16))


def test_output_over_the_activations():
    """What overlaps takes the separate kernels, which read all of x before anything of out is written."""
    from fp8_inference_toolkit_b200 import ops

    K = N = 4096
    gen = torch.Generator(device="cuda").manual_seed(1)
    wp, ws = ops.static_int4_weight_quant_grouped((torch.randn(N, K, device="cuda", generator=gen) * 0.02).to(torch.bfloat16), 128)
    x = torch.randn(1, K, device="cuda", generator=gen).to(torch.bfloat16)
    want = ops.linear(x, wp, ws, N, False)
    p, s = ops.dynamic_int4_quant_grouped(x, 128)
    ops.check(ops.lib.i4tc_linear(x.data_ptr(), ops._DTYPES[x.dtype], 1, K, K, wp.data_ptr(), ws.data_ptr(), 0, p.data_ptr(), s.data_ptr(),
                                  x.data_ptr(), N, None, 0, 0, torch.cuda.current_stream().cuda_stream), "linear")
    assert torch.equal(x, want)


@pytest.mark.parametrize("M,K,N,want", [
    (1, 4096, 6144, 1), (2, 4096, 6144, 1), (1, 4096, 12288, 1), (2, 12288, 4096, 1),     # little to quantise in a block and an SM
    (1, 4096, 16001, 2), (1, 4096, 24576, 2), (2, 12288, 16000, 2), (2, 16384, 4096, 2), (1, 65408, 8192, 2),   # it would cost more than a launch
])
def test_where_it_pays(M, K, N, want):
    from fp8_inference_toolkit_b200 import ops
    from tests.helpers import launches

    gen = torch.Generator(device="cuda").manual_seed(K)
    wp = torch.randint(0, 256, (K // 128, N, 64), dtype=torch.uint8, device="cuda", generator=gen)
    ws = torch.rand(K // 128, N, device="cuda", generator=gen)
    x = torch.randn(M, K, device="cuda", generator=gen).to(torch.bfloat16)
    assert launches(lambda: ops.linear(x, wp, ws, N, False)) == want
