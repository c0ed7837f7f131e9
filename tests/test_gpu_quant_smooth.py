"""GPU: the asymmetric quantiser with smoothing factors through its 128-bit kernel (corrected reciprocals) and through the general
one (an IEEE division per element; rows off a 16-byte boundary) gives the same codes, scales and zero points."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _both(x, sm, gs, clip):
    from fp8_inference_toolkit_b200 import ops

    M, K = x.shape
    off = torch.empty(M, K + 8, dtype=x.dtype, device="cuda")[:, 1 : K + 1]   # rows 2 bytes off: the general kernel
    off.copy_(x)
    assert off.data_ptr() % 16
    return [ops.dynamic_int4_quant_asymmetric_clipped_grouped(t, gs, clip, sm) for t in (x, off)]


def _check(x, sm, gs=128, clip=0.95):
    for a, b in zip(*_both(x, sm, gs, clip)):
        assert torch.equal(a.view(torch.uint8), b.view(torch.uint8))   # (bytes: a scale that is not a number counts too)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("M,K,gs", [(1, 128, 128), (9, 192, 64), (300, 1280, 256), (70, 4096, 128)])
def test_ordinary_factors(M, K, gs, dtype):
    gen = torch.Generator(device="cuda").manual_seed(M + K)
    x = torch.randn(M, K, device="cuda", generator=gen) * 3 + 0.75
    x[torch.rand(M, K, device="cuda", generator=gen) < 0.05] = 0.0
    sm = torch.rand(K, device="cuda", generator=gen) * 4 + 0.05
    _check(x.to(dtype), sm.to(dtype), gs)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_every_factor_significand(dtype):
    """Quotients of all pairs of significands of the factor and 127 of the value."""
    n = 128 if dtype == torch.bfloat16 else 1024
    f = (1 + torch.arange(n, device="cuda") / n).to(dtype)
    gen = torch.Generator(device="cuda").manual_seed(1)
    v = (1 + torch.randint(0, n, (128, n), device="cuda", generator=gen) / n).to(dtype)
    _check(v, f)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("factor,value", [
    (0.0, 1.0), (0.0, 0.0), (float("inf"), 1.0), (float("nan"), 1.0), (1.0, float("inf")), (1.0, float("nan")), (-2.0, 1.0),
    (1e-7, 1e4), (6e4, 1e-7), (1e30, 1e-30), (1e-30, 1e30), (1e38, 3e-39), (2.0 ** -126, 2.0 ** -120)])
def test_extreme_elements(factor, value, dtype):
    gen = torch.Generator(device="cuda").manual_seed(2)
    x = torch.randn(4, 256, device="cuda", generator=gen).to(dtype)
    sm = (torch.rand(256, device="cuda", generator=gen) + 0.5).to(dtype)
    x[1:3, 37] = value
    sm[37] = factor
    _check(x, sm)
    _check(torch.zeros_like(x), sm)


@pytest.mark.parametrize("M,K,gs", [(2048, 256, 128), (2049, 256, 128), (2049, 640, 128), (2049, 768, 128), (2049, 384, 64), (2049, 448, 64)])
def test_many_short_rows(M, K, gs):
    """Both sides of the line beyond which short rows keep the general kernel."""
    gen = torch.Generator(device="cuda").manual_seed(K)
    _check((torch.randn(M, K, device="cuda", generator=gen) + 0.75).to(torch.bfloat16),
           (torch.rand(K, device="cuda", generator=gen) + 0.5).to(torch.bfloat16), gs)


def test_many_short_rows_are_not_slowed_down():
    """16384 rows of 256: no slower than rows that the 128-bit kernel cannot take (it needed twice as long)."""
    from fp8_inference_toolkit_b200 import ops
    from tests.helpers import device_us

    M, K = 16384, 256
    x = torch.randn(M, K, device="cuda").to(torch.bfloat16)
    off = torch.empty(M, K + 8, dtype=x.dtype, device="cuda")[:, 1 : K + 1]
    off.copy_(x)
    sm = torch.ones(K, dtype=torch.bfloat16, device="cuda")
    us = [device_us(lambda: ops.dynamic_int4_quant_asymmetric_clipped_grouped(t, 128, 0.95, sm)) for t in (x, off)]
    assert us[0] < 1.2 * us[1], us
