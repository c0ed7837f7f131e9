"""GPU: the int8 row quantiser with the row in registers against the oracle and against the two-pass kernel (rows off a 16-byte
boundary), at the edges of its chunks of 2048, with exact halves, and with values that are not finite."""
import numpy as np
import pytest
import torch

from oracle import w4a4_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("K", [8, 2048, 2056, 4096, 4104, 8192, 8200, 12288, 12296, 16384, 16392])
def test_codes_equal_the_oracle(K, dtype):
    from fp8_inference_toolkit_b200 import ops

    gen = torch.Generator().manual_seed(K)
    x = torch.randn(5, K, generator=gen) * 3
    x[:, : K // 2] = torch.randint(-254, 255, (5, K // 2), generator=gen) / 2     # codes and halves of an absmax of 127
    x[1, 0] = 127.0
    x[2] = 0.0
    x[3] *= 1e-30 if dtype == torch.bfloat16 else 1e-3
    x = x.to(dtype)
    codes, scale = O.quant_rowwise_int8(x)
    q, s = ops.dynamic_int8_quant(x.cuda())
    assert np.array_equal(q.cpu().numpy(), codes)
    assert np.array_equal(s.cpu().numpy(), scale)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("value", [float("inf"), -float("inf"), float("nan")])
def test_values_that_are_not_finite(value, dtype):
    from fp8_inference_toolkit_b200 import _cabi, ops

    gen = torch.Generator(device="cuda").manual_seed(4)
    x = torch.randn(3, 264, device="cuda", generator=gen).to(dtype)
    x[1, 100:103] = value
    off = torch.empty(3, 272, dtype=dtype, device="cuda")[:, 1:265]
    off.copy_(x)
    q, s = ops.dynamic_int8_quant(x)
    q2, s2 = torch.empty_like(q), torch.empty_like(s)
    _cabi.check(_cabi.lib.i4tc_quant_rowwise_int8(off.data_ptr(), _cabi.BF16 if dtype == torch.bfloat16 else _cabi.FP16, 3, 264, 272,
                                                  q2.data_ptr(), s2.data_ptr(), torch.cuda.current_device(),
                                                  torch.cuda.current_stream().cuda_stream), "i4tc_quant_rowwise_int8")
    assert torch.equal(q, q2) and torch.equal(s, s2)
