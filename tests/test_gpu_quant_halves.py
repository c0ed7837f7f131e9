"""GPU: bf16 values whose quotient by absmax / 7 lies exactly between two codes.  Every significand of the absmax meets every
significand and exponent that can land on or beside a half, at several scales, through both quantisers; codes and scales equal
the oracle's, which divides."""
import numpy as np
import pytest
import torch

from oracle import w4a4_oracle as O

pytestmark = pytest.mark.gpu


def _groups(scale):
    """[rows, 128]: per absmax significand all smaller values of seven binades, both signs, 127 to a group beside the absmax."""
    sig = torch.arange(128, 256, dtype=torch.float64)
    values = torch.cat([sig * 2.0 ** -e for e in range(7)])
    rows = []
    for a in sig:
        v = values[values <= a]
        v = torch.cat([v, -v])
        v = torch.cat([v, torch.zeros((-len(v)) % 127, dtype=v.dtype)]).view(-1, 127)
        top = torch.full((v.shape[0], 1), float(a), dtype=v.dtype)
        top[::2] *= -1
        rows.append(torch.cat([top, v], 1))
    x = torch.cat(rows) * scale
    b = x.to(torch.bfloat16)
    assert torch.equal(b.double(), x)   # nothing was rounded
    return b


@pytest.mark.parametrize("exponent", [0, -90, 100])
def test_every_half_of_every_absmax(exponent):
    from fp8_inference_toolkit_b200 import ops

    x = _groups(2.0 ** exponent)
    # per group: 8 groups to a row, so that lanes of one warp hold different groups
    g = torch.cat([x, x[: (-x.shape[0]) % 8]]).view(-1, 1024)
    codes, scale = O.quant_grouped(g, 128, "activation")
    p, s = ops.dynamic_int4_quant_grouped(g.cuda(), 128)
    assert np.array_equal(p.cpu().numpy(), O.pack_int4(codes))
    assert np.array_equal(s.cpu().numpy(), scale)
    # per row
    codes, scale = O.quant_rowwise(x, "activation")
    p, s = ops.dynamic_int4_quant(x.cuda())
    assert np.array_equal(p.cpu().numpy(), O.pack_int4(codes))
    assert np.array_equal(s.cpu().numpy(), scale)
