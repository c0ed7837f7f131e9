"""GPU: the per-group GEMM over operands expanded to e4m3 (large M, scratch from the caller) gives the same bits as the
kernel that converts inside, over its three tile widths, both epilogues, ragged and unaligned sizes and extreme codes."""
import pytest
import torch

from oracle import w4a4_oracle as O
from tests.helpers import assert_close_bf16

pytestmark = pytest.mark.gpu


def _operands(M, N, G, azp, codes="random", seed=0):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    if codes == "random":
        a = torch.randint(0, 256, (G, M, 64), dtype=torch.uint8, device="cuda", generator=gen)
        b = torch.randint(0, 256, (G, N, 64), dtype=torch.uint8, device="cuda", generator=gen)
    else:   # every code -8 against -8 or 7: the largest sums of either sign
        a = torch.full((G, M, 64), 0x88, dtype=torch.uint8, device="cuda")
        b = torch.full((G, N, 64), 0x88, dtype=torch.uint8, device="cuda")
        b[:, ::2] = 0x77
    sa = torch.rand(G, M, device="cuda", generator=gen) * 0.1 + 1e-3
    sb = torch.rand(G, N, device="cuda", generator=gen) * 0.01 + 1e-4
    z = torch.randint(-8, 9, (G, M), device="cuda", generator=gen).float() if azp else None
    w = torch.randint(-1024, 897, (G, N), device="cuda", generator=gen).float() if azp else None
    return a, b, sa, sb, z, w


def _call(M, N, G, args, nbytes):
    from fp8_inference_toolkit_b200 import _cabi

    a, b, sa, sb, z, w = args
    out = torch.full((M, N), float("nan"), dtype=torch.bfloat16, device="cuda")
    # garbage, NaN patterns included: every byte that reaches an output has to be written by the call
    scratch = torch.full((max(nbytes, 1),), 0x7F, dtype=torch.uint8, device="cuda") if nbytes else None
    _cabi.check(_cabi.lib.i4tc_gemm_grouped_scratch(
        a.data_ptr(), b.data_ptr(), sa.data_ptr(), sb.data_ptr(), None if z is None else z.data_ptr(),
        None if w is None else w.data_ptr(), out.data_ptr(), M, N, 128, G, None if scratch is None else scratch.data_ptr(),
        nbytes, torch.cuda.current_device(), torch.cuda.current_stream().cuda_stream), "i4tc_gemm_grouped_scratch")
    return out


@pytest.mark.parametrize("azp", [False, True])
@pytest.mark.parametrize("codes", ["random", "extreme"])
# every tile width with a ragged last row tile (one row; one row of the pair's second CTA; none of its rows), ragged and odd N,
# full tiles, and several waves
@pytest.mark.parametrize("M,N,G,width", [
    (129, 1000, 64, 128), (257, 1001, 32, 128), (512, 512, 32, 128), (1537, 2568, 40, 128),
    (130, 9473, 32, 192), (1000, 6144, 32, 192),
    (1025, 3001, 32, 256), (1409, 2305, 32, 256), (769, 9465, 32, 256), (2048, 4096, 32, 256)])
def test_same_bits_as_the_converting_kernel(M, N, G, width, codes, azp):
    from fp8_inference_toolkit_b200 import _cabi, ops

    dev = torch.cuda.current_device()
    assert _cabi.lib.i4tc_gemm_grouped_expanded_width(M, N, G, int(azp), dev) == width
    nbytes = _cabi.lib.i4tc_gemm_grouped_scratch_bytes(M, N, G, int(azp), dev)
    assert nbytes > 0
    args = _operands(M, N, G, azp, codes, seed=M + N)
    ref = _call(M, N, G, args, 0)
    assert torch.equal(_call(M, N, G, args, nbytes), ref)
    assert torch.equal(_call(M, N, G, args, nbytes - 1), ref)   # too little scratch: the converting kernel again
    ops.check_status()


def _low_bit_codes(M, N, G, pattern, gen):
    """Codes of group pairs whose sums are large inside and differ by a few units: where fewer than 14 bits of a sum are kept,
    or products are aligned to its size and cut, the difference shows it."""
    def redraw(t):
        r = torch.randint(-8, 8, t.shape, device="cuda", generator=gen, dtype=torch.int8)
        return torch.where(torch.rand(t.shape, device="cuda", generator=gen) < 0.05, r, t)

    H = G // 2
    a = torch.full((H, M, 128), -8, dtype=torch.int8, device="cuda")
    b = torch.full((H, N, 128), -8, dtype=torch.int8, device="cuda")
    if pattern == "cancelling":      # half of the products are 64, half -56, in an order of its own in every group
        for h in range(H):
            b[h][:, torch.randperm(128, device="cuda", generator=gen)[:64]] = 7
    a, b = redraw(a), redraw(b)
    if pattern == "large":
        a[:, 0], b[:, 0] = -8, -8    # the largest sum of all, 2^13
    at = torch.randint(0, 128, (H, M, 1), device="cuda", generator=gen)
    old = a.gather(2, at)
    return a, b, a.scatter(2, at, torch.where(old < 7, old + 1, old - 1))


@pytest.mark.parametrize("pattern", ["large", "cancelling"])
@pytest.mark.parametrize("M,N,G,width", [(257, 1001, 32, 128), (130, 9473, 32, 192), (1025, 3001, 32, 256)])
def test_every_bit_of_a_group_sum_counts(M, N, G, width, pattern):
    from fp8_inference_toolkit_b200 import _cabi, ops

    dev = torch.cuda.current_device()
    assert _cabi.lib.i4tc_gemm_grouped_expanded_width(M, N, G, 0, dev) == width
    a, b, a2 = _low_bit_codes(M, N, G, pattern, torch.Generator(device="cuda").manual_seed(N))
    if pattern == "large":
        assert int((a[0, 0].int() * b[0, 0].int()).sum()) == 1 << 13
    pack = lambda t: (t[..., 0::2] & 15) | ((t[..., 1::2] & 15) << 4)
    both = lambda t, u: torch.stack([t, u], 1).flatten(0, 1).contiguous()     # groups 2 h and 2 h + 1
    scale = torch.tensor([1.0, -1.0], device="cuda").repeat(G // 2)[:, None]
    args = (pack(both(a, a2)).view(torch.uint8), pack(both(b, b)).view(torch.uint8), scale.expand(G, M).contiguous(),
            torch.ones(G, N, device="cuda"), None, None)
    flat = lambda t: t.transpose(0, 1).flatten(1).double()
    ref = flat(a - a2) @ flat(b).T            # small integers, every one of them a bf16 value
    assert ref.abs().max() <= 256
    nbytes = _cabi.lib.i4tc_gemm_grouped_scratch_bytes(M, N, G, 0, dev)
    assert torch.equal(_call(M, N, G, args, nbytes).double(), ref)
    ops.check_status()


def test_against_the_oracle():
    from fp8_inference_toolkit_b200 import ops

    M, N, G = 512, 512, 32
    a, b, sa, sb, _, _ = _operands(M, N, G, False, seed=5)
    out = torch.empty(M, N, dtype=torch.bfloat16, device="cuda")
    ops.cutlass_int4_fused_grouped_gemm(a, b, sa, sb, out, M, N, 128, G)
    ops.check_status()
    codes = [O.unpack_int4(t.cpu().numpy().reshape(-1, 64)).reshape(G, -1, 128) for t in (a, b)]
    ref = O.linear_grouped(codes[0], codes[1], sa.cpu().numpy(), sb.cpu().numpy())
    assert_close_bf16(out, ref, "expanded")
    assert torch.equal(out.cpu(), ref)


def test_inside_a_captured_graph():
    """Scratch comes from torch's allocator, so a capture owns it and a replay works on new inputs."""
    from fp8_inference_toolkit_b200 import ops

    M, N, G = 512, 512, 32
    a, b, sa, sb, _, _ = _operands(M, N, G, False, seed=6)
    out = torch.zeros(M, N, dtype=torch.bfloat16, device="cuda")
    run = lambda: ops.cutlass_int4_fused_grouped_gemm(a, b, sa, sb, out, M, N, 128, G)
    run()
    g = torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.graph(g):
        run()
    a.copy_(a.flip(1))
    g.replay()
    replayed = out.clone()
    run()
    assert torch.equal(replayed, out)


@pytest.mark.parametrize("azp", [False, True])
def test_without_memory_for_scratch(azp, monkeypatch):
    """The converting kernel serves the call."""
    from fp8_inference_toolkit_b200 import _cabi, ops

    M, N, G = 512, 512, 32
    a, b, sa, sb, z, w = _operands(M, N, G, azp, seed=9)
    nbytes = _cabi.lib.i4tc_gemm_grouped_scratch_bytes(M, N, G, int(azp), torch.cuda.current_device())
    x = torch.randn(M, G * 128, device="cuda").to(torch.bfloat16)

    def run():
        out = torch.full((M, N), float("nan"), dtype=torch.bfloat16, device="cuda")
        if azp:
            ops.cutlass_int4_fused_grouped_gemm_azp(a, b, sa, sb, out, z, w, M, N, 128, G)
        else:
            ops.cutlass_int4_fused_grouped_gemm(a, b, sa, sb, out, M, N, 128, G)
        return out, ops.linear(x, b, sb, N, False)

    ref = run()
    refused, empty = [], torch.empty

    def small_only(*size, **kwargs):
        if kwargs.get("dtype") == torch.uint8 and isinstance(size[0], int) and size[0] >= nbytes:
            refused.append(size[0])
            raise torch.cuda.OutOfMemoryError("no room")
        return empty(*size, **kwargs)

    monkeypatch.setattr(torch, "empty", small_only)
    got = run()
    assert len(refused) == 2 and all(torch.equal(p, q) for p, q in zip(got, ref))


def test_operands_off_a_16_byte_boundary_are_refused():
    """On the host, before anything is launched: by the GEMMs and by the one-call linear."""
    from fp8_inference_toolkit_b200 import ops

    M, N, G = 512, 512, 32
    a, b, sa, sb, z, w = _operands(M, N, G, True, seed=7)
    x = torch.randn(M, G * 128, device="cuda").to(torch.bfloat16)
    out = torch.zeros(M, N, dtype=torch.bfloat16, device="cuda")

    def off(t):
        flat = torch.zeros(t.numel() + 8, dtype=torch.uint8, device="cuda")
        flat[8:] = t.reshape(-1)
        return flat[8:].view(t.shape)

    a8, b8 = off(a), off(b)
    assert a8.data_ptr() % 16 == b8.data_ptr() % 16 == 8 and a8.is_contiguous() and b8.is_contiguous()
    for p, q in ((a8, b), (a, b8)):
        with pytest.raises(RuntimeError, match="16-byte aligned"):
            ops.cutlass_int4_fused_grouped_gemm(p, q, sa, sb, out, M, N, 128, G)
        with pytest.raises(RuntimeError, match="16-byte aligned"):
            ops.cutlass_int4_fused_grouped_gemm_azp(p, q, sa, sb, out, z, w, M, N, 128, G)
    with pytest.raises(RuntimeError, match="16-byte aligned"):
        ops.linear(x, b8, sb, N, False)
    torch.cuda.synchronize()
    assert not out.any()


def test_an_unrelated_error_leaves_the_pair_kernels_on():
    """A call that failed for its own reasons (a device that is not there) is no reason to run others without SM pairs."""
    from fp8_inference_toolkit_b200 import _cabi, ops

    M, N, G = 512, 512, 32
    dev = torch.cuda.current_device()
    a, b, sa, sb, _, _ = args = _operands(M, N, G, False, seed=8)
    nbytes = _cabi.lib.i4tc_gemm_grouped_scratch_bytes(M, N, G, 0, dev)
    assert nbytes > 0
    ref = _call(M, N, G, args, 0)
    x = torch.randn(M, G * 128, device="cuda").to(torch.bfloat16)
    y = ops.linear(x, b, sb, N, False)
    for call, want in ((lambda: _call(M, N, G, args, nbytes), ref), (lambda: ops.linear(x, b, sb, N, False), y)):
        # (fails on the host: the runtime knows no such device)
        assert _cabi.lib.i4tc_gemm_grouped(a.data_ptr(), b.data_ptr(), sa.data_ptr(), sb.data_ptr(), ref.data_ptr(), M, N, 128, G,
                                           63, torch.cuda.current_stream().cuda_stream) > 0
        assert torch.equal(call(), want)
        assert _cabi.lib.i4tc_gemm_grouped_scratch_bytes(M, N, G, 0, dev) == nbytes
