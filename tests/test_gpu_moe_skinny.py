"""GPU: the weight-streaming form of the grouped MoE GEMM gives the tile kernel's bits at the edges of its row tiles (8, 16 and 32
rows at once, experts without rows, experts that take several passes), of its blocks (N below, at and past 128 rows) and of its
pipeline (fewer groups than it keeps in flight, odd counts), and from several threads."""
import statistics
import threading

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("E,counts", [
    (1, [1]), (4, [0, 5, 0, 8]), (16, [1, 9, 0, 17, 3]),              # 8 rows at once, up to three passes
    (4, [16, 0, 33, 1]), (3, [12, 12, 12]),                            # 16 at once
    (4, [32, 31, 40, 1]), (2, [0, 52]),                                # 32 at once, the most rows per expert it takes
    (70, [1] * 33 + [100] + [0] * 30 + [9, 8, 7] + [0] * 2 + [200]),   # passes of experts in three runs of 32
    (100, [0] * 40 + [2600]),                                          # more passes than there are blocks to take them
])
@pytest.mark.parametrize("N,G", [(16, 1), (112, 2), (128, 3), (144, 16), (2048, 6)])
def test_same_bits_as_the_tile_kernel(E, counts, N, G):
    from fp8_inference_toolkit_b200 import moe, ops

    counts = counts + [0] * (E - len(counts))
    P = sum(counts)
    assert 0 < P <= 26 * E
    gen = torch.Generator(device="cuda").manual_seed(P + N + G)
    a = torch.randint(0, 256, (G, P, 64), dtype=torch.uint8, device="cuda", generator=gen)
    b = torch.randint(0, 256, (E, G, N, 64), dtype=torch.uint8, device="cuda", generator=gen)
    sa = torch.rand(G, P, device="cuda", generator=gen) * 0.1 + 1e-3
    sb = torch.rand(E, G, N, device="cuda", generator=gen) * 0.01 + 1e-4
    off = torch.tensor([sum(counts[:e]) for e in range(E + 1)], dtype=torch.int32, device="cuda")
    outs = []
    for path in (3, 0):
        ops.set_small_m_path(path)
        try:
            out = torch.full((P, N), float("nan"), dtype=torch.bfloat16, device="cuda")
            moe.moe_w4a4_grouped_gemm(a, sa, b, sb, off, out, N, G, E)
        finally:
            ops.set_small_m_path(0)
        outs.append(out)
    assert not outs[0].isnan().any()
    assert torch.equal(outs[0], outs[1])
    ops.check_status()


def test_threads_with_other_group_counts():
    """The kernel's shared-memory limit belongs to the function: a call with few groups must not lower it under a thread that is about
    to launch with many (such a launch is refused)."""
    from fp8_inference_toolkit_b200 import moe, ops

    E, P, N = 4, 80, 128
    off = torch.tensor([0, 20, 40, 60, 80], dtype=torch.int32, device="cuda")
    gen = torch.Generator(device="cuda").manual_seed(3)
    jobs, codes = [], []
    for G in (1, 24, 1, 24):     # 4 KB and 101 KB of shared memory at 32 rows at once
        a = torch.randint(0, 256, (G, P, 64), dtype=torch.uint8, device="cuda", generator=gen)
        b = torch.randint(0, 256, (E, G, N, 64), dtype=torch.uint8, device="cuda", generator=gen)
        sa, sb = torch.rand(G, P, device="cuda", generator=gen), torch.rand(E, G, N, device="cuda", generator=gen)
        want = torch.empty(P, N, dtype=torch.bfloat16, device="cuda")
        moe.moe_w4a4_grouped_gemm(a, sa, b, sb, off, want, N, G, E)
        out, stream = torch.empty_like(want), torch.cuda.Stream()
        jobs.append((a, sa, b, sb, G, want, out, stream))
    torch.cuda.synchronize()

    def work(a, sa, b, sb, G, want, out, stream):   # nothing but library calls, which run beside each other
        args = (a.data_ptr(), sa.data_ptr(), b.data_ptr(), sb.data_ptr(), off.data_ptr(), out.data_ptr(), P, N, G, E, 0, stream.cuda_stream)
        codes.append({ops.lib.i4tc_moe_grouped_gemm(*args) for _ in range(20000)})

    threads = [threading.Thread(target=work, args=j) for j in jobs]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    assert codes == [{0}] * len(jobs)
    for j in jobs:
        assert torch.equal(j[6], j[5])
    ops.check_status()


@pytest.mark.parametrize("rows_each", [1600, 200])
def test_rows_of_few_experts_run_side_by_side(rows_each):
    """All rows on one expert, or on eight of 64: no slower than twice the tile kernel, which spreads them over the device (a
    block that takes an expert's rows pass by pass needs several times as long)."""
    from fp8_inference_toolkit_b200 import moe, ops

    E, N, G, P = 64, 1536, 16, 1600
    gen = torch.Generator(device="cuda").manual_seed(rows_each)
    counts = [rows_each if e < P // rows_each else 0 for e in range(E)]
    a = torch.randint(0, 256, (G, P, 64), dtype=torch.uint8, device="cuda", generator=gen)
    b = torch.randint(0, 256, (E, G, N, 64), dtype=torch.uint8, device="cuda", generator=gen)
    sa, sb = torch.rand(G, P, device="cuda", generator=gen), torch.rand(E, G, N, device="cuda", generator=gen)
    off = torch.tensor([sum(counts[:e]) for e in range(E + 1)], dtype=torch.int32, device="cuda")
    out = torch.empty(P, N, dtype=torch.bfloat16, device="cuda")
    times = []
    for path in (3, 0):
        ops.set_small_m_path(path)
        try:
            took = []
            for _ in range(12):
                start, end = (torch.cuda.Event(enable_timing=True) for _ in range(2))
                start.record()
                for _ in range(10):
                    moe.moe_w4a4_grouped_gemm(a, sa, b, sb, off, out, N, G, E)
                end.record()
                end.synchronize()
                took.append(start.elapsed_time(end))
        finally:
            ops.set_small_m_path(0)
        times.append(statistics.median(took[2:]))
    assert times[1] < 2 * times[0], times
