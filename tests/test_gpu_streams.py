"""Streams of the caller beside the library's own."""
import pytest

import flashfftstencil_b200 as ffs

pytestmark = pytest.mark.gpu


def test_a_batch_does_not_outrank_the_callers_streams():
    """A batch runs at the priority of the stream it is launched into: ten short kernels on a stream of higher
    priority, launched once the batch fills the GPU, do not wait for the batch's queued kernels."""
    import torch
    plans = [ffs.Plan(3, "Heat-3D", (256, 256, 256), 60, boundary="periodic", form="auto") for _ in range(4)]
    assert all(p.info["tiles"] == 1 for p in plans)  # 60 launches each, on branches of the graph
    ins = [torch.rand(256, 256, 256, dtype=torch.float64, device="cuda") for _ in plans]
    outs = [torch.empty_like(x) for x in ins]
    batch = ffs.Batch(plans)
    low, high = torch.cuda.Stream(priority=0), torch.cuda.Stream(priority=-1)
    x = torch.rand(1 << 23, device="cuda")
    torch.cuda.synchronize()
    shares = []
    for rep in range(6):
        start, batch_end, short_start, short_end = (torch.cuda.Event(enable_timing=True) for _ in range(4))
        start.record(low)
        batch.execute([t.data_ptr() for t in ins], [t.data_ptr() for t in outs], low.cuda_stream)
        batch_end.record(low)
        high.wait_event(start)
        with torch.cuda.stream(high):
            torch.cuda._sleep(2_000_000)  # some 1 ms: the batch's kernels are queued by then
            short_start.record(high)
            for _ in range(10):
                x.add_(1.0)
            short_end.record(high)
        torch.cuda.synchronize()
        if rep:  # (the first captures the graph)
            shares.append(short_start.elapsed_time(short_end) / start.elapsed_time(batch_end))
    # of the batch's 12 ms the ten kernels take 0.6 among the blocks in flight, 8 behind the batch's queue
    assert sorted(shares)[len(shares) // 2] < 0.3, shares
