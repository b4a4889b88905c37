"""Device memory of plans and batches: what creation uploads is there for a first run on any stream."""
import numpy as np
import pytest

import flashfftstencil_b200 as ffs
import oracle
from tests.helpers import rel_errors, seeded_grid, seeded_weights

pytestmark = pytest.mark.gpu
TOL = 1e-12  # the FP64 forms' tolerance


def test_first_run_on_a_stream_that_does_not_wait_for_the_legacy_one():
    """Plans of every kind of table (spectra, twiddles, band boxes, tensor-core operands), each run at once on a
    non-blocking stream, and a batch of the first ones: the upload has finished when creation returns."""
    import torch
    w = seeded_weights(2, 1, 3)
    x = seeded_grid((384, 512), 5)
    d = torch.from_numpy(x).cuda()
    ref = oracle.run(x, w, 1, 20, oracle.FIXED)
    streams = [torch.cuda.Stream() for _ in range(8)]
    torch.cuda.synchronize()
    kinds = [{"form": "fp64", "tau": 6}, {"form": "fp64_fft", "tile": 64}, {"form": "fp64_fft", "tile": 128, "tau": 20},
             {"form": "ozaki"}, {"form": "fp64_fft"}, {"form": "auto"}]
    for rep in range(3):
        outs, plans = [], []
        for k, kw in enumerate(kinds):
            out = torch.full_like(d, float("nan"))
            torch.cuda.synchronize()
            plans.append(ffs.Plan(2, None, (512, 384), 20, weights=w, radius=1, boundary="fixed", **kw))
            outs.append(plans[-1].run(d, out, stream=streams[k]))
        torch.cuda.synchronize()
        for kw, out in zip(kinds, outs):
            assert rel_errors(out.cpu().numpy(), ref)[0] <= TOL, kw
        outs = [torch.full_like(d, float("nan")) for _ in plans]
        torch.cuda.synchronize()
        batch = ffs.Batch(plans)
        batch.execute([d.data_ptr()] * len(plans), [o.data_ptr() for o in outs], streams[7].cuda_stream)
        torch.cuda.synchronize()
        for kw, out in zip(kinds, outs):
            assert rel_errors(out.cpu().numpy(), ref)[0] <= TOL, kw


def test_a_plan_without_room_for_wide_tiles_takes_the_one_sm_tiles():
    """Wide tiles hold a workspace beside the grid's: where it does not fit, the plan is made without them, and the
    failed allocation is not seen by its launches."""
    import torch
    ext, T = (2048, 2048), 32
    w = seeded_weights(2, 1, 3)

    def create():
        return ffs.Plan(2, None, ext, T, weights=w, radius=1, boundary="periodic", form="fp64_fft")
    x = seeded_grid(tuple(reversed(ext)), 5)
    d = torch.from_numpy(x).cuda()
    outs = [torch.full_like(d, float("nan")) for _ in range(2)]
    wide = create()
    wide.run(d, outs[0])
    torch.cuda.synchronize()
    assert wide.info["tile"] >= 256
    grid, need = x.nbytes, wide.info["work_bytes"]  # the one-SM tiles need the grid's workspace alone
    assert need > 2 * grid + (16 << 20)
    wide.close()
    small = ffs.Plan(2, None, ext, T, weights=w, radius=1, boundary="periodic", form="fp64_fft", tile=64)
    small.run(d, outs[1])  # (its kernels are loaded before the memory is gone)
    torch.cuda.synchronize()
    small.close()
    torch.cuda.empty_cache()
    leave = (grid + need) // 2
    fill = torch.empty(torch.cuda.mem_get_info()[0] - leave, dtype=torch.uint8, device="cuda")
    try:
        assert grid + (4 << 20) < torch.cuda.mem_get_info()[0] < need - (4 << 20)
        plan = create()
        outs[1].fill_(float("nan"))
        plan.run(d, outs[1])
        torch.cuda.synchronize()
        assert plan.info["tile"] in (64, 128) and plan.info["work_bytes"] == grid
    finally:
        del fill
        torch.cuda.empty_cache()
    again = create()
    assert again.info["tile"] == wide.info["tile"]
    ref = oracle.run(x, w, 1, T, oracle.PERIODIC)
    assert all(rel_errors(o.cpu().numpy(), ref)[0] <= TOL for o in outs)
