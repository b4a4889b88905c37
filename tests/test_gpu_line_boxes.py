"""The fixed boundary's boxes beside 1-D wide tiles, at the limits of their kernels: the box at a face is r tau
cells, with as many staged beyond it.  Up to 256 staged cells a warp steps 8 a lane, up to 512 it steps 16, past
that a block steps them through shared memory."""
import pytest

import flashfftstencil_b200 as ffs
import oracle
from tests.helpers import rel_errors, seeded_grid, seeded_weights

pytestmark = pytest.mark.gpu
TOL = 1e-12  # the FP64 forms' tolerance


@pytest.mark.parametrize("in_place,offset", [(False, 1), (True, 0)])  # (offset: 8-byte-aligned buffers)
@pytest.mark.parametrize("staged,past", [(256, 0), (256, 1), (512, 0), (512, 1)])
@pytest.mark.parametrize("radius", [1, 2, 3, 4])
def test_staged_sizes(monkeypatch, radius, staged, past, in_place, offset):
    import torch
    monkeypatch.setenv("FFS_WIDE_TILE", "2048")
    n, tau = 7001, staged // (2 * radius) + past
    w = seeded_weights(1, radius, 3)
    # (deep boxes cost more than the passes they save: only runs too long for eight shallower passes come to them)
    T = tau if (staged, past) == (256, 0) else 8 * tau
    plan = ffs.Plan(1, None, (n,), T, weights=w, radius=radius, boundary="fixed", form="auto")
    assert plan.info["tile"] == 2048
    cells = 2 * radius * plan.info["tau"]
    low, high = {(256, 0): (0, 256), (512, 1): (512, 2048)}.get((staged, past), (256, 512))
    assert low < cells <= high
    x = seeded_grid((n,), 4)
    buf = torch.empty(n + offset, dtype=torch.float64, device="cuda")
    d = buf[offset:]
    d.copy_(torch.from_numpy(x))
    out = d if in_place else torch.full_like(d, float("nan"))
    plan.run(d, out)
    torch.cuda.synchronize()
    assert rel_errors(out.cpu().numpy(), oracle.run(x, w, radius, T, oracle.FIXED))[0] <= TOL


@pytest.mark.parametrize("form", ["fp64", "fp64_fft"])
@pytest.mark.parametrize("staged,past", [(256, 0), (256, 1), (512, 0), (512, 1)])
@pytest.mark.parametrize("radius", [1, 4, 5])
def test_staged_sizes_beside_one_sm_tiles(radius, staged, past, form):
    """The band kernel's own launch, with the 4096-cell tile and the step count by name; radius 5 has no warp's path."""
    import torch
    n, tau = 9001, staged // (2 * radius) + past
    T = 2 * tau + 1  # and a short last pass
    w = seeded_weights(1, radius, 3)
    plan = ffs.Plan(1, None, (n,), T, weights=w, radius=radius, boundary="fixed", form=form, tile=4096, tau=tau)
    assert plan.info["tile"] == 4096 and plan.info["tau"] == tau
    x = seeded_grid((n,), 4)
    d = torch.from_numpy(x).cuda()
    out = torch.full_like(d, float("nan"))
    plan.run(d, out)
    torch.cuda.synchronize()
    assert rel_errors(out.cpu().numpy(), oracle.run(x, w, radius, T, oracle.FIXED))[0] <= TOL
