"""Direct stepping (marching warps and register-tile blocks) of 2-D grids against the oracle: every
step count of a launch and one past it, sizes around the kernels' strips and tiles, grids smaller than
the stencil's reach, both boundaries, in-place calls, 8-byte-aligned grids and host slabs."""
import numpy as np
import pytest

import flashfftstencil_b200 as ffs
import oracle
from tests.helpers import rel_errors, seeded_grid, seeded_weights

pytestmark = pytest.mark.gpu
TOL = 1e-12  # the FP64 forms' tolerance
SHAPES = ["Heat-2D", "Box2D9P", "Star2D9P", "Box2D25P"]


def _weights(shape):
    info = ffs.shape_info(shape)
    full = seeded_weights(2, info.radius, 9)
    keep = info.weights.reshape(full.shape) != 0.0
    w = np.where(keep, full, 0.0)
    return info.radius, w / w.sum()


def _check(monkeypatch, kernel, shape, ext, T, boundary, in_place=False, offset=0):
    import torch
    monkeypatch.setenv("FFS_DIRECT", kernel)
    r, w = _weights(shape)
    plan = ffs.Plan(2, shape, ext, T, weights=w, boundary=boundary, form="auto")
    assert plan.info["tiles"] == 1  # stepped directly
    x = seeded_grid((ext[1], ext[0]), 4)
    buf = torch.empty(x.size + offset, dtype=torch.float64, device="cuda")
    d = buf[offset:].view(x.shape)
    d.copy_(torch.from_numpy(x))
    out = d if in_place else torch.full_like(d, float("nan"))
    plan.run(d, out)
    torch.cuda.synchronize()
    ref = oracle.run(x, w, r, T, oracle.FIXED if boundary == "fixed" else oracle.PERIODIC)
    assert rel_errors(out.cpu().numpy(), ref)[0] <= TOL, (shape, ext, T, boundary)


@pytest.mark.parametrize("boundary", ["fixed", "periodic"])
@pytest.mark.parametrize("kernel", ["march", "blocks"])
@pytest.mark.parametrize("shape", SHAPES)
def test_every_step_count(monkeypatch, kernel, shape, boundary):
    for T in list(range(1, 10)) + [16, 17]:
        _check(monkeypatch, kernel, shape, (259, 141), T, boundary)


@pytest.mark.parametrize("boundary", ["fixed", "periodic"])
@pytest.mark.parametrize("kernel", ["march", "blocks"])
@pytest.mark.parametrize("ext", [(1, 1), (3, 5), (1, 70), (90, 2), (56, 56), (57, 64), (64, 65), (112, 120), (113, 119),
                                 (121, 8), (700, 9), (9, 700)])
def test_small_and_ragged_grids(monkeypatch, kernel, ext, boundary):
    _check(monkeypatch, kernel, "Box2D9P", ext, 4, boundary)
    _check(monkeypatch, kernel, "Star2D9P", ext, 4, boundary)


@pytest.mark.parametrize("kernel", ["march", "blocks"])
@pytest.mark.parametrize("T", [4, 12, 20])
def test_in_place_and_unaligned(monkeypatch, kernel, T):
    for boundary in ("fixed", "periodic"):
        _check(monkeypatch, kernel, "Box2D9P", (301, 203), T, boundary, in_place=True)
        _check(monkeypatch, kernel, "Box2D9P", (301, 203), T, boundary, offset=1)


@pytest.mark.parametrize("boundary", ["fixed", "periodic"])
@pytest.mark.parametrize("kernel", ["march", "blocks"])
def test_host_slabs(monkeypatch, kernel, boundary):
    """Slabs have open faces: no ring there, and rows beyond them do not count."""
    monkeypatch.setenv("FFS_DIRECT", kernel)
    monkeypatch.setenv("FFS_HOST_SLABS", "3")
    r, w = _weights("Star2D9P")
    plan = ffs.Plan(2, "Star2D9P", (130, 300), 6, weights=w, boundary=boundary, form="auto")
    assert plan.info["host_slabs"] == 3 and plan.info["tiles"] == 1
    x = seeded_grid((300, 130), 6)
    ref = oracle.run(x, w, r, 6, oracle.FIXED if boundary == "fixed" else oracle.PERIODIC)
    assert rel_errors(plan.run_host(x), ref)[0] <= TOL


def _check3(monkeypatch, shape, ext, T, boundary, in_place=False, offset=0):
    import torch
    monkeypatch.setenv("FFS_DIRECT", "march")
    full = seeded_weights(3, 1, 9)
    w = np.where(ffs.shape_info(shape).weights.reshape(full.shape) != 0.0, full, 0.0)
    w /= w.sum()
    plan = ffs.Plan(3, shape, ext, T, weights=w, boundary=boundary, form="auto")
    assert plan.info["tiles"] == 1
    x = seeded_grid(tuple(reversed(ext)), 4)
    buf = torch.empty(x.size + offset, dtype=torch.float64, device="cuda")
    d = buf[offset:].view(x.shape)
    d.copy_(torch.from_numpy(x))
    out = d if in_place else torch.full_like(d, float("nan"))
    plan.run(d, out)
    torch.cuda.synchronize()
    ref = oracle.run(x, w, 1, T, oracle.FIXED if boundary == "fixed" else oracle.PERIODIC)
    assert rel_errors(out.cpu().numpy(), ref)[0] <= TOL, (shape, ext, T, boundary)


@pytest.mark.parametrize("boundary", ["fixed", "periodic"])
@pytest.mark.parametrize("shape", ["Heat-3D", "Box3D27P"])
@pytest.mark.parametrize("ext", [(1, 1, 1), (3, 2, 5), (64, 32, 1), (65, 33, 2), (63, 31, 7), (130, 70, 40), (7, 200, 9)])
def test_3d_grids(monkeypatch, shape, ext, boundary):
    for T in (1, 2, 5):
        _check3(monkeypatch, shape, ext, T, boundary)


def test_3d_in_place_unaligned_and_slabs(monkeypatch):
    _check3(monkeypatch, "Box3D27P", (51, 40, 33), 3, "fixed", in_place=True)
    _check3(monkeypatch, "Heat-3D", (51, 40, 33), 4, "periodic", in_place=True, offset=1)
    monkeypatch.setenv("FFS_HOST_SLABS", "3")
    w = seeded_weights(3, 1, 2)
    x = seeded_grid((60, 30, 44), 6)
    for boundary in ("fixed", "periodic"):
        plan = ffs.Plan(3, "Box3D27P", (44, 30, 60), 4, weights=w, boundary=boundary, form="auto")
        assert plan.info["host_slabs"] == 3 and plan.info["tiles"] == 1
        ref = oracle.run(x, w, 1, 4, oracle.FIXED if boundary == "fixed" else oracle.PERIODIC)
        assert rel_errors(plan.run_host(x), ref)[0] <= TOL


@pytest.mark.parametrize("boundary", ["fixed", "periodic"])
@pytest.mark.parametrize("radius", [1, 2, 3, 4])
@pytest.mark.parametrize("n", [1, 5, 192, 193, 300, 5001, 100_003])
def test_lines(monkeypatch, n, radius, boundary):
    import torch
    monkeypatch.setenv("FFS_DIRECT", "march")
    w = seeded_weights(1, radius, 3)
    for T in (1, 7, 40, 230):  # 8 and 16 cells a lane, one launch and several
        plan = ffs.Plan(1, None, (n,), T, weights=w, radius=radius, boundary=boundary, form="auto")
        assert plan.info["tiles"] == 1
        x = seeded_grid((n,), T)
        buf = torch.empty(n + 1, dtype=torch.float64, device="cuda")
        d = buf[T % 2:T % 2 + n]  # every other one starts on an 8-byte boundary
        d.copy_(torch.from_numpy(x))
        out = d if T == 7 else torch.full_like(d, float("nan"))
        plan.run(d, out)
        torch.cuda.synchronize()
        ref = oracle.run(x, w, radius, T, oracle.FIXED if boundary == "fixed" else oracle.PERIODIC)
        assert rel_errors(out.cpu().numpy(), ref)[0] <= TOL, (n, radius, T, boundary)


def test_forms_and_edges_asked_for_by_name_keep_their_kernels(monkeypatch):
    monkeypatch.setenv("FFS_DIRECT", "march")
    for kw in ({"form": "fp64_fft"}, {"form": "fp64"}, {"form": "ozaki"}, {"form": "auto", "tile": 64}, {"form": "auto", "tau": 2}):
        assert ffs.describe(2, "Box2D9P", (300, 260), 4, boundary="fixed", **kw)["tiles"] > 1
