"""Wide tiles (256 .. 2048 cells per axis, three kernels per pass) against the oracle: every edge in x
and in y, both boundaries, grids below, at and just past one tile, odd sizes and 8-byte-aligned
grids, in-place calls, several passes with a shorter last one, and host slabs (open faces)."""
import numpy as np
import pytest

import flashfftstencil_b200 as ffs
import oracle
from tests.helpers import rel_errors, seeded_grid, seeded_weights

pytestmark = pytest.mark.gpu
TOL = 1e-12  # the FP64 forms' tolerance


def _solve(ext, T, boundary, radius=1, weights=None, form="auto", in_place=False, offset=0):
    import torch
    w = seeded_weights(2, radius, 3) if weights is None else weights
    plan = ffs.Plan(2, None, ext, T, weights=w, radius=radius, boundary=boundary, form=form)
    x = seeded_grid((ext[1], ext[0]), 4)
    buf = torch.empty(x.size + offset, dtype=torch.float64, device="cuda")
    d = buf[offset:].view(x.shape)
    d.copy_(torch.from_numpy(x))
    out = d if in_place else torch.full_like(d, float("nan"))
    plan.run(d, out)
    torch.cuda.synchronize()
    ref = oracle.run(x, w, radius, T, oracle.FIXED if boundary == "fixed" else oracle.PERIODIC)
    return plan, rel_errors(out.cpu().numpy(), ref)[0]


@pytest.mark.parametrize("boundary", ["fixed", "periodic"])
@pytest.mark.parametrize("edge", ["256x256", "512x256", "256x512", "1024x512", "512x1024", "2048x256", "256x2048"])
def test_every_edge_matches_the_oracle(monkeypatch, edge, boundary):
    monkeypatch.setenv("FFS_WIDE_TILE", edge)
    plan, err = _solve((333, 291), 17, boundary)
    assert plan.info["tile"] == int(edge.split("x")[0]) and plan.info["tau"] == 17
    assert err <= TOL


@pytest.mark.parametrize("boundary", ["fixed", "periodic"])
@pytest.mark.parametrize("ext,T,radius", [
    ((128, 128), 5, 1),    # the smallest sides
    ((226, 226), 15, 1),   # one tile of useful cells, to the cell (periodic)
    ((227, 453), 15, 1),   # one and two tiles and a cell
    ((511, 300), 40, 2),   # r tau of 80
    ((300, 260), 13, 3),   # radius without strip stepping: the band's boxes
])
def test_tile_remainders(monkeypatch, ext, T, radius, boundary):
    monkeypatch.setenv("FFS_WIDE_TILE", "256x256")
    plan, err = _solve(ext, T, boundary, radius)
    assert plan.info["tile"] == 256 and err <= TOL


@pytest.mark.parametrize("in_place,offset", [(True, 0), (False, 1), (True, 1)])
@pytest.mark.parametrize("T", [30, 250])  # one pass, several with a shorter last one
def test_in_place_and_unaligned(monkeypatch, T, in_place, offset):
    monkeypatch.setenv("FFS_WIDE_TILE", "256x256")
    plan, err = _solve((301, 277), T, "fixed", in_place=in_place, offset=offset)
    assert plan.info["tile"] == 256 and err <= TOL


@pytest.mark.parametrize("boundary", ["fixed", "periodic"])
def test_host_slabs_of_a_wide_grid(monkeypatch, boundary):
    monkeypatch.setenv("FFS_WIDE_TILE", "256x256")
    monkeypatch.setenv("FFS_HOST_SLABS", "3")
    w = seeded_weights(2, 1, 5)
    plan = ffs.Plan(2, None, (320, 900), 20, weights=w, radius=1, boundary=boundary, form="auto")
    assert plan.info["tile"] == 256 and plan.info["host_slabs"] == 3
    x = seeded_grid((900, 320), 6)
    ref = oracle.run(x, w, 1, 20, oracle.FIXED if boundary == "fixed" else oracle.PERIODIC)
    assert rel_errors(plan.run_host(x), ref)[0] <= TOL


def test_signed_weights_and_a_star(monkeypatch):
    monkeypatch.setenv("FFS_WIDE_TILE", "512x256")
    w = np.random.default_rng(2).standard_normal((5, 5))
    w /= np.abs(np.fft.fft2(w, s=(256, 256))).max()
    assert _solve((400, 350), 24, "periodic", 2, w)[1] <= TOL
    star = np.zeros((5, 5))
    star[2] = [0.1, 0.15, 0.3, 0.15, 0.1]
    star[:, 2] += [0.05, 0.05, 0.0, 0.05, 0.05]
    assert _solve((400, 350), 24, "fixed", 2, star)[1] <= TOL


def test_repeats_use_each_input(monkeypatch):
    """Calls on alternating buffers share the workspace: each result is its own input's, bit for bit."""
    import torch
    monkeypatch.setenv("FFS_WIDE_TILE", "256x256")
    plan = ffs.Plan(2, "Box2D9P", (300, 300), 20, boundary="fixed", form="auto")
    xs = [torch.from_numpy(seeded_grid((300, 300), k)).cuda() for k in range(2)]
    first = [plan.run(x).clone() for x in xs]
    streams = [torch.cuda.Stream() for _ in range(2)]
    torch.cuda.synchronize()
    outs = [torch.empty_like(x) for x in xs]
    for _ in range(4):
        for x, o, s in zip(xs, outs, streams):
            plan.run(x, o, stream=s)
    torch.cuda.synchronize()
    assert all(torch.equal(a, b) for a, b in zip(first, outs))


def _line(n, T, boundary, radius, in_place=False, offset=0):
    import torch
    w = seeded_weights(1, radius, 3)
    plan = ffs.Plan(1, None, (n,), T, weights=w, radius=radius, boundary=boundary, form="auto")
    x = seeded_grid((n,), 4)
    buf = torch.empty(n + offset, dtype=torch.float64, device="cuda")
    d = buf[offset:]
    d.copy_(torch.from_numpy(x))
    out = d if in_place else torch.full_like(d, float("nan"))
    plan.run(d, out)
    torch.cuda.synchronize()
    ref = oracle.run(x, w, radius, T, oracle.FIXED if boundary == "fixed" else oracle.PERIODIC)
    return plan, rel_errors(out.cpu().numpy(), ref)[0]


@pytest.mark.parametrize("boundary", ["fixed", "periodic"])
@pytest.mark.parametrize("edge", [1024, 2048, 4096])
@pytest.mark.parametrize("cells", [
    lambda e, u: e,              # the smallest line: the tile wraps around it once
    lambda e, u: e + 1,
    lambda e, u: 4 * u,          # whole pairs, to the cell (periodic)
    lambda e, u: 4 * u + 1,      # a tile with one cell, and no partner
    lambda e, u: 9 * e + 77,
])
def test_lines_in_wide_tiles(monkeypatch, cells, edge, boundary):
    monkeypatch.setenv("FFS_WIDE_TILE", str(edge))
    plan, err = _line(cells(edge, edge - 2 * 2 * 21), 21, boundary, 2)
    assert plan.info["tile"] == edge and plan.info["passes"] == 1 and err <= TOL


@pytest.mark.parametrize("n,T,radius,in_place,offset", [
    (30011, 85, 1, False, 1),   # boxes of 255 staged cells, 8-byte-aligned buffers
    (30011, 100, 1, True, 0),   # 300
    (30011, 170, 1, False, 0),  # 510
    (30011, 60, 3, True, 1),    # 540: past a warp's 16 cells a lane
    (30011, 40, 5, False, 0),   # a radius without a warp's path
    (7001, 900, 2, True, 0),    # several passes, the last one shorter
])
def test_boxes_beside_line_tiles(monkeypatch, n, T, radius, in_place, offset):
    monkeypatch.setenv("FFS_WIDE_TILE", "2048")
    plan, err = _line(n, T, "fixed", radius, in_place, offset)
    assert plan.info["tile"] == 2048 and err <= TOL


@pytest.mark.parametrize("form,tile", [("fp64", 0), ("fp64_fft", 64), ("fp64_fft", 128), ("ozaki", 0)])
@pytest.mark.parametrize("ext,T,radius,in_place,offset", [
    ((200, 150), 16, 1, False, 0),   # the shallowest frame of a short grid, two launches
    ((201, 149), 20, 1, True, 1),    # odd, in place, 8-byte aligned
    ((700, 324), 8, 1, False, 0),    # the shallowest of a long one, one launch
    ((131, 907), 4, 2, False, 1),
    ((310, 260), 33, 2, True, 0),    # several passes, the last one shorter
    ((90, 75), 32, 1, False, 0),     # the exact window is small, the strips overlap
])
def test_band_of_one_sm_tiles_on_a_frame(ext, T, radius, in_place, offset, form, tile):
    import torch
    w = seeded_weights(2, radius, 3)
    plan = ffs.Plan(2, None, ext, T, weights=w, radius=radius, boundary="fixed", form=form, tile=tile)
    x = seeded_grid((ext[1], ext[0]), 4)
    buf = torch.empty(x.size + offset, dtype=torch.float64, device="cuda")
    d = buf[offset:].view(x.shape)
    d.copy_(torch.from_numpy(x))
    out = d if in_place else torch.full_like(d, float("nan"))
    plan.run(d, out)
    torch.cuda.synchronize()
    assert rel_errors(out.cpu().numpy(), oracle.run(x, w, radius, T, oracle.FIXED))[0] <= TOL


def test_autotune_returns_a_count_for_one_sm_tiles():
    """A plan given the returned count runs that many steps a pass, whichever route was the fastest."""
    tau, ms = ffs.autotune(2, "Box2D25P", (1100, 1000), 120, boundary="periodic", form="auto", candidates=2)
    info = ffs.Plan(2, "Box2D25P", (1100, 1000), 120, boundary="periodic", form="auto", tau=tau).info
    assert info["tau"] == tau and info["tile"] in (64, 128) and ms > 0
