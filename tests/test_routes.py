"""The plan builder's choice between the one-SM tiles, wide tiles and direct steps (describe(), no GPU)."""
import os
import subprocess
import sys
import time

import numpy as np
import pytest

import flashfftstencil_b200 as ffs

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _direct(info):
    """Direct steps report one tile a pass; these grids take several of any other kind."""
    return info["tiles"] == 1


@pytest.mark.parametrize("axis", [0, 1, 2])
def test_direct_steps_in_3d_stop_below_2_to_the_30(monkeypatch, axis):
    """The 3-D kernel marks an open face with a coordinate of 2^30: cells past it would be held."""
    monkeypatch.setenv("FFS_DIRECT", "march")
    ext = [1, 1, 1]
    for n, direct in ((2 ** 30 - 1, True), (2 ** 30, False)):
        ext[axis] = n
        info = ffs.describe(3, "Heat-3D", tuple(ext), 4, boundary="fixed", form="auto", open_faces=3 << (2 * axis))
        assert _direct(info) == direct, (ext, info)


@pytest.mark.parametrize("radius", [7, 8])
@pytest.mark.parametrize("boundary", ["fixed", "periodic"])
def test_radius_without_room_in_a_16_tile(radius, boundary):
    """Halos of 8 cells fill a 16^3 tile: that edge is refused, the open choice takes 32^3."""
    w = np.full((2 * radius + 1,) * 3, 1.0 / (2 * radius + 1) ** 3)
    kw = {"weights": w, "radius": radius, "boundary": boundary}
    for tau in (0, 1):
        info = ffs.describe(3, None, (60, 50, 40), 2, form="auto", tau=tau, **kw)
        assert info["tile"] == 32 and info["useful"] == 16 and info["tau"] == 1
        for refused in ({"form": "auto", "tile": 16}, {"form": "fp64"}, {"form": "ozaki"}, {"form": "bf16x3"}):
            with pytest.raises(ffs.FFSError) as e:
                ffs.describe(3, None, (60, 50, 40), 2, tau=tau, **refused, **kw)
            assert e.value.status == ffs.ERR_UNSUPPORTED


# (dim, shape, extents, T, boundary), and the class as the table names it
VOLUME = (3, "Box3D27P", (512, 512, 512), 16, "fixed")
PLATE = (2, "Box2D9P", (4096, 4096), 32, "periodic")
SMALL = (2, "Box2D9P", (100, 100), 40, "periodic")  # below the wide tiles' least side
VOLUME_CLASS = "f4.d3.r1.k27.b1.o0.T16.n9_9_9"
PLATE_CLASS = "f4.d2.r1.k9.b0.o0.T32.n12_12_0"
SMALL_CLASS = "f4.d2.r1.k9.b0.o0.T40.n7_7_0"


def _routes(table, tmp_path):
    """Route ("tiles", "wide", "direct") of each grid for both forms, by a process with this table."""
    cache = tmp_path / "table"
    cache.write_text("".join(line + "\n" for line in table))
    code = ("import sys; sys.path.insert(0, %r); import flashfftstencil_b200 as f\n"
            "for g in %r:\n"
            "    for form in ('auto', 'fp64_fft'):\n"
            "        i = f.describe(*g[:4], boundary=g[4], form=form)\n"
            "        wide = i['tile'] >= 256\n"
            "        print('wide' if wide else 'direct' if i['tiles'] == 1 else 'tiles')" %
            (ROOT, [VOLUME, PLATE, SMALL]))
    env = {k: v for k, v in os.environ.items() if not k.startswith("FFS_")}
    r = subprocess.run([sys.executable, "-c", code], env=dict(env, FFS_TUNE_CACHE=str(cache)), capture_output=True, text=True,
                       timeout=300)
    assert r.returncode == 0, r.stderr
    got = r.stdout.split()
    return {name: tuple(got[2 * k:2 * k + 2]) for k, name in enumerate(("volume", "plate", "small"))}


MODEL = {"volume": ("direct", "tiles"), "plate": ("wide", "wide"), "small": ("tiles", "tiles")}


@pytest.mark.parametrize("table,changed", [
    ([], {}),
    # a measured one-SM edge ranks the edges only: it was not timed against the other routes
    (["E." + VOLUME_CLASS + " 16", "E." + PLATE_CLASS + " 128"], {}),
    # entries of either form's tuning by an earlier version, whose key did not tell them apart
    (["E." + VOLUME_CLASS + " 2", "E." + PLATE_CLASS + " 2"], {}),
    # each form's measured route is its own
    (["RA." + VOLUME_CLASS + " 3"], {"volume": ("tiles", "tiles")}),
    (["R." + VOLUME_CLASS + " 3", "R." + PLATE_CLASS + " 3"], {"plate": ("wide", "tiles")}),
    (["RA." + PLATE_CLASS + " 2"], {"plate": ("direct", "wide")}),
    (["RA." + PLATE_CLASS + " 3", "R." + PLATE_CLASS + " 1"], {"plate": ("tiles", "wide")}),
    # a route that the form may not take, or that does not fit this grid of the class: the model's
    (["R." + PLATE_CLASS + " 2", "RA." + SMALL_CLASS + " 1", "R." + SMALL_CLASS + " 1"], {}),
])
def test_tuned_routes_of_the_two_forms(table, changed, tmp_path):
    """(auto, fp64_fft by name): tuning one form leaves the other's choice alone."""
    assert _routes(table, tmp_path) == dict(MODEL, **changed)


@pytest.mark.parametrize("dim,shape,ext", [(1, "Heat-1D", (10_000,)), (2, "Heat-2D", (300, 260)), (2, "Box2D25P", (300, 260))])
def test_plans_for_very_many_steps_are_made_at_once(dim, shape, ext):
    """The step counts looked at are bounded by the kernels' most steps a launch, not by T (9 s for 10^9 steps
    when every pass count was)."""
    start = time.perf_counter()
    for boundary in ("fixed", "periodic"):
        info = ffs.describe(dim, shape, ext, 10 ** 9, boundary=boundary, form="auto")
        assert (info["passes"] - 1) * info["tau"] + info["tau_last"] == 10 ** 9
    assert time.perf_counter() - start < 0.2  # 1 to 10 ms


@pytest.mark.parametrize("form", ["auto", "fp64_fft"])
@pytest.mark.parametrize("edge", [0, 64, 128])
def test_slab_passes_are_those_of_the_one_sm_tiles(edge, form, tmp_path):
    """A decomposed solve takes the tuned edge's step counts, or the modelled edge's, whatever the route of one
    grid; in 1-D those of the 4096-cell tile."""
    cache = tmp_path / "table"
    cache.write_text("E.%s %d\n" % (PLATE_CLASS, edge) if edge else "")
    code = ("import sys; sys.path.insert(0, %r)\n"
            "import flashfftstencil_b200 as f\n"
            "from flashfftstencil_b200.slab import SlabPlan\n"
            "for g, tile in ((%r, %r), ((1, 'Heat-1D', (1 << 20,), 500, 'fixed'), 4096)):\n"
            "    p = SlabPlan(*g[:4], boundary=g[4], rank=1, world=4, form=%r)\n"
            "    i = f.describe(*g[:4], boundary=g[4], form=%r, tile=tile)\n"
            "    print([q.tau for q in p.passes] == [i['tau']] * (i['passes'] - 1) + [i['tau_last']])" %
            (ROOT, PLATE, edge or 128, form, form))
    env = {k: v for k, v in os.environ.items() if not k.startswith("FFS_")}
    r = subprocess.run([sys.executable, "-c", code], env=dict(env, FFS_TUNE_CACHE=str(cache)), capture_output=True, text=True,
                       timeout=300)
    assert r.returncode == 0, r.stderr
    assert r.stdout.split() == ["True", "True"]


@pytest.mark.parametrize("shape,ext,T,slabs", [("Box3D27P", (200, 180, 160), 10, 4), ("Heat-3D", (200, 208, 170), 13, 3)])
def test_host_slabs_of_direct_steps_are_not_charged_the_tiles_passes(shape, ext, T, slabs):
    """A slab's pass of one direct step has no band to wait for: with the tiles' 25 us a pass these grids went in one
    slab less or half of them (Box3D27P 1908 us, 1590 in four slabs, 1727 in four on the tiles)."""
    info = ffs.describe(3, shape, ext, T, boundary="fixed", form="auto")
    assert _direct(info) and info["host_slabs"] == slabs


@pytest.mark.parametrize("form", ["auto", "fp64_fft"])
@pytest.mark.parametrize("n,T,radius", [(3_416, 458, 7), (188_069, 134, 8), (893_929, 268, 7), (91_237, 1_838, 7),
                                        (1_259_431, 1_146, 2), (2_437_720, 820, 3)])
def test_lines_do_not_pay_for_deep_boxes_with_few_passes(n, T, radius, form):
    """A block's step of the box at a face costs with its cells and taps (0.4 to 3.6 us, where 0.5 was modelled): boxes of
    1600 to 3800 staged cells took 1.6 to 4 times as long as the one-SM tiles' solve (188069 cells, radius 8, T = 134
    in one pass 335 us, in three 122)."""
    w = np.full(2 * radius + 1, 1.0 / (2 * radius + 1))
    info = ffs.describe(1, None, (n,), T, weights=w, radius=radius, boundary="fixed", form=form)
    assert 2 * radius * info["tau"] <= 1024


@pytest.mark.parametrize("shape,ext,T,boundary,us", [
    ("Heat-2D", (4130, 5900), 1, "fixed", 85), ("Heat-2D", (4130, 5900), 4, "fixed", 108),
    ("Box2D9P", (4130, 5900), 1, "periodic", 83), ("Star2D9P", (4130, 5900), 2, "fixed", 98),
    ("Box2D25P", (4130, 5900), 1, "fixed", 100), ("Box2D25P", (3390, 1840), 1, "fixed", 31),
    ("Box2D9P", (1047, 1415), 1, "periodic", 8.5), ("Heat-2D", (300, 260), 12, "fixed", 13.7),
])
def test_the_model_of_few_steps_holds_on_large_grids(shape, ext, T, boundary, us):
    """Measured on a B200.  The block kernel's tiles were modelled without their loads and stores after the first wave:
    it took one step of 4130 x 5900 cells in 162 to 218 us, modelled 42 to 92."""
    info = ffs.describe(2, shape, ext, T, boundary=boundary, form="auto")
    assert _direct(info) and us / 1.3 < info["model_ms"] * 1e3 < us * 1.3


@pytest.mark.parametrize("shape,ext,T", [("Heat-2D", (184, 246), 7), ("Box2D25P", (174, 176), 4)])
def test_small_fixed_grids_stay_on_one_sm_tiles(shape, ext, T):
    """fp64_fft by name, a single wave whose boxes run beside it: 9.0 and 10.6 us, on wide tiles 13.2 and 13.0."""
    assert ffs.describe(2, shape, ext, T, boundary="fixed", form="fp64_fft")["tile"] == 64


@pytest.mark.parametrize("radius,ext,T", [(7, (874, 938), 33), (7, (1774, 1392), 3), (3, (314, 340), 6), (3, (1270, 916), 34)])
def test_wide_tiles_do_not_take_deep_boxes_for_few_passes(radius, ext, T):
    """From radius 3 on the band of a wide pass goes by boxes: past 2048 staged cells they took several times what was
    modelled (radius 7, 874 x 938, T = 33 2728 us in eleven wide passes, 1250 on 64 x 64 tiles)."""
    w = np.full((2 * radius + 1,) * 2, 1.0 / (2 * radius + 1) ** 2)
    info = ffs.describe(2, None, ext, T, weights=w, radius=radius, boundary="fixed", form="fp64_fft")
    depth = radius * info["tau"]
    assert info["tile"] < 256 or 2 * depth * (32 + 2 * depth) <= 2048  # (a box at a face stages two depths of it)
