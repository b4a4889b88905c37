"""The plan builder's choice between the one-SM tiles, wide tiles and direct steps (describe(), no GPU)."""
import numpy as np
import pytest

import flashfftstencil_b200 as ffs


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
