"""The plan builder's choice between the one-SM tiles, wide tiles and direct steps (describe(), no GPU)."""
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
