"""ss_render refuses a camera that has no view plane, before anything is launched."""
import ctypes as C

import pytest

from smokesim_b200 import abi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pos,target,up", [
    ((0.5, 0.5, 0.5), (0.5, 0.5, 0.5), (0, 1, 0)),       # no direction
    ((0.5, 3.0, 0.5), (0.5, 0.5, 0.5), (0, 1, 0)),       # straight down, up along y
    ((0.5, 0.5, 2.0), (0.5, 0.5, 0.5), (0, 0, -3)),
    ((0.5, 0.5, 2.0), (0.5, 0.5, 0.5), (0, 0, 0)),
    ((0.5, 0.5, 1e30), (0.5, 0.5, 0.5), (0, 1, 0)),      # its length overflows
])
def test_camera_without_a_view_plane(pos, target, up):
    from smokesim_b200 import Sim
    g = Sim(abi.make_desc(3, (16, 16, 16), cell_size=1.0, density_channels=1, enclosed=1, min_coarse=4))
    d = g.render_desc(8, 8)
    for k in range(3):
        d.camera_pos[k], d.camera_target[k], d.camera_up[k] = pos[k], target[k], up[k]
    rgba = (C.c_uint8 * (8 * 8 * 4))()
    assert g.L.ss_render(g.h, C.byref(d), rgba, 0, None) == abi.SS_E_INVALID
    # 2D pictures have no camera: the same description is drawn
    q = Sim(abi.make_desc(2, (16, 16, 1), cell_size=1.0, density_channels=1, enclosed=1, min_coarse=4))
    assert q.L.ss_render(q.h, C.byref(d), rgba, 0, None) == abi.SS_OK
