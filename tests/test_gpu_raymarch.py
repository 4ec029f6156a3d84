"""The ray marcher where its batches and tiles end: odd numbers of shadow samples,
pictures that are no multiple of a tile, boxes that are no cube, light along an
axis so that the shadow march leaves the box early, and smoke up to the walls."""
import numpy as np
import pytest

from smokesim_b200 import abi, scene
from test_gpu_render import _close

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,nch", [((24, 40, 17), 1), ((33, 16, 20), 3)])
@pytest.mark.parametrize("shadow,light", [(0, (1, 1, 1)), (1, (0, 1, 0)), (5, (-1, 0.5, 0)), (8, (0.2, -1, 0.4))])
def test_raymarch_edges(n, nch, shadow, light):
    from oracle.oracle import OracleSim
    from smokesim_b200 import Sim
    desc = abi.make_desc(3, n, cell_size=1.0, density_channels=nch, enclosed=1, min_coarse=4)
    g, o = Sim(desc), OracleSim(desc)
    a = scene.random_state(scene.Rng(5), 3, n, nch)[abi.FIELD_DENSITY][: int(np.prod(g.shape(abi.FIELD_DENSITY)))]
    a = np.abs(a) * np.float32(0.1)
    for s in (g, o):
        s.set_field(abi.FIELD_DENSITY, a)
    d = g.render_desc(61, 37)
    d.shadow_steps = shadow
    for k in range(3):
        d.light_direction[k] = light[k]
    img = g.render(d)
    assert img[..., 3].max() > 0
    _close(img, o.render(d))
