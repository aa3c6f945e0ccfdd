"""The splats' depth pass on both sides of the distance from which they are no longer culled
(csrc/kernels_ssfr.cu): bit for bit the oracle."""
import numpy as np
import pytest

from particles4all_b200.params import default_ssfr
from test_gpu_render_edges import block, camera  # noqa: F401  (block is a fixture)

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("radii", [20.0, 269.0, 271.0, 400.0])
def test_distance_in_radii(block, radii):  # noqa: F811
    g, o = block
    cam = camera(320, 240, 30.0)
    dist = float(np.linalg.norm(np.array(cam["eye"][:3]) - 0.5 * np.array([40.0, 24.0, 20.0])))
    sp = dict(default_ssfr(), **cam, splat_radius=dist / radii / 0.5)  # spacing 0.5
    g.ssfr(sp)
    o.ssfr(sp)
    for name in ("rawZ", "eyeZ", "thick", "image"):
        assert np.array_equal(g.ssfr_read(name), o.ssfr_read(name)), name
