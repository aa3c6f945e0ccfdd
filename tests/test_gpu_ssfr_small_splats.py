"""Few splats of a few pixels are drawn without the culling passes (csrc/kernels_ssfr.cu
ssfr_cull_setup): both sides of 2.5 pixels are bit for bit the oracle, and the smaller
ones take two launches less."""
import numpy as np
import pytest

from particles4all_b200 import _lib
from particles4all_b200.params import default_ssfr
from test_gpu_render_edges import block, camera  # noqa: F401  (block is a fixture)

pytestmark = pytest.mark.gpu


def test_both_sides_of_the_size(block):  # noqa: F811
    g, o = block
    cam = camera(320, 240, 30.0)
    dist = float(np.linalg.norm(np.array(cam["eye"][:3]) - 0.5 * np.array([40.0, 24.0, 20.0])))
    launches = []
    for px in (2.55, 2.45):
        sp = dict(default_ssfr(), **cam, splat_radius=px * dist / (cam["proj"][5] * 0.5 * 240) / 0.5)  # spacing 0.5
        before = _lib.lib().p4a_kernel_launches()
        g.ssfr(sp)
        launches.append(_lib.lib().p4a_kernel_launches() - before)
        o.ssfr(sp)
        for name in ("rawZ", "eyeZ", "thick", "image"):
            assert np.array_equal(g.ssfr_read(name), o.ssfr_read(name)), (px, name)
    assert launches[0] - launches[1] == 2, launches
