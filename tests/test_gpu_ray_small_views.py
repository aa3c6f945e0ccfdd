"""Small images of a coarse field are marched without the field's ranges (csrc/kernels_ray.cu
launch_ray): both sides of the image size and of the count of blocks are bit for bit the
oracle, and the ranges' launch is left out on one of them."""
import numpy as np
import pytest

from particles4all_b200 import _lib
from particles4all_b200.params import default_mesh, default_ray
from test_gpu_render_edges import block, camera  # noqa: F401  (block is a fixture)

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("resolution,w,h,launches", [
    (64, 320, 250, 1), (64, 321, 250, 2),  # 17 x 11 x 9 blocks, 80,000 pixels and more
    (72, 80, 61, 2), (24, 80, 61, 1)])     # 19 x 12 x 10 blocks
def test_both_sides_of_each_size(block, resolution, w, h, launches):  # noqa: F811
    g, o = block
    for s in (g, o):
        s.mesh(dict(default_mesh(), resolution=resolution))
    rp = dict(default_ray(), **camera(w, h, 18.0), use_surface=0)
    before = _lib.lib().p4a_kernel_launches()
    g.ray(rp)
    assert _lib.lib().p4a_kernel_launches() - before == launches
    assert np.array_equal(g.ray_read(), o.ray(rp))
