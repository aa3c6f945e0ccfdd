"""The ray pass on a field that the caller wrote (Sim.write): infinities, values so large that
their interpolation overflows and NaN, at a few vertices, at many and at all of them, where
the field's ranges and the quotients by the iso band (csrc/kernels_ray.cu) leave work out.
Bit for bit the oracle, through the field and on the mesh surface."""
import numpy as np
import pytest

import oracle
from particles4all_b200 import Sim, configs
from particles4all_b200.params import default_mesh, default_ray
from test_gpu_render_edges import camera

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def block(built):
    p, sc = configs.dam_break_32k(side=16)
    g, o = Sim(), oracle.OracleSim()
    for s in (g, o):
        s.reset_scene(p, sc)
        for _ in range(4):
            s.step(1 / 60)
        s.mesh(dict(default_mesh(), resolution=40))
    yield g, o, g.read("meshField").copy()
    g.close()


@pytest.mark.parametrize("use_surface", [0, 1])
@pytest.mark.parametrize("share", [0.001, 0.05, 1.0])
@pytest.mark.parametrize("value", [np.inf, -np.inf, np.nan, 3.0e38, 1.0e37, 1.0e6, 0.5, -5.0])
def test_values_in_the_field(block, value, share, use_surface):
    g, o, field = block
    f = field.copy()
    flat = f.reshape(-1)
    flat[np.random.default_rng(3).permutation(flat.size)[:max(1, int(share * flat.size))]] = value
    for s in (g, o):
        s.write("meshField", f)
    for debug in (0, 3):
        rp = dict(default_ray(), **camera(160, 121, 18.0), use_surface=use_surface, debug=debug)
        g.ray(rp)
        assert np.array_equal(g.ray_read(), o.ray(rp)), debug
