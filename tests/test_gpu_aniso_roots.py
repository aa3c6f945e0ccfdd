"""The anisotropic pass's root without range tests (csrc/kernels_misc.cu), on both sides of
the radii it is used for, with particles that coincide and particles less than 1e-19
apart (their weight is 1 whatever the root), rows of every remainder of four: bit for bit
the oracle."""
import numpy as np
import pytest

from particles4all_b200 import configs
from test_gpu_parity import pair, small_params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("radius_scale", [1.0e-10, 2.0e-9, 3.0e-9, 1.0e-3, 0.7, 1.0, 2.0, 3.0])
@pytest.mark.parametrize("n", [1, 3, 500, 1501])
def test_aniso_radii(n, radius_scale):
    g, o = pair(small_params(targetParticleCount=n, bodies=[], surfaceTensionK=0.4))
    if n >= 500:  # the oracle's step of a few particles ends in NaN (test_gpu_group_lanes.check)
        for s in (g, o):
            s.step(1 / 60)
    n = g.info()["n"]
    pos = g.read("pos")[:n].copy()
    pos[: min(n, 4), :3] = np.float32([[0, 0, 0], [1.0e-20, 0, 0], [0, 3.0e-12, 0], [0, 0, 0]])[: min(n, 4)]
    a = dict(configs.medium_aniso_params(), radius_scale=radius_scale)
    for moved in (False, True):
        if moved:
            g.write("pos", pos)
            o.write("pos", pos)
        for s in (g, o):
            s.aniso(a)
        for name, count in (("smoothPos", n), ("aniso", 2 * n)):
            assert np.array_equal(g.read(name)[:count], o.buffer(name)[:count], equal_nan=True), (name, moved)
    g.close()
