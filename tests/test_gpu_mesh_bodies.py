"""Body particles take no part in the surface mesh's density field (src/mesh_wgsl.js:23-69),
wherever they are: at their places, far outside the box, at infinity and at NaN. Bit for
bit the oracle."""
import numpy as np
import pytest

from particles4all_b200 import configs
from particles4all_b200.params import default_mesh
from test_gpu_mesh import pair

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("at", [None, 1.0e30, np.inf, -np.inf, np.nan])
def test_body_particles_are_skipped(built, at):
    p, sc = configs.medium_bodies_264k(side=16, n_cubes=2)
    g, o = pair(p, sc, 2)
    if at is not None:
        n = g.info()["n"]
        pos = g.read("pos")[:n].copy()
        rows = np.flatnonzero(g.read("body")[:n, 0] > 0)[::3]
        pos[rows, 0] = at
        pos[rows[::2], 2] = at
        for s in (g, o):
            s.write("pos", pos)
    m = dict(default_mesh(), resolution=48)
    assert g.mesh(m) == o.mesh(m) > 0
    for name in ("meshField", "meshNField"):
        assert np.array_equal(g.read(name), o.buffer(name)), name
    g.close()
