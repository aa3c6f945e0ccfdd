"""Scenes of a few particles, and of particles with hardly a neighbour, that stay finite: the
rest denominator is given, since a scene whose particles have no neighbours calibrates it
to 0. Groups, warps and lists that are nearly empty, with one thread per particle (the
batch) and with a group of lanes (a sim of its own): bit for bit the oracle."""
import numpy as np
import pytest

from particles4all_b200 import Batch, configs
from test_gpu_batch import assert_same
from test_gpu_parity import compare, pair

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tension", [0.0, 0.4])
@pytest.mark.parametrize("spacing", [0.45, 0.9])
@pytest.mark.parametrize("n", [1, 2, 7, 8, 9, 15, 16, 17, 31, 33, 129, 1331])
def test_few_neighbours(built, n, spacing, tension):
    rng = np.random.default_rng(7)
    p = configs._base_params([11.0, 8.0, 10.0], iterations=4, tension=tension, xsph=0.01)
    side = int(np.ceil(n ** (1 / 3)))
    at = 0.2 + np.arange(side) * spacing
    fluid = np.stack([a.ravel() for a in np.meshgrid(at, at, at, indexing="ij")], 1)[:n]
    fluid = fluid + rng.uniform(-0.02, 0.02, size=fluid.shape)
    sc = dict(configs._assemble(fluid, [], p, configs.lattice_mass(0.5, 1.0)), denom_rest=30.0)
    g, o = pair(p, sc)
    b = Batch(max_particles=4096, max_cells=1 << 16)
    sid = b.add_scene(p, sc)
    for _ in range(3):
        assert g.step(1 / 60) == o.step(1 / 60)
        b.step([sid], 1 / 60)
        assert np.isfinite(o.buffer("pos")).all()
        compare(g, o)
        assert_same(g, b, sid)
    g.close()
    b.close()
