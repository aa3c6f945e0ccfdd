"""Shape matching (csrc/kernels_body.cu) for bodies of one particle to more than the block
keeps in registers (1,024), next to one another in a scene: bit for bit the oracle, alone
and in a batch (another block size)."""
import numpy as np
import pytest

from particles4all_b200 import Batch, configs
from test_gpu_batch import assert_same
from test_gpu_parity import compare, pair

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes", [(1, 2, 31, 33), (255, 256, 257), (511, 512, 513), (1023, 1024, 1025), (2049, 3, 1100)])
def test_body_sizes(sizes):
    d = 0.5
    rng = np.random.default_rng(sizes[0])
    p = configs._base_params([40.0, 20.0, 12.0], iterations=4, tension=0.0, xsph=0.01)
    at = np.arange(13) * d
    lattice = np.stack([a.ravel() for a in np.meshgrid(at, at, at, indexing="ij")], 1)
    bodies = [{"centre": np.array([5.0 + 9.0 * k, 9.0, 6.0]), "offsets": lattice[:m] - lattice[:m].mean(0),
               "density": 0.5 + 0.2 * k} for k, m in enumerate(sizes)]
    fluid = configs._fluid_lattice(60, 8, 18, d, 0.01 * d, rng, np.array([d, d, d]))
    sc = configs._assemble(fluid, bodies, p, configs.lattice_mass(d, 1.0))
    g, o = pair(p, sc)
    b = Batch(max_particles=1 << 16, max_cells=1 << 20)
    sid = b.add_scene(p, sc)
    for _ in range(3):
        assert g.step(1 / 60) == o.step(1 / 60)
        b.step([sid], 1 / 60)
    assert_same(g, b, sid)
    compare(g, o)
    for name in ("bodyCentre", "bodyRot"):
        assert np.array_equal(g.read(name), o.buffer(name)[: len(g.read(name))]), name
    g.close()
    b.close()
