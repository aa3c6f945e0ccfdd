"""The neighbour passes with a group of lanes per particle (csrc/kernels_group.cu) on both
sides of the sizes at which a scene changes to 16, to 8 and to one lane per particle: bit
for bit the oracle, and bit for bit the batch, whose passes always have one thread per
particle. Odd particle counts leave the last group and block part empty; spacings outside
the ranges of the pair arithmetic take the IEEE operations; crowded particles overflow
their lists and take the direct walk; averaging divides by the neighbour count."""
import numpy as np
import pytest

from particles4all_b200 import Batch, configs
from test_gpu_batch import assert_same
from test_gpu_parity import compare, pair, small_params

pytestmark = pytest.mark.gpu


def check(p, scene=None, frames=2):
    g, o = pair(p, scene)
    b = Batch(max_particles=1 << 16, max_cells=1 << 20)
    sid = b.add_preset(p) if scene is None else b.add_scene(p, scene)
    for _ in range(frames):
        assert g.step(1 / 60) == o.step(1 / 60)
        b.step([sid], 1 / 60)
    assert_same(g, b, sid)
    # a few particles without tension can leave a substep with infinite positions, where the
    # oracle's clamp keeps a NaN and the device's does not; the batch has the device's clamp
    if np.isfinite(o.buffer("pos")).all():
        compare(g, o)
    g.close()
    b.close()


@pytest.mark.parametrize("n", [1, 9, 17, 6000, 6001, 20000, 20001])
@pytest.mark.parametrize("tension", [0.0, 0.4])
def test_both_sides_of_each_size(n, tension):
    box = [1.0, 0.8, 0.8] if n > 9999 else [0.8, 0.7, 0.6]  # room for all
    p = small_params(targetParticleCount=n, box=box, surfaceTensionK=tension)
    check(p, frames=1 if n > 9999 else 2)


@pytest.mark.parametrize("scale", [0.05, 1.0e4])
@pytest.mark.parametrize("n", [601, 6601])
def test_outside_the_ranges(n, scale):
    p = small_params(targetParticleCount=n, box=[b * scale for b in (0.8, 0.7, 0.6)], surfaceTensionK=0.4)
    check(dict(p, spacing=p["spacing"] * scale, gravity=p["gravity"] * scale))


@pytest.mark.parametrize("n", [1500, 7000])
@pytest.mark.parametrize("over", [dict(bodies=["sphere:0.5", "box:1.4"], bodySize=0.05), dict(noBoundary=True),
                                  dict(iterations=3, sorAverage=True, omega=1.2), dict(iterations=17, substeps=1)])
def test_options(n, over):
    check(small_params(targetParticleCount=n, box=[0.8, 0.7, 0.6], **over))


@pytest.mark.parametrize("sparse", [1500, 7000])
@pytest.mark.parametrize("tension", [0.0, 0.5])
def test_crowded_lists(sparse, tension):
    rng = np.random.default_rng(4)
    p = configs._base_params([12.0, 12.0, 12.0], iterations=4, tension=tension, xsph=0.01)
    at = np.arange(8) * 0.15
    dense = np.stack([a.ravel() for a in np.meshgrid(at, at, at, indexing="ij")], 1) + [3.0, 1.0, 3.0]
    loose = rng.uniform([5.0, 1.0, 1.0], [11.0, 11.0, 11.0], size=(sparse, 3))
    fluid = np.concatenate([dense, loose]) + rng.uniform(-0.005, 0.005, size=(512 + sparse, 3))
    check(p, configs._assemble(fluid, [], p, configs.lattice_mass(0.5, 1.0)))
