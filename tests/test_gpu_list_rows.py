"""Neighbour lists built row by row with a bit per candidate (csrc/neighbours.cuh): rows of
a few to more than 64 candidates, lists that just fit and lists that overflow, next to
walls, with particles that move between the builds. A batch's passes have one thread per
particle at every size; bit for bit the oracle."""
import numpy as np
import pytest

from particles4all_b200 import Batch, Sim, configs
from test_gpu_batch import assert_same
from test_gpu_parity import compare, pair

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("spacing", [0.9, 0.5, 0.45, 0.41, 0.37, 0.35, 0.3])
@pytest.mark.parametrize("tension", [0.0, 0.5])
def test_row_lengths(spacing, tension):
    rng = np.random.default_rng(7)
    p = configs._base_params([10.0, 8.0, 9.0], iterations=4, tension=tension, xsph=0.01)
    at = 0.2 + np.arange(11) * spacing
    fluid = np.stack([a.ravel() for a in np.meshgrid(at, at, at, indexing="ij")], 1)
    fluid += rng.uniform(-0.02, 0.02, size=fluid.shape)
    sc = configs._assemble(fluid, [], p, configs.lattice_mass(0.5, 1.0))
    g, o = pair(p, sc)
    b = Batch(max_particles=fluid.shape[0], max_cells=1 << 16)
    sid = b.add_scene(p, sc)
    for _ in range(2):
        assert g.step(1 / 60) == o.step(1 / 60)
        b.step([sid], 1 / 60)
    assert_same(g, b, sid)
    if np.isfinite(o.buffer("pos")).all():  # see test_gpu_group_lanes.check
        compare(g, o)
    g.close()
    b.close()


@pytest.mark.parametrize("n", [20001, 20031])
def test_one_thread_per_particle_at_the_end_of_the_arrays(n):
    from test_gpu_parity import small_params
    g, o = pair(small_params(targetParticleCount=n, box=[1.0, 0.8, 0.8]))  # the scene fills its buffers
    for _ in range(2):
        assert g.step(1 / 60) == o.step(1 / 60)
    compare(g, o)
    g.close()


@pytest.mark.parametrize("side", [84, 85])
def test_both_sides_of_the_prefetched_lists(side):
    # 592,704 and 614,125 particles: in the batch lambda, alone delta never prefetches
    p, sc = configs.dam_break_32k(side=side)
    p = dict(p, box=[1.5 * side, side, side])
    g = Sim()
    g.reset_scene(p, sc)
    b = Batch(max_particles=side ** 3, max_cells=1 << 23)
    sid = b.add_scene(p, sc)
    for _ in range(2):
        g.step(1 / 60)
        b.step([sid], 1 / 60)
    assert_same(g, b, sid)
    g.close()
    b.close()

