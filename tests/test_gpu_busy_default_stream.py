"""New device buffers are cleared and filled on the streams that use them: with a program's
work keeping the default stream busy, a new handle's first mesh, an environment and a new
batch's first frames come out as ever. (Cleared on the default stream, they would be
zeroed when that work ends, after what had been written to them by then.)"""
import numpy as np
import pytest

import oracle
from particles4all_b200 import Batch, Sim, configs
from particles4all_b200.params import default_mesh
from test_gpu_batch import assert_same
from test_gpu_env import panorama
from test_gpu_mesh import pair

pytestmark = pytest.mark.gpu


@pytest.fixture
def busy(built):
    import torch
    torch.cuda.init()
    yield lambda: torch.cuda._sleep(400_000_000)  # about 0.2 s of the default stream
    torch.cuda.synchronize()


def test_first_mesh(busy):
    p, sc = configs.dam_break_32k(side=12)
    g, o = pair(p, sc, 2)
    m = dict(default_mesh(), resolution=64)
    want = o.mesh(m)
    busy()
    for _ in range(2):
        assert g.mesh(m) == want > 0
        assert np.array_equal(g.read("meshVerts"), o.buffer("meshVerts").reshape(-1, 2))
    g.close()


def test_environment(busy):
    g, o = Sim(), oracle.OracleSim()
    rgb = panorama(160, 80)
    o.set_environment(rgb)
    busy()
    g.set_environment(rgb)
    assert np.array_equal(g.environment(), o.environment())
    g.close()


@pytest.mark.parametrize("lanes", [1, 2])
def test_new_batch(busy, lanes):
    import torch
    scenes = [configs.dam_break_32k(side=10), configs.medium_bodies_264k(side=12, n_cubes=2)]
    sims = []
    for p, sc in scenes:
        s = Sim()
        s.reset_scene(p, sc)
        for _ in range(2):
            s.step(1 / 60)
        sims.append(s)
    busy()
    b = Batch(max_particles=50_000, max_cells=200_000, max_scenes=4)
    b.set_lanes(lanes, 0)
    ids = [b.add_scene(p, sc) for p, sc in scenes]
    for _ in range(2):
        b.step(ids, 1 / 60)
    b.synchronize()
    torch.cuda.synchronize()
    for s, sid in zip(sims, ids):
        assert_same(s, b, sid)
        s.close()
    b.close()
