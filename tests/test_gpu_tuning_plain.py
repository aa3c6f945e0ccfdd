"""Every launch shape gives the same bits where it is used: the plain passes of scenes above
the sizes that a group of lanes per particle takes (csrc/api.cu group_lanes), lambda with
and without the prefetch of lists that come from DRAM, and the batched passes of frames on
both sides of that size."""
import re
from pathlib import Path

import numpy as np
import pytest

from particles4all_b200 import Batch, Sim, _lib, configs
from test_gpu_tuning import NAMES, force, need_gpu, run  # noqa: F401  (need_gpu restores the tables)

pytestmark = pytest.mark.gpu
GROUPED = int(re.search(r"kGroup8 = (\d+)", (Path(_lib.__file__).parent / "csrc" / "api.cu").read_text()).group(1))


def test_plain_shapes():
    p, sc = configs.medium_bodies_264k(side=28, n_cubes=2)  # tension on: the normals pass runs
    assert sc["pos"].shape[0] > GROUPED
    _lib.lib().p4a_tune_clear(-1)
    ref = run(p, sc, frames=2)
    for kernel in range(4):
        for v in range(1, 6):
            force(kernel, v)
            got = run(p, sc, frames=2)
            for k in ref:
                assert np.array_equal(np.asarray(ref[k]), np.asarray(got[k])), (kernel, v, k)


def large():
    p, sc = configs.dam_break_32k(side=85)  # 614,125 particles
    return dict(p, box=[130.0, 85.0, 85.0]), sc


def test_lambda_shapes_with_prefetch():
    p, sc = large()
    _lib.lib().p4a_tune_clear(-1)
    ref = None
    for v in range(6):
        force(0, v)
        s = Sim()
        s.reset_scene(p, sc)
        s.step(1 / 60)
        got = {k: s.read(k)[: sc["pos"].shape[0]].copy() for k in ("pos", "vel", "density", "lambda_")}
        s.close()
        ref = ref or got
        for k in ref:
            assert np.array_equal(ref[k], got[k]), (v, k)


@pytest.mark.parametrize("prefetch", [False, True])
def test_batched_shapes(prefetch):
    scenes = [configs.dam_break_32k(side=10), configs.medium_bodies_264k(side=28, n_cubes=2)]
    if prefetch:
        scenes.append(large())
    L = _lib.lib()
    ref = None
    for v in range(6):
        L.p4a_tune_clear(-1)
        for k in range(3):
            L.p4a_tune_set(k, 1 << 40, v)
        b = Batch(max_particles=700_000, max_cells=2_000_000, max_scenes=4)
        ids = [b.add_scene(p, sc) for p, sc in scenes]
        b.step(ids, 1 / 60)
        b.synchronize()
        got = [b.read(i, k)[: sc["pos"].shape[0]].copy() for i, (_, sc) in zip(ids, scenes) for k in NAMES[:5]]
        b.close()
        ref = ref or got
        for x, y in zip(ref, got):
            assert np.array_equal(x, y), v
    L.p4a_tune_clear(-1)
