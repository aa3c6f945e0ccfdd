"""Scenes whose parameters lie outside the ranges of the pair arithmetic (pair_math_ranges)
take the IEEE operations, on list walks that load ahead as the others do. A dam break of
32,768 particles scaled to h = 2^-9 takes 1.40 times the time of the unscaled one; with one
dependent gather after another it took 1.82 times. Both are timed in turn, so that the
ratio does not depend on the clocks."""
import time

import numpy as np
import pytest

from particles4all_b200 import Sim, configs

pytestmark = pytest.mark.gpu


def scaled(params, scene, s):
    p = dict(params, spacing=params["spacing"] * s, box=[b * s for b in params["box"]], gravity=params["gravity"] * s)
    sc = dict(scene, mass=0.0, vel=scene["vel"] * np.float32(s), body_centre=scene["body_centre"] * s)
    for k in ("pos", "rest"):
        sc[k] = scene[k].copy()
        sc[k][:, :3] *= s
    return p, sc


def test_frames_outside_the_ranges_keep_the_load_ahead(built):
    scene = configs.dam_break_32k(0)
    sims = []
    for p, sc in (scene, scaled(*scene, 1 / 512)):
        s = Sim()
        s.reset_scene(p, sc)
        for _ in range(8):
            s.step(1 / 60)
        s.synchronize()
        sims.append(s)
    best = [1.0, 1.0]
    for _ in range(30):
        for k, s in enumerate(sims):
            t = time.perf_counter()
            s.step(1 / 60)
            s.synchronize()
            best[k] = min(best[k], time.perf_counter() - t)
    assert np.isfinite(sims[1].read("pos")).all()
    assert best[1] < 1.6 * best[0], best
    for s in sims:
        s.close()
