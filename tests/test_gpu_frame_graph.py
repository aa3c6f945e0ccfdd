"""Frames that p4a_step replays as a graph: runs of equal frames long enough to be replayed,
broken by everything that changes what a frame launches (a drag, an impulse, appended
particles, a resized box, frames of other lengths, profiling, another stream, a new
scene), with an even and an odd number of substeps, stay bit for bit the oracle's; the
count of launches goes on as without graphs."""
import numpy as np
import pytest

from particles4all_b200 import Sim, _lib
from test_gpu_parity import compare, pair, small_params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("substeps", [1, 2, 3])
@pytest.mark.parametrize("n,tension", [(1500, 0.4), (9000, 0.0), (21000, 0.4)])
def test_runs_of_frames_with_changes_between(n, tension, substeps):
    import torch
    p = small_params(targetParticleCount=n, box=[1.0, 0.8, 0.8], bodies=["sphere:0.5", "box:1.4"], bodySize=0.05,
                     surfaceTensionK=tension, substeps=substeps, iterations=2, pour=True)
    g, o = pair(p)
    other = torch.cuda.Stream()

    def both(call, count=1):
        for _ in range(count):
            a, b = call(g), call(o)
        assert a == b

    frames = 6 if n < 20000 else 5
    both(lambda s: s.step(1 / 60), frames)
    both(lambda s: s.holdBody(1, [0.25, 0.3, 0.15], 10.0, 4.0))
    both(lambda s: s.step(1 / 60), 2)
    both(lambda s: s.releaseBody())
    both(lambda s: s.step(1 / 60), frames)
    both(lambda s: s.applyRayImpulse([0.0, 0.1, 0.15], [1.0, 0.0, 0.0], [3.0, 1.0, 0.0], 0.2, 2.0))
    g.set_stream(other.cuda_stream)
    both(lambda s: s.step(1 / 60), 2)
    pos3 = np.float32([[0.3, 0.6, 0.3], [0.4, 0.6, 0.4]])
    both(lambda s: s.appendFluid(pos3, 0 * pos3))
    both(lambda s: s.step(1 / 30), frames)
    g.profile(True)
    both(lambda s: s.step(1 / 60), 2)
    g.profile(False)
    both(lambda s: s.resizeBox([0.9, 0.8, 0.8]))
    both(lambda s: s.step(1 / 60), frames)
    compare(g, o)
    assert g.get_stats()["raw"] == o.stats()["raw"]
    g.reset(p)
    o.reset(p)
    both(lambda s: s.step(1 / 60), frames)
    compare(g, o)
    g.close()


def test_launches_are_counted_in_replays_too():
    s = Sim()
    s.reset(small_params(targetParticleCount=600))
    counts = []
    for _ in range(8):
        before = _lib.lib().p4a_kernel_launches()
        s.step(1 / 60)
        counts.append(_lib.lib().p4a_kernel_launches() - before)
    assert min(counts) == max(counts) > 0
    s.close()
