"""The pair arithmetic without range tests (csrc/pair_math.cuh) against the oracle's IEEE
operations: lists of odd and even lengths with and without boundary samples inside the
ranges the host admits, and scenes outside them (spacing too small or too large, a
tension too weak), which take the IEEE operations one entry at a time. Bit for bit."""
import numpy as np
import pytest

from test_gpu_parity import compare, pair, small_params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scale", [1.0, 0.09, 0.11, 0.05, 6.0e3, 6.8e3, 1.0e4])
@pytest.mark.parametrize("tension", [0.0, 0.4, 1.0e-12])
def test_scenes_inside_and_outside_the_ranges(scale, tension):
    # h = 0.04 scale; the ranges end at h = 2^-8 (scale 0.098) and 2^8 (scale 6400)
    base = small_params(bodies=["sphere:0.5", "box:1.4"], bodySize=0.05, targetParticleCount=1500)
    p = dict(base, spacing=base["spacing"] * scale, box=[b * scale for b in base["box"]],
             bodySize=0.05 * scale, gravity=base["gravity"] * scale, surfaceTensionK=tension)
    g, o = pair(p)
    for _ in range(2):
        assert g.step(1 / 60) == o.step(1 / 60)
    compare(g, o)
    assert np.isfinite(g.read("pos")[:g.info()["n"]]).all()


@pytest.mark.parametrize("n", [1, 2, 31, 33, 257])
def test_few_particles(n):
    # lists of zero, one and a few entries, and warps that are not full
    g, o = pair(small_params(targetParticleCount=n, bodies=[], surfaceTensionK=0.4))
    for _ in range(3):
        assert g.step(1 / 60) == o.step(1 / 60)
    compare(g, o)
