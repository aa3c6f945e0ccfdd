"""The mesh scan's epochs are counted on the device, next to its ticket (csrc/kernels_grid.cu
k_scan): meshes before, at and after the wrap at 2^30 are the same triangles, bit for bit
the oracle's."""
import numpy as np
import pytest

from particles4all_b200 import _abi, _lib, configs
from particles4all_b200.params import default_mesh
from test_gpu_mesh import pair

pytestmark = pytest.mark.gpu


def test_meshes_around_the_wrap(built):
    p, sc = configs.dam_break_32k(side=12)
    g, o = pair(p, sc, 2)
    L = _lib.lib()
    assert L.p4a_test_mesh_epoch(g._h, 5) == _abi.P4A_ERR_STATE  # no mesh yet
    m = dict(default_mesh(), resolution=64)
    g.mesh(m)
    want = o.mesh(m)
    assert L.p4a_test_mesh_epoch(g._h, 0x40000000) == _abi.P4A_ERR_ARG
    assert L.p4a_test_mesh_epoch(g._h, 0x3ffffffd) == 0
    for k in range(5):
        assert g.mesh(m) == want > 0, k
        assert np.array_equal(g.read("meshVerts"), o.buffer("meshVerts").reshape(-1, 2)), k
    g.close()
