"""The render passes' shortcuts at their edges, bit for bit against the oracle: the
occlusion culling of the depth splats for every tile size, for a camera inside the
near plane of part of the fluid, far away (splats of less than a pixel) and with
matrices that turn it off; the marching of blocks of 256 voxels with a triangle cap
inside a voxel; and the field's ranges on grids that are no whole number of blocks and
for iso levels that no block, some and every block lies off."""
import numpy as np
import pytest

import oracle
from particles4all_b200 import Sim, configs
from particles4all_b200.camera import Camera, frame_matrices
from particles4all_b200.params import default_aniso, default_mesh, default_ray, default_ssfr

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def block(built):
    p, sc = configs.dam_break_32k(side=16)
    g, o = Sim(), oracle.OracleSim()
    for s in (g, o):
        s.reset_scene(p, sc)
        for _ in range(4):
            s.step(1 / 60)
        s.aniso(default_aniso())
    yield g, o
    g.close()


def camera(w, h, dist, target=(4.0, 3.0, 4.0), el=0.35):
    cam = Camera()
    cam.target, cam.az, cam.el, cam.dist = list(target), -0.5, el, dist
    m = frame_matrices(cam, w, h)
    return {k: m[k] for k in ("view", "proj", "inv_view_proj", "inv_view", "eye", "width", "height")}


@pytest.mark.parametrize("w,h,dist", [(96, 72, 40.0), (101, 67, 22.0), (160, 120, 17.0), (320, 241, 17.0), (400, 300, 9.0),
                                      (64, 48, 95.0), (96, 72, 3.0)])
def test_culled_splats(block, w, h, dist):
    g, o = block
    sp = dict(default_ssfr(), **camera(w, h, dist))
    g.ssfr(sp)
    o.ssfr(sp)
    for name in ("rawZ", "eyeZ", "thick", "image"):
        assert np.array_equal(g.ssfr_read(name), o.ssfr_read(name)), name


@pytest.mark.parametrize("what", ["scaled view", "sheared projection", "other rays"])
def test_splats_without_culling(block, what):
    g, o = block
    sp = dict(default_ssfr(), **camera(96, 72, 20.0))
    if what == "scaled view":
        sp["view"] = [1.25 * x if k % 4 < 3 and k < 12 else x for k, x in enumerate(sp["view"])]
    elif what == "sheared projection":
        sp["proj"] = [0.2 if k == 8 else x for k, x in enumerate(sp["proj"])]
    else:
        sp["inv_view_proj"] = camera(96, 72, 20.5, el=0.3)["inv_view_proj"]
    g.ssfr(sp)
    o.ssfr(sp)
    for name in ("rawZ", "image"):
        assert np.array_equal(g.ssfr_read(name), o.ssfr_read(name), equal_nan=name == "rawZ"), name


@pytest.mark.parametrize("resolution,cap", [(5, 3_000_000), (33, 1), (47, 1000), (50, 1001)])
def test_mesh_blocks(block, resolution, cap):
    g, o = block
    m = dict(default_mesh(), resolution=resolution, max_triangles=cap)
    assert g.mesh(m) == o.mesh(m)
    for name in ("meshField", "meshNField"):
        assert np.array_equal(g.read(name), o.buffer(name))
    assert np.array_equal(g.read("meshVerts"), o.buffer("meshVerts").reshape(-1, 2))


@pytest.mark.parametrize("resolution", [6, 31, 48])
@pytest.mark.parametrize("iso", [0.02, 0.4, 0.99, 3.0, 0.0, -0.1])
@pytest.mark.parametrize("use_surface", [0, 1])
def test_ray_ranges(block, resolution, iso, use_surface):
    g, o = block
    m = dict(default_mesh(), resolution=resolution)
    g.mesh(m)
    o.mesh(m)
    rp = dict(default_ray(), **camera(80, 61, 18.0), iso=iso, use_surface=use_surface)
    for debug in (0, 3):
        rp["debug"] = debug
        g.ray(rp)
        assert np.array_equal(g.ray_read(), o.ray(rp)), debug
