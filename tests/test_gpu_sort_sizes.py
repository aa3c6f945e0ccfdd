"""The grid sort at the sizes where its launches change (one or four particles per
thread, whole and partial scan words) and on a workspace that is aligned to 8 bytes
only, against a stable sort of the same keys: bit for bit."""
import ctypes as C

import numpy as np
import pytest

from particles4all_b200 import _abi, _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,dims,shift", [(0, (3, 5, 7), 0), (1, (1, 1, 1), 0), (255, (8, 1, 1), 8), (1025, (9, 9, 9), 0),
                                          (299999, (40, 31, 33), 0), (300000, (40, 32, 33), 8), (300001, (41, 31, 33), 0),
                                          (301057, (64, 32, 32), 0)])
def test_sort_sizes(built, n, dims, shift):
    import torch
    rng = np.random.default_rng(n + shift)
    h, cells = 0.5, int(np.prod(dims))
    pos = np.ones((n, 4), np.float32)
    pos[:, :3] = rng.uniform(-0.2, 1.2, (n, 3)) * np.array(dims) * h
    vel = rng.normal(size=(n, 4)).astype(np.float32)
    body = rng.integers(0, 4, (n, 4)).astype(np.uint32)
    rest = rng.normal(size=(n, 4)).astype(np.float32)
    grid = _abi.Grid((C.c_float * 3)(0, 0, 0), h, (C.c_int32 * 3)(*dims))
    t_in = [torch.from_numpy(a.view(np.int32) if a.dtype == np.uint32 else a).cuda() for a in (pos, vel, body, rest)]
    t_out = [torch.full((max(n, 1), 4), -7, dtype=t.dtype, device="cuda") for t in (t_in[0], t_in[0], t_in[0], t_in[2], t_in[0])]
    cs = torch.full((cells + 1,), -7, dtype=torch.int32, device="cuda")
    slot = torch.full((max(n, 1),), -7, dtype=torch.int32, device="cuda")
    size = _lib.lib().p4a_grid_sort_workspace_size(n, cells)
    ws = torch.zeros(size + 16, dtype=torch.uint8, device="cuda")
    ptrs = [t.data_ptr() for t in t_in + t_out] + [cs.data_ptr(), slot.data_ptr()]
    rc = _lib.lib().p4a_grid_sort(C.byref(grid), n, 1 / 240, 9.81, *ptrs, ws.data_ptr() + shift, size, None,
                                  torch.cuda.current_stream().cuda_stream)
    assert rc == 0
    f = np.float32
    v = vel[:, :3].copy()
    v[:, 1] = v[:, 1] + f(f(1 / 240) * f(-9.81))
    pred = pos[:, :3] + f(1 / 240) * v
    c = np.clip(np.floor(pred / f(h)).astype(np.int64), 0, np.array(dims) - 1)
    key = (c[:, 2] * dims[1] + c[:, 1]) * dims[0] + c[:, 0]
    order = np.argsort(key, kind="stable")
    got = [t.cpu().numpy()[:n] for t in t_out]
    assert np.array_equal(got[0], pos[order])
    assert np.array_equal(got[1][:, :3], v[order]) and np.array_equal(got[2][:, :3], pred[order])
    assert np.array_equal(got[3].view(np.uint32), body[order]) and np.array_equal(got[4], rest[order])
    start = np.concatenate([[0], np.cumsum(np.bincount(key, minlength=cells))])
    assert np.array_equal(cs.cpu().numpy(), start)
    inverse = np.empty(n, np.int64)
    inverse[order] = np.arange(n)
    assert np.array_equal(slot.cpu().numpy()[:n], inverse)
