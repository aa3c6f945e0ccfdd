"""Boundary samples that a caller writes, through Sim.write or through the device pointers of
Sim.buffer_ptr, are the ones that the next frames see: bit for bit the oracle, with a group
of lanes and with one thread per particle, before and after frames that are replayed as
graphs; with weights far outside the ranges of the pair arithmetic too."""
import numpy as np
import pytest

from test_gpu_parity import compare, pair, small_params

pytestmark = pytest.mark.gpu


class View:
    def __init__(self, ptr, shape):
        self.__cuda_array_interface__ = {"data": (ptr, False), "shape": shape, "typestr": "<f4", "version": 3}


@pytest.mark.parametrize("pointer", [False, True])
@pytest.mark.parametrize("name,scale", [("bpsi", 0.25), ("bpsi", 1.0e-33), ("bpsi", 1.0e9), ("bpsi", -3.0),
                                        ("bpos", 0.97)])
@pytest.mark.parametrize("n", [1500, 21000])
def test_written_samples(built, n, name, scale, pointer):
    import torch
    p = small_params(targetParticleCount=n, box=[1.0, 0.8, 0.8] if n > 20000 else [0.5, 0.4, 0.3], surfaceTensionK=0.3)
    g, o = pair(p)
    nb = g.info()["n_boundary"]
    shape = (nb, 4) if name == "bpos" else (nb,)

    def write(values):
        o.write(name, values)
        if not pointer:
            g.write(name, values)
            return
        dptr, nbytes = g.buffer_ptr(name)
        assert nbytes == 4 * values.size
        torch.as_tensor(View(dptr, shape), device="cuda").copy_(torch.from_numpy(values))
        torch.cuda.synchronize()

    first = o.buffer(name).reshape(shape).copy()
    for values in (first * np.float32(scale), first):
        for s in (g, o):
            for _ in range(1 if n > 20000 else 4):
                s.step(1 / 60)
        write(np.ascontiguousarray(values, np.float32))
        for s in (g, o):
            s.step(1 / 60)
        compare(g, o)
        assert np.array_equal(g.read(name).reshape(shape), values)
    g.close()
