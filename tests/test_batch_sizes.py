"""m16_batch_workspace_bytes_min: the largest of the instances' own least sizes,
found without laying every one out (a batch of a thousand volumes asks for it on
each call)."""
import ctypes
import time

import numpy as np


def _describe(shapes, volumes):
    from miccai2016_gb300 import _native as N
    fake = ctypes.c_void_p(256)
    one = (ctypes.c_double * 3)(1, 1, 1)
    vd = (N.BatchVolume * len(shapes))()
    for k, s in enumerate(shapes):
        vd[k] = N.BatchVolume(*s, 0, fake, fake, fake, fake, fake, one)
    idesc = (N.BatchInstance * len(volumes))()
    for k, v in enumerate(volumes):
        idesc[k] = N.BatchInstance(v, 0, 0.1, 3.0, fake if k % 2 else None, one, fake)
    return vd, idesc


def test_the_least_size_is_the_largest_instance_alone():
    from miccai2016_gb300 import _native as N
    L = N.lib()
    rng = np.random.RandomState(4)
    for _ in range(60):
        shapes = [tuple(int(round(np.exp(rng.uniform(0, np.log(120))))) for _ in range(3)) for _ in range(7)]
        volumes = [int(v) for v in rng.randint(0, 7, 9)]
        vd, idesc = _describe(shapes, volumes)
        alone = []
        for v in volumes:
            _, one = _describe(shapes, [v])
            alone.append(L.m16_batch_workspace_bytes_min(vd, 7, one, 1))
            assert alone[-1] == L.m16_batch_steps_bytes_min(vd, 7, one, 1)
        assert L.m16_batch_workspace_bytes_min(vd, 7, idesc, 9) == max(alone) > 0


def test_a_thousand_volumes_cost_no_thousand_layouts():
    from miccai2016_gb300 import _native as N
    L = N.lib()
    vd, idesc = _describe([(20, 24, 28 + k % 5) for k in range(1000)], list(range(1000)))
    L.m16_batch_workspace_bytes_min(vd, 1000, idesc, 1000)
    t = time.perf_counter()
    assert L.m16_batch_workspace_bytes_min(vd, 1000, idesc, 1000) > 0
    assert time.perf_counter() - t < 0.01   # 0.07 s where each was laid out, 0.0001 now
