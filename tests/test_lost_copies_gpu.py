"""Bounded waits of the tile sweeps (csrc/tile_sweep.cuh, csrc/gvf_tile.cuh):
a sweep whose bulk copies do not arrive gives up after the planes that were under
way, marches to its end without asking for more, sets the error word and the stop
state, and the launches behind it write nothing and wait for nothing
(tests/native/lost_copies.cu loses the copies).  Then the host's side: a call
that finds the error word set returns M16_ERR_TIMEOUT, and a server stays
refused after it."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))
# 2^18 tries of at least 1.5 us for each plane of a ring of at most five that is asked for
# before the sweep gives up, the longest try 4 us
GIVE_UP_MS, ALL_MS = 390.0, 5 * 1100.0
NOTHING_MS = 200.0       # a launch that has nothing to do

class Outcome(ctypes.Structure):
    _fields_ = [("error", ctypes.c_int), ("stop", ctypes.c_int), ("untouched", ctypes.c_int), ("ms", ctypes.c_float)]


@pytest.fixture(scope="module")
def parts(tmp_path_factory):
    from miccai2016_gb300 import build as B
    out = tmp_path_factory.mktemp("lost")
    src = os.path.join(HERE, "native", "lost_copies.cu")
    jobs = []
    for part in range(3):
        so = str(out / ("part%d.so" % part))
        cmd = [B.nvcc_path()] + B.ARCH + B.NVCC_FLAGS + ["-DPART=%d" % part, "-I", B.CSRC, "-shared", "-o", so, src,
                                                         "-cudart", "static"]
        jobs.append((so, subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)))
    libs = []
    for so, job in jobs:
        text, _ = job.communicate()
        assert job.returncode == 0, text
        libs.append(ctypes.CDLL(so))
    return libs


# the max-flow (two iterations, one), the gradient vector flow (without and with a response) and the batch through more
# planes than any ring has slots; a single plane
@pytest.mark.parametrize("part,variant,shape", [(0, 0, (60, 20, 40)), (0, 1, (60, 20, 40)), (1, 0, (60, 20, 40)),
                                                (1, 1, (60, 20, 40)), (2, 0, (60, 20, 40)), (0, 2, (1, 14, 30)),
                                                (1, 0, (1, 14, 30))])
def test_a_lost_copy_ends_the_sweep(parts, part, variant, shape):
    import torch
    torch.zeros(1, device="cuda")   # the context
    out = (Outcome * 3)()
    assert parts[part].lost_copies(variant, *shape, out) == 0
    lost, after, whole = out
    assert lost.error == 1 and lost.stop & 1
    assert GIVE_UP_MS <= lost.ms <= ALL_MS
    assert after.error == 1 and after.stop & 1 and after.untouched   # since the call before
    assert after.ms <= NOTHING_MS
    assert whole.error == 0 and whole.stop == 0 and not whole.untouched
    assert whole.ms <= NOTHING_MS


def _batch_inputs(shape):
    import torch
    g = torch.Generator(device="cuda")
    g.manual_seed(1)
    f = lambda *s: torch.rand(s, generator=g, device="cuda")
    return f(*shape), f(*shape, 3), f(*shape), f(*shape), f(*shape)


def test_an_error_word_ends_a_batch_and_a_field():
    """The error words of a batch (the last of its workspace) and of a gradient
    vector flow continued from its workspace."""
    import torch
    from miccai2016_gb300 import _native as N
    from miccai2016_gb300.batched import BatchedCut
    L = N.lib()
    p = BatchedCut.CutParameters()
    p.num_iter, p.update, p.error_bound = 20, 5, -1.0
    shape = (8, 17, 35)
    img, quats, cs, ct, grad2 = _batch_inputs(shape)
    for failed in (False, True):
        cut = BatchedCut(p)
        vol = cut.prepare_volume(img, quats, cs, ct, grad2=grad2)
        steps = cut.begin([vol], [dict(volume=0, weighting=0.1, decay=3.0, eigs=(1.0, 0.1, 0.1))] * 3)
        steps.iterate(7)
        nbytes = L.m16_batch_workspace_bytes(steps._vd, 1, steps._idesc, 3)
        word = steps._ws[nbytes - 256:nbytes - 252].view(torch.int32)
        assert int(word) == 0
        if failed:
            word.fill_(1)
            with pytest.raises(Exception, match="timed out"):
                steps.end()
        else:
            steps.end()


def test_a_server_stays_refused_after_a_lost_copy():
    import torch
    from miccai2016_gb300 import _native as N
    from miccai2016_gb300.serving import CutServer
    L = N.lib()
    shape = (8, 17, 35)
    names = ("img", "quats", "cs", "ct", "grad2")
    inputs = {k: t.cpu().pin_memory() for k, t in zip(names, _batch_inputs(shape))}
    u = torch.empty(shape, pin_memory=True)
    s = CutServer(num_iter=300, update=10, error_bound=-1.0, workspace_bytes=64 << 20, max_slots=4, max_work_items=4096)
    assert s.admit(1, inputs, 0.1, 3.0, (1.0, 0.1, 0.1), u)
    s.step()
    s.step()
    torch.cuda.synchronize()
    end = L.m16_server_table_bytes(4, 4096)
    word = s._ws[end - 256:end - 252].view(torch.int32)
    assert int(word) == 0
    word.fill_(1)
    torch.cuda.synchronize()
    with pytest.raises(Exception, match="timed out"):
        for _ in range(3):   # found by the step after the one that copies the word
            s.step()
    steps = s.info()["steps"]
    for call in (s.step, lambda: s.admit(2, inputs, 0.1, 3.0, (1.0, 0.1, 0.1), u), s.poll):
        with pytest.raises(Exception, match="timed out"):
            call()
    assert s.info()["steps"] == steps
    s.close()
