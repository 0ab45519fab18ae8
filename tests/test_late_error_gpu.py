"""A stop inside a sweep of several iterations runs the iterations up to it again,
after the call has read its control word.  A copy lost there must end in
M16_ERR_TIMEOUT too (tests/native/late_error.cu sets the word's error field behind
that read)."""
import ctypes
import os
import subprocess

import pytest

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def parts(tmp_path_factory):
    from miccai2016_gb300 import build as B
    out = tmp_path_factory.mktemp("late")
    jobs = []
    for part in range(2):
        so = str(out / ("part%d.so" % part))
        cmd = [B.nvcc_path()] + B.ARCH + B.NVCC_FLAGS + ["-DPART=%d" % part, "-I", B.CSRC, "-shared", "-o", so,
                                                         os.path.join(HERE, "native", "late_error.cu"), "-cudart", "static"]
        jobs.append((so, subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)))
    libs = []
    for so, job in jobs:
        text, _ = job.communicate()
        assert job.returncode == 0, text
        libs.append(ctypes.CDLL(so))
    return libs


# one read of the control word, then the rerun; failures before and after it
@pytest.mark.parametrize("reads,status", [(0, "M16_OK"), (1, "M16_ERR_TIMEOUT")])
def test_the_error_of_a_rerun(parts, reads, status):
    import torch
    from miccai2016_gb300 import _native as N
    N.lib()
    shape = (9, 18, 34)
    g = torch.Generator(device="cuda")
    g.manual_seed(2)
    f = lambda *s: torch.rand(s, generator=g, device="cuda")
    img, quats, alpha, cs, ct, out = f(*shape), f(*shape, 3), f(*shape), f(*shape), f(*shape), f(*shape, 3)
    ws = torch.zeros(64 << 20, dtype=torch.uint8, device="cuda")
    it, n = ctypes.c_int32(0), ctypes.c_int32(0)
    p = N.CutParams(0.2, 0.11, 1e30, 10, 1, (ctypes.c_double * 3)(1, 1, 1))   # stops at iteration 0, the first of a pair
    L = parts[0]
    L.m16_maxflow_solve.argtypes = N.lib().m16_maxflow_solve.argtypes
    L.fail_after(reads)
    st = L.m16_maxflow_solve(N.ptr(img), N.ptr(quats), (ctypes.c_double * 3)(1.0, 0.3, 0.3), None, N.ptr(alpha), 0.0,
                             N.ptr(cs), N.ptr(ct), None, *shape, ctypes.byref(p), N.ptr(out), ctypes.byref(it), None, 0,
                             ctypes.byref(n), N.ptr(ws), ws.numel(), N.stream_ptr())
    assert it.value == 1 and n.value == 1
    assert st == getattr(N, status)
    stopped = ctypes.c_int32(0)
    L = parts[1]
    L.m16_gvf_run.argtypes = N.lib().m16_gvf_run.argtypes
    L.fail_after(reads)
    st = L.m16_gvf_run(N.ptr(quats), None, *shape, (ctypes.c_double * 3)(1, 1, 1), 0.2, 0.1, 0, 10, 1, 1e30, 0,
                       N.ptr(out), ctypes.byref(it), ctypes.byref(stopped), None, 0, ctypes.byref(n), N.ptr(ws),
                       ws.numel(), N.stream_ptr())
    assert it.value == 1 and stopped.value == 1
    assert st == getattr(N, status)
    torch.cuda.synchronize()
