"""Batches in less workspace than they ask for, and the compact sweeps.

A batch in a small workspace is solved in cohorts: every instance's u has the
bits of the batch that fits (the sweeps compute a voxel the same way whatever
shares the launch).  In the least workspace each instance takes the compact
sweeps, as do the instances of volumes whose rows would be padded by more than an
eighth; these are compared with the oracle at the max-flow's tolerance."""
import ctypes

import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu
U_TOL = 1e-3
E = 10 ** -1.5
PADDED = (53, 990, 5)   # 262350 voxels in rows of 5 (padded to 8): no tile sweeps


def _volume(seed, shape):
    rng = np.random.RandomState(seed)
    f = lambda lo, hi: rng.uniform(lo, hi, shape).astype(np.float32)
    quats = np.stack([rng.uniform(-np.pi, np.pi, shape), rng.uniform(0, np.pi, shape),
                      rng.uniform(-np.pi, np.pi, shape)], -1).astype(np.float32)
    return dict(img=rng.normal(0.5, 0.5, shape).astype(np.float32), quats=quats, cs=f(0, 1), ct=f(0, 1),
                grad2=f(0, 4), shape=shape)


def _cut(num_iter, update):
    from miccai2016_gb300.batched import BatchedCut
    p = BatchedCut.CutParameters()
    p.num_iter, p.update, p.error_bound = num_iter, update, -1.0
    return BatchedCut(p)


def _alpha(v):
    return (0.05 * np.exp(-1.0 / 9.0 * v["grad2"].astype(np.float64))).astype(np.float32)


def _instances(vols):
    out = []
    for k, v in enumerate(vols):
        for eigs in ((1.0, E, E), (1.0, 1.0, 1.0), (1.0, 0.3, 0.05)):
            out += [dict(volume=k, weighting=0.05, decay=3.0, eigs=eigs), dict(volume=k, alpha=_alpha(v), eigs=eigs)]
    return out


def _against_the_oracle(vols, insts, us, num_iter, update):
    for inst, u in zip(insts, us):
        v = vols[inst["volume"]]
        ru, _, _ = O.maxflow_solve(v["img"], v["quats"], inst["eigs"], _alpha(v), v["cs"], v["ct"], num_iter=num_iter,
                                   update=update, error_bound=-1.0)
        assert np.max(np.abs(u - ru)) <= U_TOL, (inst["volume"], inst["eigs"], "alpha" in inst)


class Workspaces:
    """N.workspace with a device that has room for `limit` bytes."""

    def __init__(self, monkeypatch, limit):
        import torch
        from miccai2016_gb300 import _native as N
        self.asked, real = [], N.workspace

        def workspace(nbytes):
            self.asked.append(int(nbytes))
            if nbytes > limit:
                raise torch.cuda.OutOfMemoryError("no room")
            return real(nbytes)
        monkeypatch.setattr(N, "workspace", workspace)


@pytest.mark.parametrize("part", [1.0, 0.6, 0.3, 0.0])   # of the way from the least workspace to the whole
def test_a_batch_in_cohorts(monkeypatch, part):
    import torch
    from miccai2016_gb300 import _native as N
    L = N.lib()
    vols = [_volume(1, (24, 33, 61)), _volume(2, (17, 29, 32)), _volume(3, (9, 40, 90))]
    insts = _instances(vols)
    whole = _cut(31, 7)
    dv = [whole.prepare_volume(v["img"], v["quats"], v["cs"], v["ct"], grad2=v["grad2"]) for v in vols]
    us = [u.cpu().numpy() for u in whole.solve(dv, insts)]
    vd, idesc, _, _ = whole._describe(dv, insts)
    full = L.m16_batch_workspace_bytes(vd, len(dv), idesc, len(insts))
    least = L.m16_batch_workspace_bytes_min(vd, len(dv), idesc, len(insts))
    assert 0 < least < L.m16_batch_steps_bytes_min(vd, len(dv), idesc, len(insts)) < full
    limit = least + int(part * (full - least))
    ws = Workspaces(monkeypatch, limit)
    small = _cut(31, 7)
    got = [u.cpu().numpy() for u in small.solve(dv, insts)]
    assert np.all(small.last_iterations == 31)
    assert ws.asked[0] == full and least <= ws.asked[-1] <= limit and (part == 1.0) == (len(ws.asked) == 1)
    if part == 0.0:
        _against_the_oracle(vols, insts, got, 31, 7)
    else:
        for a, b in zip(us, got):
            assert np.array_equal(a.view(np.uint32), b.view(np.uint32))


def test_less_than_the_least_is_refused(monkeypatch):
    import torch
    from miccai2016_gb300 import _native as N
    L = N.lib()
    vols = [_volume(1, (24, 33, 61))]
    insts = _instances(vols)[:3]
    c = _cut(5, 5)
    dv = [c.prepare_volume(v["img"], v["quats"], v["cs"], v["ct"], grad2=v["grad2"]) for v in vols]
    vd, idesc, us, _ = c._describe(dv, insts)
    cp = N.CutParams(0.2, 0.11, -1.0, 5, 5, (ctypes.c_double * 3)(1, 1, 1))
    for least, begin in ((L.m16_batch_workspace_bytes_min(vd, 1, idesc, 3), False),
                         (L.m16_batch_steps_bytes_min(vd, 1, idesc, 3), True)):
        ws = torch.empty(least, dtype=torch.uint8, device="cuda")
        for nbytes, status in ((least - 1, N.M16_ERR_WORKSPACE), (least, N.M16_OK)):
            if begin:
                h = ctypes.c_void_p()
                assert L.m16_batch_begin_min(vd, 1, idesc, 3, ctypes.byref(cp), N.ptr(ws), nbytes, N.stream_ptr(),
                                             ctypes.byref(h)) == status
                if status == N.M16_OK:
                    assert L.m16_batch_end(h, None, None, N.stream_ptr()) == status
            else:
                assert L.m16_batch_solve(vd, 1, idesc, 3, ctypes.byref(cp), None, None, N.ptr(ws), nbytes,
                                         N.stream_ptr(), None) == status
    with pytest.raises(torch.cuda.OutOfMemoryError):
        Workspaces(monkeypatch, 1000)
        c.solve(dv, insts)


def test_steps_without_room_take_the_compact_sweeps(monkeypatch):
    from miccai2016_gb300 import _native as N
    vols = [_volume(4, (24, 33, 61)), _volume(5, (9, 40, 90))]
    insts = _instances(vols)
    c = _cut(23, 5)
    dv = [c.prepare_volume(v["img"], v["quats"], v["cs"], v["ct"], grad2=v["grad2"]) for v in vols]
    vd, idesc, _, _ = c._describe(dv, insts)
    least = N.lib().m16_batch_steps_bytes_min(vd, 2, idesc, len(insts))
    Workspaces(monkeypatch, least)
    steps = c.begin(dv, insts)
    assert steps._ws.numel() == least
    for n in (1, 4, 11, 7):
        steps.iterate(n)
    us = [u.cpu().numpy() for u in steps.end()]
    assert np.all(steps.iterations == 23)
    _against_the_oracle(vols, insts, us, 23, 5)


def test_padded_rows_take_the_compact_sweeps():
    """Both radius sources, alone and beside instances of the tile sweeps, and a
    served request with an alpha field."""
    import torch
    from miccai2016_gb300 import _native as N
    from miccai2016_gb300.serving import CutServer
    vols = [_volume(6, PADDED), _volume(7, (17, 29, 32))]
    insts = _instances(vols)
    c = _cut(13, 4)
    dv = [c.prepare_volume(v["img"], v["quats"], v["cs"], v["ct"], grad2=v["grad2"]) for v in vols]
    us = [u.cpu().numpy() for u in c.solve(dv, insts)]
    _against_the_oracle(vols, insts, us, 13, 4)
    for only in (0, 1):   # one radius source in the launch
        u = c.solve(dv, [insts[only]])[0].cpu().numpy()
        assert np.array_equal(u.view(np.uint32), us[only].view(np.uint32))

    v = vols[0]
    host = {k: torch.from_numpy(v[k]).pin_memory() for k in ("img", "quats", "cs", "ct")}
    alpha = torch.from_numpy(_alpha(v)).pin_memory()
    out = torch.empty(PADDED).pin_memory()
    srv = CutServer(num_iter=12, update=4, error_bound=-1.0, workspace_bytes=64 << 20, max_slots=2, max_work_items=8192)
    sq = (ctypes.c_double * 3)(*np.sqrt([1.0, E, E]))
    req = N.ServeRequest(*PADDED, 0, host["img"].data_ptr(), host["quats"].data_ptr(), None, alpha.data_ptr(),
                         host["cs"].data_ptr(), host["ct"].data_ptr(), (ctypes.c_double * 3)(1, 1, 1), 0.0, 0.0, sq,
                         out.data_ptr(), 7)
    ok = ctypes.c_int32(0)
    N.check("m16_server_admit", N.lib().m16_server_admit(srv._h, ctypes.byref(req), ctypes.byref(ok)))
    assert ok.value == 1
    done = []
    for _ in range(2000):
        srv.step()
        done += srv.poll()
        if done:
            break
    assert [d[:2] for d in done] == [(7, 12)]
    srv.close()
    _against_the_oracle(vols, [insts[1]], [out.numpy()], 12, 4)
