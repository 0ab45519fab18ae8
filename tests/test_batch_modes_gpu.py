"""The batched engine's and the server's modes: instances of every kind of
launch side by side (metric, radius field, volume sizes at the tiles' edges),
each equal bit for bit to its own batch of one; the compact sweeps of the
server where the tile sweeps' fields do not fit; the last steps of requests
that never stop, for update 1, odd and even."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
U_TOL = 1e-3
E = 10 ** -1.5


def _volume(seed, shape):
    from miccai2016_gb300.serving import helix_request
    p = helix_request(shape, 0.8, seed)
    p["shape"] = shape
    return p


def _cut(num_iter, update, bound):
    from miccai2016_gb300.batched import BatchedCut
    p = BatchedCut.CutParameters()
    p.num_iter, p.update, p.error_bound = num_iter, update, bound
    return BatchedCut(p)


def _plain(p, eigs, alpha, num_iter, update, bound):
    from miccai2016_gb300.continuous_cut_anisotropic_gpu import CmfCutQAnisotropicGpu
    prm = CmfCutQAnisotropicGpu.CutParameters()
    prm.num_iter, prm.update, prm.error_bound = num_iter, update, bound
    c = CmfCutQAnisotropicGpu(prm)
    u = c.execute(p["img"].cuda(), p["quats"].cuda(), eigs, alpha, p["cs"].cuda(), p["ct"].cuda(), verbose=False)
    return u, c.last_iterations


@pytest.mark.parametrize("update,num_iter,bound", [(7, 60, -1.0), (10, 200, 2e-3), (1, 9, -1.0)])
def test_every_kind_of_instance_side_by_side(update, num_iter, bound):
    import torch
    vols = [_volume(1, (24, 33, 61)), _volume(2, (17, 29, 32))]
    fields = [v["grad2"].cuda() for v in vols]
    insts = []
    for v in (0, 1):
        for eigs in ((1.0, E, E), (E, E, 1.0), (1.0, 1.0, 1.0), (1.0, 0.3, 0.05)):
            insts.append(dict(volume=v, weighting=0.05, decay=3.0, eigs=eigs))
            insts.append(dict(volume=v, alpha=0.05 * torch.exp(-fields[v] / 9.0), eigs=eigs))
    b = _cut(num_iter, update, bound)
    dv = [b.prepare_volume(v["img"], v["quats"], v["cs"], v["ct"], grad2=v["grad2"]) for v in vols]
    us = b.solve(dv, insts)
    its = b.last_iterations.copy()
    for k, inst in enumerate(insts):
        one = _cut(num_iter, update, bound)
        u1 = one.solve(dv, [inst])[0]
        if one.last_iterations[0] == its[k]:   # residual sums follow the tiling
            assert torch.equal(us[k], u1), k
        alpha = 0.05 * torch.exp(-fields[inst["volume"]] / 9.0)
        u, it = _plain(vols[inst["volume"]], inst["eigs"], alpha, num_iter, update, bound)
        assert abs(it - its[k]) <= update
        if it == its[k]:
            assert float((us[k] - u).abs().max()) <= U_TOL, k
    if bound < 0:
        assert np.all(its == num_iter)


def _serve(reqs, workspace_bytes, num_iter, update, bound, max_slots=4):
    import torch
    from miccai2016_gb300.serving import CutServer
    srv = CutServer(num_iter=num_iter, update=update, error_bound=bound, workspace_bytes=workspace_bytes,
                    max_slots=max_slots, max_work_items=4096)
    out, queue = {}, list(enumerate(reqs))
    for _ in range(20000):
        while queue:
            tag, (p, eigs) = queue[0]
            u = torch.empty(p["shape"], dtype=torch.float32).pin_memory()
            if not srv.admit(tag, p, 0.05, 3.0, eigs, u):
                break
            out[tag] = [u, None]
            queue.pop(0)
        srv.step()
        for tag, it, _ in srv.poll():
            out[tag][1] = it
        if not queue and all(v[1] is not None for v in out.values()):
            break
    assert not queue and all(v[1] is not None for v in out.values())
    srv.close()
    return out


@pytest.mark.parametrize("update,num_iter", [(1, 1), (1, 6), (2, 2), (3, 9), (4, 12), (30, 60)])
def test_served_requests_run_exactly_num_iter(update, num_iter):
    reqs = [(_volume(3, (20, 31, 45)), (1.0, E, E)), (_volume(4, (12, 16, 33)), (1.0, 1.0, 1.0)),
            (_volume(5, (9, 40, 29)), (1.0, 0.3, 0.05))]
    out = _serve(reqs, 64 << 20, num_iter, update, -1.0)
    for tag, (p, eigs) in enumerate(reqs):
        assert out[tag][1] == num_iter
        u, _ = _plain(p, eigs, 0.05 * np.exp(-1.0 / 9.0 * p["grad2"].cuda().cpu().numpy()), num_iter, update, -1.0)
        assert np.max(np.abs(out[tag][0].numpy() - u.cpu().numpy())) <= U_TOL, tag


def test_a_request_that_fits_only_the_compact_fields_is_served():
    from miccai2016_gb300 import _native as N
    from miccai2016_gb300.serving import CutServer
    p = _volume(6, (40, 48, 52))
    n = 40 * 48 * 52
    tables = int(N.lib().m16_server_table_bytes(4, 4096))
    full = CutServer.request_bytes(p["shape"])
    assert full >= 72 * n
    reqs = [(p, (1.0, E, E)), (p, (1.0, 0.3, 0.05))]
    tight = _serve(reqs, tables + full - 2 * n, 90, 30, 1e-3)
    roomy = _serve(reqs, tables + 4 * full, 90, 30, 1e-3)
    for tag in (0, 1):
        assert tight[tag][1] == roomy[tag][1]
        assert np.max(np.abs(tight[tag][0].numpy() - roomy[tag][0].numpy())) <= U_TOL
