"""Volumes of few rows: which sweeps a solve, a batch and a served request take
(csrc/tile_sweep.cuh, tile_rows_ok), and the same labelling either way.

The tile sweeps need 3 (isotropic), 5 (one eigenvalue differs) or 7 rows where the
tiles times planes exceed 6 (a solve) or 16 (an instance of a batch) per SM.
Against the oracle and the single solve the tolerance is the max-flow's."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu
U_TOL = 1e-3
E = 10 ** -1.5
LEAST = {"axis": 5, "iso": 3, "const": 7, "field": 7}
EIGS = {"axis": (1.0, E, E), "iso": (1.0, 1.0, 1.0), "const": (1.0, 0.3, 0.05)}


def _inputs(shape):
    rng = np.random.RandomState(shape[1])
    f = lambda lo, hi: rng.uniform(lo, hi, shape).astype(np.float32)
    quats = np.stack([rng.uniform(-np.pi, np.pi, shape), rng.uniform(0, np.pi, shape),
                      rng.uniform(-np.pi, np.pi, shape)], -1).astype(np.float32)
    return dict(img=rng.normal(0.5, 0.5, shape).astype(np.float32), quats=quats, alpha=f(0.01, 0.5), cs=f(0, 1),
                ct=f(0, 1), field=rng.uniform(0.05, 2, shape + (3,)), labels=rng.randint(0, 3, shape).astype(np.uint8))


def _params(num_iter, update):
    from miccai2016_gb300.continuous_cut_anisotropic_gpu import CmfCutQAnisotropicGpu
    p = CmfCutQAnisotropicGpu.CutParameters()
    p.num_iter, p.update, p.error_bound = num_iter, update, -1.0
    return p


def _tiles(shape):   # tiles x planes: 28 written columns of 32, 13 rows of 16
    d0, d1, d2 = shape
    nx = 1 if d2 <= 32 else -(-(d2 - 32) // 28) + 1
    return nx * d0   # one row of tiles


# 25 tiles a plane: 1000 and 900 (the limit is 912); one tile a plane: 913 and 912 planes
@pytest.mark.parametrize("d0,d2", [(40, 700), (36, 700), (913, 9), (912, 9)])
@pytest.mark.parametrize("d1", [1, 2, 3, 4, 5, 6, 7, 8])
@pytest.mark.parametrize("metric", ["axis", "iso", "const", "field"])
def test_the_sweeps_of_a_solve(metric, d0, d1, d2):
    from miccai2016_gb300.continuous_cut_anisotropic_gpu import CmfCutQAnisotropicGpu
    shape = (d0, d1, d2)
    inp = _inputs(shape)
    eigs = EIGS.get(metric, inp["field"])
    labels = inp["labels"] if d1 % 2 else None
    c = CmfCutQAnisotropicGpu(_params(6, 4))
    u = c.execute(inp["img"], inp["quats"], eigs, inp["alpha"], inp["cs"], inp["ct"], labels=labels, verbose=False)
    tiles = d1 >= LEAST[metric] or _tiles(shape) <= 6 * 152
    assert (c.last_stats.pair_launches, c.last_stats.p_launches) == ((3, 0) if tiles else (0, 6))
    ru, _, res = O.maxflow_solve(inp["img"], inp["quats"], eigs, inp["alpha"], inp["cs"], inp["ct"], labels=labels,
                                 num_iter=6, update=4, error_bound=-1.0)
    assert np.max(np.abs(u - ru)) <= U_TOL
    np.testing.assert_allclose(c.last_residuals, res[:len(c.last_residuals)], rtol=1e-3, atol=1e-7)


@pytest.mark.parametrize("d0,d1,d2", [(98, 2, 700), (98, 4, 700), (98, 6, 700), (98, 7, 700), (97, 1, 700)])   # 2450, 2425
def test_a_batch_and_a_server_of_few_rows(d0, d1, d2):
    import torch
    from miccai2016_gb300.batched import BatchedCut
    from miccai2016_gb300.continuous_cut_anisotropic_gpu import CmfCutQAnisotropicGpu
    from miccai2016_gb300.serving import CutServer
    shape = (d0, d1, d2)
    inp = _inputs(shape)
    grad2 = (4 * inp["alpha"]).astype(np.float32)
    alpha = (0.05 * np.exp(-1.0 / 9.0 * grad2.astype(np.float64))).astype(np.float32)
    b = BatchedCut(_params(8, 4))
    vol = b.prepare_volume(inp["img"], inp["quats"], inp["cs"], inp["ct"], grad2=grad2)
    insts = [dict(volume=0, weighting=0.05, decay=3.0, eigs=e) for e in EIGS.values()]
    insts += [dict(volume=0, alpha=alpha, eigs=e) for e in EIGS.values()]
    us = b.solve([vol], insts)
    single = []
    for e in EIGS.values():
        c = CmfCutQAnisotropicGpu(_params(8, 4))
        single.append(c.execute(inp["img"], inp["quats"], e, alpha, inp["cs"], inp["ct"], verbose=False))
    for k, u in enumerate(us):
        assert np.max(np.abs(u.cpu().numpy() - single[k % 3])) <= U_TOL, k
    host = {k: torch.from_numpy(v).pin_memory() for k, v in dict(inp, grad2=grad2).items()
            if k in ("img", "quats", "cs", "ct", "grad2")}
    # a workspace for three such requests by the size that the server gives
    from miccai2016_gb300 import _native as N
    tables = int(N.lib().m16_server_table_bytes(3, 1 << 16))
    srv = CutServer(num_iter=8, update=4, error_bound=-1.0, max_slots=3, max_work_items=1 << 16,
                    workspace_bytes=tables + 3 * CutServer.request_bytes(shape) + 3 * 4 * d0 * d1 * d2)
    outs = [torch.empty(shape).pin_memory() for _ in EIGS]
    for tag, e in enumerate(EIGS.values()):
        assert srv.admit(tag, host, 0.05, 3.0, e, outs[tag])
    done = 0
    for _ in range(2000):
        srv.step()
        done += len(srv.poll())
        if done == 3:
            break
    assert done == 3
    srv.close()
    for k, u in enumerate(outs):
        assert np.max(np.abs(u.numpy() - single[k])) <= U_TOL, k
