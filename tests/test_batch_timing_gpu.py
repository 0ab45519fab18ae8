"""m16_solve_stats of a batch with time_kernels: pair_launches counts launches of
two iterations only, not the single ones that an odd interval starts with and not
the compact sweeps, which have none; the result has the same bits as untimed."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
E = 10 ** -1.5


@pytest.mark.parametrize("padded,tiled", [(False, True), (True, True), (True, False)])
# iteration 0, whole intervals, the rest: 0 + 4 x 3 + 1 pairs; 0 + 5 x 3; none; 0 + 1
@pytest.mark.parametrize("num_iter,update,pairs", [(31, 7, 13), (31, 6, 15), (1, 3, 0), (9, 1, 0), (3, 30, 1)])
def test_pairs_are_counted(padded, tiled, num_iter, update, pairs):
    import torch
    from miccai2016_gb300.batched import BatchedCut
    g = torch.Generator(device="cuda")
    g.manual_seed(3)
    f = lambda *s: torch.rand(s, generator=g, device="cuda")
    p = BatchedCut.CutParameters()
    p.num_iter, p.update, p.error_bound = num_iter, update, -1.0
    cut = BatchedCut(p)
    shapes = [(53, 990, 5)] * padded + [(17, 33, 40), (9, 20, 61)] * tiled   # the first takes the compact sweeps
    vols = [cut.prepare_volume(f(*s), f(*s, 3), f(*s), f(*s), grad2=f(*s)) for s in shapes]
    insts = [dict(volume=k, weighting=0.05, decay=3.0, eigs=e) for k in range(len(vols))
             for e in ((1.0, E, E), (1.0, 1.0, 1.0))]
    timed = cut.solve(vols, insts, time_kernels=True)
    st = cut.last_stats
    assert st.pair_launches == (pairs if tiled else 0)
    assert (st.pair_ms > 0) == (st.pair_launches > 0) and st.pair_ms < 1000
    plain = cut.solve(vols, insts)
    assert cut.last_stats.pair_launches == 0 and cut.last_stats.pair_ms == 0
    for a, b in zip(timed, plain):
        assert torch.equal(a.view(torch.int32), b.view(torch.int32))
