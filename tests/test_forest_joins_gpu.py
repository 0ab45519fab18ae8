"""The joins of many small trees (m16_ridge_forest_joins where the trees times
the points exceed four keys a point, one group of ranks and several) against
the dense stable Kruskal of the oracle (oracle/adjust.py:stable_mst): the same
edges, on integer points full of equal distances."""
import numpy as np
import pytest

from oracle import adjust as A

pytestmark = pytest.mark.gpu


def _trees(rng, n, longest, box):
    pts = [rng.randint(3, box, 3) + np.cumsum(rng.randint(-1, 2, (rng.randint(1, longest + 1), 3)), axis=0)
           for _ in range(n)]
    pts = np.unique(np.concatenate(pts), axis=0)
    pts = pts[pts.min(1) >= 0].astype(np.int64)
    return pts[rng.permutation(len(pts))]


# two points; ten trees; isolated points (a warp's queries from one to three);
# trees longer than a warp and than a chunk of targets; several groups of ranks
@pytest.mark.parametrize("n,longest,box", [(2, 1, 40), (10, 4, 60), (150, 1, 90), (31, 60, 200), (12, 700, 150),
                                           (700, 3, 120)])
def test_joins_of_many_trees(n, longest, box):
    from miccai2016_gb300 import ridge_mst as M
    rng = np.random.RandomState(n + longest)
    pts = _trees(rng, n, longest, box)
    vs = np.ones(3)
    r, offsets = M._local_offsets(vs)
    d_pts, d_edges = M._local_mst_device(pts, vs, r, offsets)
    joins = M._joins_gpu(d_pts, d_edges)
    assert joins is not None   # taken on the device
    e = d_edges.cpu().numpy()
    a, b = np.concatenate([e[:, 0], joins[0]]), np.concatenate([e[:, 1], joins[1]])
    t = A.stable_mst(pts, (1, 1, 1)).tocoo()
    pairs = lambda i, j: set(zip(np.minimum(i, j).tolist(), np.maximum(i, j).tolist()))
    assert len(a) == len(pts) - 1
    assert pairs(a, b) == pairs(t.row, t.col)
