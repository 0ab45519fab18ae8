"""The projection of the tile sweeps at the ends of float32: a flow whose squared
norm overflows is scaled to zero (rad / inf, as the two sweeps and the oracle do),
one under an infinite radius is not scaled, one under radius 0 vanishes.  Steps of
1e25 make every flow's squared norm overflow as long as neighbouring values of tmp
differ by more than their rounding; the solve runs as many iterations as that holds
for (with no flow left a voxel's iterates depend on nothing else)."""
import os
import sys

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, os.path.join(HERE, "golden"))

import inputs as I  # noqa: E402
from oracle import oracle as O  # noqa: E402

pytestmark = pytest.mark.gpu
U_TOL = 1e-3   # the max-flow's, after a fixed iteration count
E = 10 ** -1.5


def _overflowing_iterations(img, cs, ct, least_eig, steps, most, cc=0.2):
    """How many iterations, up to `most`, every flow's squared norm overflows by a
    factor of 100, from a recursion without flow in float64."""
    u = img.astype(np.float64) / img.max()
    rcc, pt, tmp = 1 / cc, np.minimum(cs, ct).astype(np.float64), None
    tmp = -u * rcc
    for n in range(most):
        g2 = np.zeros(u.shape)
        for ax in range(3):
            d = np.diff(tmp, axis=ax) * steps
            g2[tuple(slice(0, k) for k in d.shape)] += d * d
        g2[-1, -1, -1] = np.inf   # no forward neighbour: no flow
        if g2.min() * least_eig < 100 * float(np.finfo(np.float32).max):
            return n
        ps = np.minimum(cs, pt - rcc * (u - 1))
        pt = np.minimum(ct, ps + rcc * u)
        err = pt - ps
        u = u - err / rcc
        tmp = err - u * rcc
    return most


@pytest.mark.parametrize("eigs", [(1.0, E, E), (1.0, 1.0, 1.0), (1.0, 0.3, 0.05), "field"])
@pytest.mark.parametrize("steps,radius", [(1e25, 0.3), (0.11, 0.0), (0.11, np.inf)])
@pytest.mark.parametrize("num_iter", [1, 4, 7])
def test_the_projection_at_the_ends_of_the_range(eigs, steps, radius, num_iter):
    from miccai2016_gb300.batched import BatchedCut
    from miccai2016_gb300.continuous_cut_anisotropic_gpu import CmfCutQAnisotropicGpu
    shape = (9, 18, 34)
    rng = np.random.RandomState(3)
    f = lambda lo, hi: rng.uniform(lo, hi, shape).astype(np.float32)
    img, quats, cs, ct = f(0, 1), I.random_squeezed(rng, shape), f(0, 1), f(0, 1)
    alpha = np.full(shape, radius, np.float32)
    if eigs == "field":
        eigs = rng.uniform(0.1, 2, shape + (3,))
    if steps > 1:
        num_iter = _overflowing_iterations(img, cs, ct, np.min(eigs), steps, num_iter)
        assert num_iter > 0
    p = CmfCutQAnisotropicGpu.CutParameters()
    p.num_iter, p.update, p.error_bound, p.steps = num_iter, 3, -1.0, steps
    ru, _, _ = O.maxflow_solve(img, quats, eigs, alpha, cs, ct, num_iter=num_iter, update=3, error_bound=-1.0,
                               steps=steps)
    assert np.all(np.isfinite(ru)) and np.max(np.abs(ru)) < 10
    for path in (0, 1):
        c = CmfCutQAnisotropicGpu(p)
        c.iteration_path = path
        u = c.execute(img, quats, eigs, alpha, cs, ct, verbose=False)
        assert np.max(np.abs(u - ru)) <= U_TOL, path
    if not isinstance(eigs, np.ndarray):
        b = BatchedCut(p)
        u = b.solve([b.prepare_volume(img, quats, cs, ct)], [dict(volume=0, alpha=alpha, eigs=eigs)])[0]
        assert np.max(np.abs(u.cpu().numpy() - ru)) <= U_TOL
