"""The Frangi passes where their tiles end.

x pass (four columns per lane, 128 per warp, any radius): one scale's squeezed
quaternions are those of the eigendecomposition of the plain Hessian kernel bit
for bit -- both accumulate the taps in the same order with the same fused
multiply-adds, and solve with the same rounding -- and c is half the largest
norm of its eigenvalues (a float32 square root of a sum of three squares: 4
ulp).  z and y passes for any radius: the Hessian in float64 with the same taps,
within the rounding of three passes of K multiply-adds."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _filter(sigma, c):
    from miccai2016_gb300.qfrangi_gpu import FeatureFilter, VesselnessCalculation
    p = VesselnessCalculation.Parameters()
    p.c, p.bright_objects, p.scales = c, True, (sigma, sigma, 1)
    return FeatureFilter(p, verbose=False)


# radius round(4 sigma): 1, 2, 3, 4, 12, 15, 16 (instantiated), 17, 18, 63 (any)
@pytest.mark.parametrize("sigma", [0.25, 0.5, 0.75, 1.0, 3.0, 3.75, 4.0, 4.25, 4.5, 15.75])
@pytest.mark.parametrize("shape", [(1, 1, 1), (3, 9, 31), (2, 5, 32), (2, 4, 33), (2, 8, 128), (4, 3, 129), (1, 6, 160),
                                   (1, 6, 161), (2, 17, 257)])
def test_x_pass_equals_the_plain_kernels(shape, sigma):
    from miccai2016_gb300.qfrangi_gpu import eigendecomposition, hessian
    rng = np.random.RandomState(shape[2] + int(100 * sigma))
    img = rng.normal(0.5, 0.5, shape).astype(np.float32)
    e = eigendecomposition(hessian(img, (sigma,) * 3)).reshape(-1, 6)
    norm = np.sqrt(np.max(np.sum(e[:, :3].astype(np.float64) ** 2, 1)))
    for c in (None, 0.4):
        f = _filter(sigma, c)
        val, quat, _ = f.execute_for(img, None)
        assert np.isfinite(val).all() or not np.isfinite(e).all() or norm == 0
        taken = val.reshape(-1) > -np.inf
        q = np.where(taken[:, None], e[:, 3:], np.float32(0))
        assert np.array_equal(q.view(np.uint32), quat.reshape(-1, 3).view(np.uint32))
        want = 0.5 * norm if c is None else c
        assert abs(float(f.last_c[0]) - want) <= 4 * 2.0 ** -23 * abs(want)


def _axis_matrix(taps, n):
    """out = M @ line: the true convolution with the mirror boundary."""
    K, m = len(taps), np.zeros((n, n))
    for x in range(n):
        for j in range(K):
            p = x - K // 2 + j
            period = max(2 * (n - 1), 1)
            p %= period
            m[x, p if p < n else period - p] += taps[K - 1 - j]
    return m


@pytest.mark.parametrize("shape,sigma", [((1, 1, 1), 4.4), ((70, 5, 9), 4.4), ((6, 71, 33), 5.0), ((3, 4, 40), 15.7)])
def test_any_radius_hessian_within_its_rounding(shape, sigma):
    from miccai2016_gb300.qfrangi_gpu import hessian, pack_taps
    rng = np.random.RandomState(sum(shape))
    img = rng.normal(0.5, 0.5, shape).astype(np.float32)
    h = hessian(img, (sigma,) * 3).astype(np.float64)
    taps, radius = pack_taps((sigma,) * 3)
    K = 2 * radius[0] + 1
    t = [[taps[0, a, o, :K[a]].astype(np.float64) for o in range(3)] for a in range(3)]
    for k, orders in enumerate([(2, 0, 0), (0, 2, 0), (0, 0, 2), (1, 1, 0), (1, 0, 1), (0, 1, 1)]):
        z, y, x = [_axis_matrix(t[a][orders[a]], shape[a]) for a in range(3)]
        want = np.einsum("az,by,cx,zyx->abc", z, y, x, img.astype(np.float64), optimize=True)
        # K multiply-adds per pass, each rounded once: K u sum |tap| |input|
        size = np.prod([np.sum(np.abs(t[a][orders[a]])) for a in range(3)]) * np.max(np.abs(img))
        assert np.max(np.abs(h[..., k] - want)) <= 1.01 * K.sum() * 2.0 ** -24 * size
