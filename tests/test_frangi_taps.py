"""pack_taps against gauss_kernel_with, kernel by kernel: the same bits, for
equal and unequal sigmas of the axes, the smallest radius and the largest."""
import numpy as np
import pytest

from miccai2016_gb300.qfrangi_gpu import MAX_TAPS, gauss_kernel_with, pack_taps


@pytest.mark.parametrize("sigmas", [[[0.1, 0.1, 0.1]], [[1, 1, 1], [2, 2, 2], [3, 3, 3]],
                                    [[2.1, 1.0, 0.7], [0.7, 4.4, 2.1], [15.8, 2.1, 15.8]]])
@pytest.mark.parametrize("n_sigmas,round_up,gamma", [(4, False, 1), (3, True, 1), (2.5, False, 0.5)])
def test_taps_equal_the_single_kernels(sigmas, n_sigmas, round_up, gamma):
    taps, radius = pack_taps(sigmas, n_sigmas, round_up, gamma)
    for s, row in enumerate(sigmas):
        for a, sg in enumerate(float(v) for v in row):
            for o in range(3):
                k = gauss_kernel_with(sg, o, sg ** (o * gamma), n_sigmas, round_up)
                assert radius[s, a] == len(k) // 2
                assert np.array_equal(taps[s, a, o, :len(k)].view(np.uint32), k.view(np.uint32))
                assert not taps[s, a, o, len(k):].any()


def test_too_wide_a_kernel_is_refused():
    with pytest.raises(ValueError, match="sigma 20 needs 161 taps; at most %d" % MAX_TAPS):
        pack_taps([[1.0, 20.0, 1.0]])
