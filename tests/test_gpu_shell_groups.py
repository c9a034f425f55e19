"""Shell_1 elements are formed in groups of ten per CTA: groups that are full,
one short, one over and of a single element, with and without follower pressure
in one group, against the oracle and, bit for bit, against each element alone."""
import numpy as np
import pytest

from oracle import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("area_update", [1, 0])
@pytest.mark.parametrize("n", [1, 9, 10, 11, 23])
def test_groups_of_elements(gpu_ctx, n, area_update):
    rng = np.random.default_rng(n)
    corner = np.array([[0.0, 0.0, 0.0], [1.0, 0.1, 0.05], [0.2, 0.9, -0.1]])
    mid = np.array([(corner[0] + corner[1]) / 2, (corner[1] + corner[2]) / 2, (corner[2] + corner[0]) / 2])
    xyz = np.stack([np.concatenate([corner, mid]) * (1.0 + 0.1 * rng.random()) for _ in range(n)])
    mat = np.tile([2.0e11, 0.3, 7800.0], (n, 1))
    thick = 0.01 * (1.0 + rng.random(n))
    hist = 0.01 * rng.normal(size=(n, 2, 27))
    disp = 0.01 * rng.normal(size=(n, 27))
    p = np.where(np.arange(n) % 3 == 2, np.nan, 1.0e6 * (1.0 + rng.random(n)))
    K, f = gpu_ctx.shell_elements(xyz, mat, thick, hist, disp, p, area_update)
    for e in range(n):
        pe = None if np.isnan(p[e]) else float(p[e])
        Ko, fo = oracle.shell_element(xyz[e], mat[e], float(thick[e]), hist[e], disp[e], pe, area_update)
        # a few hundred roundings of terms no larger than the largest entry
        assert np.abs(K[e] - Ko).max() <= 1e-11 * np.abs(Ko).max()
        assert np.abs(f[e] - fo).max() <= 1e-11 * np.abs(fo).max()
        one = gpu_ctx.shell_elements(xyz[e:e + 1], mat[e:e + 1], thick[e:e + 1], hist[e:e + 1], disp[e:e + 1],
                                     p[e:e + 1], area_update)
        assert np.array_equal(one[0][0], K[e]) and np.array_equal(one[1][0], f[e])
