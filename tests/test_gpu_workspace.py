"""gf_beam_mount beyond the 512 MB of device workspace that a context keeps: the same bits
as in calls of a few elements, before and after it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_mounts_beyond_the_kept_workspace(gpu_ctx, golden):
    g = golden("ref_beam_elements.npz")
    m = len(g["K"])
    lag = np.zeros((m, 2, 21))
    lag[:, :, [0, 4, 8]] = 1.0
    lag[:, :, 20] = 1.0
    args = (g["xyz"], g["mat"], g["sec6"], g["cs"], lag, g["disp"])
    K, f = gpu_ctx.beam_mount(*args)
    # 342 results and 84 inputs of 8 bytes an element, and its constants and history
    k = -(-(600 << 20) // (8 * (342 + 84)) // m)
    Kl, fl = gpu_ctx.beam_mount(*[np.tile(a, (k,) + (1,) * (a.ndim - 1)) for a in args])
    assert np.array_equal(Kl.reshape(k, m, -1), np.broadcast_to(K.reshape(m, -1), (k, m, K[0].size)))
    assert np.array_equal(fl.reshape(k, m, -1), np.broadcast_to(f.reshape(m, -1), (k, m, f[0].size)))
    K1, f1 = gpu_ctx.beam_mount(*args)
    assert np.array_equal(K1, K) and np.array_equal(f1, f)
