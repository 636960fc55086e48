"""The network's gradient at the edges of its tiling: rows short of and past a
tile, more tiles than the update has groups, more tiles than the GPU has SMs.  The
gradient of n rows is the sum of its tiles' own, up to the rounding of the sum."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 127, 128, 129, 32 * 128, 32 * 128 + 1, 152 * 128, 152 * 128 + 1, 305 * 128 + 77])
def test_gradient_is_the_sum_of_its_tiles(built, n):
    import torch

    torch.cuda.set_device(0)
    from shapes_gb300 import _lib

    rng = np.random.default_rng(n)
    feat = rng.normal(0, 1, (n, 16)).astype(np.float32)
    tgt = rng.normal(0, 1, (n, 2)).astype(np.float32)
    net = _lib.Mlp(2)
    g, loss = net.gradient(feat, tgt)
    tiles = range(0, n, 128)
    want, mag, want_loss = np.zeros(g.size), np.zeros(g.size), 0.0
    for k in tiles:
        rows = min(128, n - k)
        gt, lt = net.gradient(feat[k:k + 128], tgt[k:k + 128])
        want += gt.astype(np.float64) * rows / n
        mag += np.abs(gt.astype(np.float64)) * rows / n
        want_loss += float(lt) * rows / n
    # each group adds len/32 tiles, 32 groups are added, and a tile's own gradient is rounded where it is scaled
    eps = (len(tiles) / 32 + 36) * 2.0 ** -24
    assert np.all(np.abs(g - want) <= eps * mag + 1e-30)
    assert abs(loss - want_loss) <= eps * want_loss
    net.close()
