"""The network's gradient at tile edges and where a block has several tiles
(two blocks an SM: more than 304 tiles of 128 rows), against the oracle's
gradient of the same precision."""
import numpy as np
import pytest

import mlp_oracle as M
import xpbd_gb300 as G

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 127, 128, 129, 38_912, 38_913, 100_000])
def test_gradient_at_tile_edges(lib, n):
    X, tets, _ = G.grid_mesh(2, 2, 2, 0.5)
    s = G.XPBDSolver(X, tets, None, 3e3, 0.45, 1000.0)
    p = M.init_params(5)
    for k in (1, 3, 5, 7):
        p[k] = 0.1 * np.random.default_rng(k).standard_normal(p[k].shape).astype(np.float32)
    s.set_mlp_params(M.flatten(p))
    rng = np.random.default_rng(n)
    X = np.zeros((n, 16), np.float32)
    X[:, :14] = rng.standard_normal((n, 14))
    Y = rng.standard_normal((n, 2)).astype(np.float32)
    loss, g = s.mlp_loss_grad(X, Y)
    ref_loss, ref = M.loss_and_grads(p, X, Y)
    # as for the sizes inside a tile: BF16 flips of single activations (2^-8)
    # bound a layer's gradient to a percent, and a single row's loss to 2^-8
    assert abs(loss - ref_loss) <= (4e-3 if n == 1 else 1e-3) * ref_loss
    for a, b in zip(M.unflatten(g), ref):
        assert np.linalg.norm(a - b) <= 1e-2 * np.linalg.norm(b) + 1e-7
    s.close()
