"""The dataflow sweeps where a colour has no patch for some of its tasks."""
import numpy as np
import pytest

import xpbd_gb300 as G

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("patch", [1, 5])
def test_empty_shares_of_a_colour(lib, patch):
    """A grid whose colours take several tasks each beside a fan of tets around
    one edge, which has colours that the grid has no patch of (and the grid
    some that the fan has none of): variants 2, 3 (bulk copies of a task's
    records) and 4 give the same states, and those of the colour launches."""
    X, tets, _ = G.grid_mesh(9, 10, 11, 0.01)
    rng = np.random.default_rng(4)
    n = 70
    ang = np.linspace(0, 2 * np.pi, n, endpoint=False)
    ring = np.stack([0.02 * np.cos(ang), 0.02 * np.sin(ang), 0.005 + 0.001 * rng.uniform(-1, 1, n)], 1)
    Xf = np.concatenate([[[0, 0, 0], [0, 0, 0.01]], ring])
    tf = np.array([[0, 1, 2 + k, 2 + (k + 1) % n] for k in range(n)], np.int32)
    x = np.concatenate([X, Xf])
    x = x + 2e-4 * rng.uniform(-1, 1, x.shape)
    fixed = np.concatenate([X[:, 2] == 0, np.arange(len(Xf)) == 0])
    out = {}
    for var in (0, 2, 3, 4):
        s = G.XPBDSolver(instances=[(X, tets, None, 3e3, 0.45, 1000.0), (Xf, tf, None, 3e3, 0.45, 1000.0)],
                         num_iters=5, gs_variant=var, gs_patch_tets=patch, collision_rate=0.0)
        s.fix_vertices(fixed)
        s.set_positions(x)
        if var == 4:
            s.set_latency_stamps(True)  # the versioned sweep, not the on-chip one
        s.step(2)
        s.synchronize()
        out[var] = s.positions(), s.lambdas()
        s.close()
    for var in (3, 4):
        np.testing.assert_array_equal(out[var][0], out[2][0])
        np.testing.assert_array_equal(out[var][1], out[2][1])
    assert np.abs(out[2][0] - out[0][0]).max() <= 1e-6
