"""The bounded waits of the on-chip sweep of several blocks."""
import numpy as np
import pytest

import xpbd_gb300 as G

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("faces,separate", [(False, False), (True, False), (False, True)])
def test_an_on_chip_wait_that_runs_out_reports_timeout_and_the_context_recovers(lib, faces, separate):
    """A vertex of two blocks whose due version is never written (the test hook)
    makes its patches' waits give up after 4,096 polls. Their warps skip the
    rest, their neighbours' waits give up in turn, every block waits for the
    copies into it and returns: xpbd_synchronize reports the time-out,
    xpbd_health clears it, and with the tables restored the context steps on
    as a fresh one does. 10 x 40 x 10 hexes: four blocks whose tet records do
    not stay in shared memory, so copies are in flight when a wait gives up."""
    X, tets, F = G.grid_mesh(10, 40, 10, 0.01)
    rng = np.random.default_rng(3)
    x = X + 5e-4 * rng.uniform(-1, 1, X.shape)

    def solver():
        s = G.XPBDSolver(X, tets, F if faces else None, 3e3, 0.45, 1000.0, num_iters=4, collision_rate=0.0,
                         constraint_type=G.CONSTRAINT_SEPARATE if separate else G.CONSTRAINT_COMBINED)
        s.fix_vertices(X[:, 2] == 0)
        return s

    def start(s):
        s.set_positions(x)
        s.set_velocities(np.zeros_like(x))
        if faces:
            s.set_spheres(np.array([[0.05, 0.1, 0.145], [0.05, 0.3, 0.145]]), np.full(2, 0.05))
            s.detect_collisions()

    s = solver()
    start(s)
    s.step(1)
    s.synchronize()
    held = []
    for v in range(len(X)):
        try:
            s.debug_stall_on_chip(v, 4096)
            held.append(v)
            break
        except G.XPBDError as e:
            assert e.status == G.XPBD_ERR_STATE
    assert held
    s.step(1)
    with pytest.raises(G.XPBDError) as e:
        s.synchronize()
    assert e.value.status == G.XPBD_ERR_TIMEOUT
    s.health()  # clears the counters
    s.debug_stall_on_chip(-1)
    f = solver()
    out = []
    for c in (s, f):
        start(c)
        c.step(3)
        c.synchronize()
        assert c.health()[0] == 0
        out.append((c.positions(), c.lambdas()))
        c.close()
    for a, b in zip(*out):
        np.testing.assert_array_equal(a, b)


def test_stall_hook_needs_several_blocks(lib):
    X, tets, _ = G.grid_mesh(3, 3, 3, 0.1)
    s = G.XPBDSolver(X, tets, None, 3e3, 0.45, 1000.0)
    with pytest.raises(G.XPBDError) as e:
        s.debug_stall_on_chip(0, 64)
    assert e.value.status == G.XPBD_ERR_STATE
    s.close()
