"""Which meshes and batches the on-chip sweep takes, and what it gives on them."""
import numpy as np
import pytest

import xpbd_gb300 as G

pytestmark = pytest.mark.gpu


def _batch(count, dims, **kw):
    X, tets, _ = G.grid_mesh(*dims, 0.01)
    E = np.exp(np.random.default_rng(1).uniform(np.log(1e3), np.log(1e4), len(tets)))
    s = G.XPBDSolver(instances=[(X, tets, None, E, 0.45, 1000.0)] * count, num_iters=3, collision_rate=0.0, **kw)
    rng = np.random.default_rng(0)
    x = np.concatenate([X + 5e-4 * rng.uniform(-1, 1, X.shape) for _ in range(count)])
    s.fix_vertices(np.tile(X[:, 2] == 0, count))
    s.set_positions(x)
    return s


@pytest.mark.parametrize("count,dims", [(1, (10, 10, 10)), (1, (12, 12, 12)), (1, (16, 16, 16)), (1, (18, 18, 18)),
                                        (1, (22, 22, 22)), (1, (10, 100, 10)), (6, (16, 16, 16)), (8, (22, 22, 22)),
                                        (9, (22, 22, 22)), (13, (22, 22, 22)), (15, (20, 20, 20)), (9, (13, 60, 13))])
def test_on_chip_clusters_fit_the_device_and_agree_with_the_versioned_sweep(lib, count, dims):
    """A batch goes on chip where the device holds the cluster of every instance
    at once (a second wave costs what the first does); one block to sixteen.
    The states equal the versioned sweep's bit for bit."""
    out = []
    for stamps in (False, True):
        s = _batch(count, dims)
        s.set_latency_stamps(stamps)
        route, blocks, held = s.debug_sweep_route()
        if stamps:
            assert route == "versioned"
        elif route == "chip":
            assert held >= count
        else:
            assert route == "versioned" and count > 1
        if not stamps and count == 1:
            assert route == "chip" and (blocks > 1) == (dims != (10, 10, 10))
        s.step(2)
        s.synchronize()
        assert s.health()[0] == 0
        out.append((s.positions(), s.velocities(), s.lambdas()))
        s.close()
    for a, b in zip(*out):
        np.testing.assert_array_equal(a, b)


def test_small_instances_that_share_tasks_equal_each_alone(lib):
    """1,500 instances of 12 hexes: more than the device has warps for, so a task
    of the versioned sweep holds patches of several of them. An instance's
    states equal those of a context of its own bit for bit."""
    X, tets, _ = G.grid_mesh(2, 3, 2, 0.01)
    K = 1500
    rng = np.random.default_rng(2)
    E = np.exp(rng.uniform(np.log(1e3), np.log(1e4), (K, len(tets))))
    x = np.stack([X + 5e-4 * rng.uniform(-1, 1, X.shape) for _ in range(K)])

    def run(ks):
        s = G.XPBDSolver(instances=[(X, tets, None, E[k], 0.45, 1000.0) for k in ks], num_iters=5, collision_rate=0.0)
        s.fix_vertices(np.tile(X[:, 2] == 0, len(ks)))
        s.set_positions(x[ks].reshape(-1, 3))
        if len(ks) > 1:
            assert s.debug_sweep_route()[0] == "versioned"
        s.step(3)
        s.synchronize()
        out = s.positions().reshape(len(ks), -1, 3), s.lambdas().reshape(len(ks), len(tets), 2)
        s.close()
        return out

    P, lam = run(list(range(K)))
    for k in (0, 1, 37, 700, 1499):
        p, m = run([k])
        np.testing.assert_array_equal(P[k], p[0])
        np.testing.assert_array_equal(lam[k], m[0])
