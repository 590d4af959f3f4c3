"""The on-chip Gauss-Seidel sweep (small meshes: one thread-block cluster per
instance, positions and multipliers in shared memory) against the routes it
stands in for: the versioned sweep (latency stamps keep a context on it) for
the combined constraints, the colour launches for the separate ones. The same
projections in the same order and arithmetic, so the states are equal bit for
bit."""
import numpy as np
import pytest

import workloads as W
import xpbd_gb300 as G

pytestmark = pytest.mark.gpu


def _state(dims, h=0.01, seed=0):
    X, tets, faces = G.grid_mesh(*dims, h)
    rng = np.random.default_rng(seed)
    x = X + 0.05 * h * rng.uniform(-1, 1, X.shape)
    v = 0.05 * rng.uniform(-1, 1, X.shape)
    return X, tets, faces, x, v


def _solver(dims, faces=False, **kw):
    X, tets, F, x, v = _state(dims)
    E = np.exp(np.random.default_rng(1).uniform(np.log(1e3), np.log(1e4), len(tets)))
    s = G.XPBDSolver(X, tets, F if faces else None, E, 0.45, 1000.0, dt=1e-3, collision_rate=0.0, **kw)
    s.fix_vertices(X[:, 2] == 0)
    s.set_positions(x)
    s.set_velocities(v)
    return s, X


def _press(s, X, n=2):
    w, top = X[:, 0].max(), X[:, 2].max()
    r = 0.5 * w
    c = np.array([[w / 2, X[:, 1].max() * (k + 0.5) / n, top + 0.9 * r] for k in range(n)])
    s.set_spheres(c, np.full(n, r))
    s.detect_collisions()


# one block of one warp's colours up to the largest cluster; ragged shares; a
# generic (not grid-hex) patch layout with patch sizes 3 and 1
CASES = [((1, 1, 1), 5), ((3, 5, 2), 5), ((5, 7, 3), 5), ((10, 10, 10), 5), ((11, 13, 9), 5), ((17, 16, 15), 5),
         ((10, 100, 10), 5), ((20, 37, 21), 5), ((33, 17, 21), 5),
         ((25, 25, 20), 5), ((5, 7, 3), 3), ((9, 8, 7), 1), ((12, 30, 11), 3)]


@pytest.mark.parametrize("dims,patch", CASES)
def test_on_chip_sweep_equals_versioned_sweep(lib, dims, patch):
    out = []
    for versioned in (False, True):
        s, _ = _solver(dims, num_iters=4, gs_patch_tets=patch)
        if versioned:
            s.set_latency_stamps(True)
        s.step(3)
        s.synchronize()
        assert s.health() == (0, 0)
        out.append((s.positions(), s.velocities(), s.lambdas(), s.prev_positions()))
        s.close()
    for a, b in zip(*out):
        np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("dims", [(4, 4, 4), (10, 20, 4), (10, 60, 10)])
def test_on_chip_contacts_equal_versioned_sweep(lib, dims):
    out = []
    for versioned in (False, True):
        s, X = _solver(dims, faces=True, num_iters=5)
        if versioned:
            s.set_latency_stamps(True)
        _press(s, X)
        l0 = s.launch_count()
        s.step(1)
        first = s.collisions()
        s.step(3)
        n = s.launch_count() - l0
        s.synchronize()
        out.append((s.positions(), s.collisions(), first, n))
        s.close()
    assert (out[0][2][:, 11] != 0).sum() > 3  # projected contacts
    assert out[0][3] < out[1][3]
    for a, b in zip(out[0][:3], out[1][:3]):
        np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("dims,patch,faces", [((3, 4, 2), 5, False), ((11, 13, 9), 5, True), ((10, 60, 10), 5, False),
                                              ((6, 9, 5), 2, True)])
def test_on_chip_separate_constraints_equal_colour_launches(lib, dims, patch, faces):
    out = []
    for var in (4, 0):
        s, X = _solver(dims, faces=faces, num_iters=4, gs_variant=var, gs_patch_tets=patch,
                       constraint_type=G.CONSTRAINT_SEPARATE)
        if faces:
            _press(s, X)
        l0 = s.launch_count()
        s.step(3)
        n = s.launch_count() - l0
        s.synchronize()
        out.append((s.positions(), s.lambdas(), n))
        s.close()
    assert out[0][2] < out[1][2]
    np.testing.assert_array_equal(out[0][0], out[1][0])
    np.testing.assert_array_equal(out[0][1], out[1][1])


def test_on_chip_careful_pass_and_modes(lib):
    """A layer squashed to |det F| ~ 1e-4 takes the FP64 guard; first order,
    the residual per substep, update() without velocities, solve() alone and a
    batch of uneven instances, against the versioned sweep."""
    def squash(s, X, versioned):
        x = X.copy()
        top = X[:, 2] == X[:, 2].max()
        x[top, 2] = X[:, 2].max() - 0.01 + 1e-6
        s.set_positions(x)
        s.set_velocities(np.zeros_like(x))
        s.step(1)

    def every_substep(s, X, versioned):
        s.step(2)

    def solve(s, X, versioned):
        s.update()
        s.solve()
        s.velocity_update()

    for act, kw in ((squash, {}), (every_substep, dict(residual_policy=G.RESIDUAL_EVERY_SUBSTEP)), (solve, {}),
                    (every_substep, dict(first_order=1, damping_multiplier=2e4))):
        out = []
        for versioned in (False, True):
            s, X = _solver((10, 13, 6), num_iters=3, **kw)
            if versioned:
                s.set_latency_stamps(True)
            act(s, X, versioned)
            out.append((s.positions(), s.velocities(), s.lambdas(), s.residual_history(), s.health()))
            s.close()
        if act is squash:
            assert out[0][4][1] > 0  # the guard ran
        assert out[0][4] == out[1][4]
        for a, b in zip(out[0][:4], out[1][:4]):
            np.testing.assert_array_equal(a, b)


def test_on_chip_batch_equals_versioned_batch(lib):
    out = []
    for versioned in (False, True):
        b = W.batched(n=7, seed=3, t_range=(200, 6000), iters=5)
        s = W.make_batch_solver(b)
        if versioned:
            s.set_latency_stamps(True)
        W.drive_batch(s, b)
        s.detect_collisions()
        s.step(3)
        s.synchronize()
        out.append((s.positions(), s.collisions()))
        s.close()
    np.testing.assert_array_equal(out[0][0], out[1][0])
    np.testing.assert_array_equal(out[0][1], out[1][1])


@pytest.mark.parametrize("n", [3, 23, 24])
def test_residual_and_energy_sums_at_both_tets_per_thread(lib, n):
    """Below and above the size from which a thread adds up four tets (65,536;
    a last block that is partly empty): the residual's norm against the sum of
    the per-constraint residuals it also writes, and the strain energy against
    FP64 numpy from the same positions, within the FP32 rounding of the terms."""
    s, X = _solver((n, n, n), num_iters=2, residual_policy=G.RESIDUAL_EVERY_SUBSTEP)
    s.step(1)
    r = s.constraint_residual()
    a, _ = s.residual()
    hist = s.residual_history()[-1]
    # every term rounds once to FP32 (2^-24 relative) in the per-constraint vector
    assert abs(hist - np.sqrt((r * r).sum())) <= 2 ** -23 * hist
    assert a > 0 and abs(s.residual_noalloc() - a) <= 1e-13 * a
    x = s.positions()
    tets, E = s._meshes[0].tets, s._meshes[0].E
    D0 = (X[tets[:, :3]] - X[tets[:, 3:]]).transpose(0, 2, 1)
    F = (x[tets[:, :3]] - x[tets[:, 3:]]).transpose(0, 2, 1) @ np.linalg.inv(D0)
    vol = np.abs(np.linalg.det(D0)) / 6
    mu, la = E / 2.9, E * 0.45 / (1.45 * 0.1)
    J = np.linalg.det(F)
    d = J - 1
    Ch = np.where(J >= 1, np.log(np.maximum(J, 1)), d - d * d / 2 + d ** 3 / 3) - mu / la
    ref = (mu * vol * (F * F).sum((1, 2)) + la * vol * Ch * Ch).sum()
    # FP32 positions (1e-2 m edges in a 0.24 m mesh): F to 3e-6, the energy to twice that
    assert abs(s.strain_energy() - ref) <= 2e-5 * abs(ref)
    s.close()
