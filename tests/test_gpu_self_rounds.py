"""Self-collisions of a Gauss-Seidel context are projected in rounds of contacts
that share no vertex, earlier contacts of a vertex in earlier rounds: the state
must be the one that walking the contacts in detection order gives."""
import numpy as np
import pytest

import xpbd_gb300 as G

pytestmark = pytest.mark.gpu


def _pair(n, seed):
    X, t, f = G.grid_mesh(n, n, n, 0.1 / n)
    X2 = np.vstack([X, X + [0.102, 0.013, 0.007]])
    rng = np.random.default_rng(seed)
    x = np.vstack([X, X + [0.1 - 0.1 / n / 4, 0.013, 0.007]]) + rng.uniform(-1, 1, X2.shape) * 0.1 / n * 0.01
    return X2, np.vstack([t, t + len(X)]), np.vstack([f, f + len(X)]), x.astype(np.float32).astype(np.float64)


def _walk(x, w, pairs, faces, at):
    """FP64, one contact after the other (C = (q - p1) . a / |a| + 1e-5)."""
    x = x.copy()
    lam = np.zeros(len(pairs))
    for j, (v, f) in enumerate(pairs):
        ids = [v, *faces[f]]
        q, p1, p2, p3 = x[ids]
        a = np.cross(p2 - p1, p3 - p1)
        n = np.linalg.norm(a)
        C = (q - p1) @ a / n + 1e-5
        if C > 0:
            continue
        r1, r2 = ((u / n - a * (a @ u) / n ** 3) for u in (q - p1, q - p2))
        g = np.stack([a / n, -a / n + np.cross(r1, p3 - p2), np.cross(r1, p1 - p3), np.cross(r2, p2 - p1)])
        dl = -C / (at + (w[ids] * (g * g).sum(1)).sum())
        lam[j] += dl
        x[ids] += w[ids, None] * g * dl
    return x, lam


@pytest.mark.parametrize("n", [3, 8, 17, 53])
def test_rounds_equal_walking_the_contacts_in_order(lib, n):
    """One iteration on a mesh so soft that the tets' own projections leave the
    positions (compliance 1e-9 of the contacts'): from one contact to more than
    the 4,096 whose bids fit shared memory."""
    X, tets, faces, x = _pair(n, n)
    s = G.XPBDSolver(X, tets, faces, 1e-6, 0.3, 1000.0, g_accel=0.0, num_iters=1, self_collisions=1)
    s.set_positions(x)
    s.detect_collisions()
    pairs, _ = s.self_contacts()
    assert (len(pairs) > 4096) == (n == 53) and len(pairs) >= 3
    x0 = s.positions()
    s.solve()
    got, lam = s.positions(), s.self_contacts()[1]
    ref, rlam = _walk(x0, 1 / s.masses(), pairs, faces, 1e-8 / 1e-6)
    # each contact moves its vertices by up to an edge's quarter; FP32 keeps 6e-8 of 0.2 m and about 1e-5 of the move
    scale = np.abs(ref - x0).max()
    assert scale > 1e-6
    assert np.abs(got - ref).max() <= 1e-6 * 0.2 + 1e-3 * scale
    assert np.abs(lam - rlam).max() <= 1e-3 * np.abs(rlam).max() + 1e-12
    s.close()
