"""Self-contacts with many vertices on one face: no plan of rounds is kept for
them, and the contacts are walked in detection order."""
import time

import numpy as np
import pytest

import xpbd_gb300 as G
from test_gpu_self_rounds import _walk

pytestmark = pytest.mark.gpu


def _on_one_face(n):
    """A hex of 1 m with its top at z = 0, and over it a plate of n x n x 2 hexes
    whose bottom vertices lie 1 mm inside."""
    A = G.grid_mesh(1, 1, 1, 1.0)
    X, t, f = G.grid_mesh(n, n, 2, 0.4 / n)
    top = A[0] - [0, 0, 1.0]
    X = X + [0.25, 0.1, 0.001]
    rest = np.vstack([top, X])
    return (rest, np.vstack([A[1], t + len(top)]), np.vstack([A[2], f + len(top)]),
            np.vstack([top, X - [0, 0, 0.002]]).astype(np.float32).astype(np.float64))


# 64 rounds are planned for; 289 and 1,681 contacts; more than the 4,096 whose bids fit shared memory
@pytest.mark.parametrize("n", [7, 16, 40, 66])
def test_many_contacts_on_one_face_equal_walking_them(lib, n):
    X, tets, faces, x = _on_one_face(n)
    s = G.XPBDSolver(X, tets, faces, 1e-6, 0.3, 1000.0, g_accel=0.0, num_iters=1, self_collisions=1)
    s.set_positions(x)
    s.detect_collisions()
    pairs, _ = s.self_contacts()
    most = np.unique(pairs[:, 1], return_counts=True)[1].max()
    assert len(pairs) >= (n + 1) ** 2 and most > 0.8 * (n + 1) ** 2
    x0 = s.positions()
    s.solve()
    got, lam = s.positions(), s.self_contacts()[1]
    ref, rlam = _walk(x0, 1 / s.masses(), pairs, faces, 1e-8 / 1e-6)
    # moves along z, where coordinates are below 4 mm (half an ulp 1.2e-10), once a contact of a vertex;
    # x and y keep 6e-8 of 1 m; each move is good to 1e-3
    scale = np.abs(ref - x0).max()
    assert scale > 1e-4
    assert np.abs(got - ref).max() <= 2e-7 + 2e-10 * most + 1e-3 * scale
    assert np.abs(lam - rlam).max() <= 1e-3 * np.abs(rlam).max() + 1e-12
    s.close()


def test_detection_does_not_plan_a_round_for_each_contact(lib):
    """10,201 contacts, most of them on one face: planning them a round each took
    five times as long as the whole detection (244 against 40 ms). Detection
    with and without the contacts may differ by a quarter of that."""
    X, tets, faces, x = _on_one_face(100)
    s = G.XPBDSolver(X, tets, faces, 1e5, 0.45, 1000.0, g_accel=0.0, num_iters=1, self_collisions=1)
    took = []
    for pos in (X, x):
        s.set_positions(pos)
        t = []
        for _ in range(4):
            s.synchronize()
            t0 = time.perf_counter()
            s.detect_collisions()
            s.synchronize()
            t.append(time.perf_counter() - t0)
        took.append(min(t))
    assert len(s.self_contacts()[0]) > 10000
    assert took[1] < took[0] + 0.05
    s.close()
