"""The deterministic Jacobi variant adds a vertex's updates up per block of 160
tets and then over the blocks: at block edges and in tet orders without
locality (the 256-vertex cap) against the vector-atomics variant."""
import numpy as np
import pytest

import xpbd_gb300 as G

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ckind", [G.CONSTRAINT_COMBINED, G.CONSTRAINT_SEPARATE])
@pytest.mark.parametrize("dims,shuffle", [((1, 1, 1), False), ((4, 4, 2), False), ((3, 11, 1), False),
                                          ((7, 9, 5), False), ((7, 9, 5), True), ((12, 11, 13), True)])
def test_block_sums_equal_atomics(lib, dims, shuffle, ckind):
    X, tets, faces = G.grid_mesh(*dims, 0.1 / 64)
    if shuffle:
        tets = np.random.default_rng(0).permutation(tets)
    x = X + 1e-5 * np.random.default_rng(1).uniform(-1, 1, X.shape)
    def run(var, press):
        s = G.XPBDSolver(X, tets, faces, 3e3, 0.45, 1000.0, dt=2e-4, num_iters=6, solver_type=G.SOLVER_JACOBI,
                         jacobi_variant=var, constraint_type=ckind, collision_rate=0.0)
        s.fix_vertices(X[:, 2] == 0)
        s.set_positions(x)
        if press:
            s.set_spheres([[X[:, 0].max() / 2, X[:, 1].max() / 2, X[:, 2].max() + 0.98e-2]], [1e-2])
            s.detect_collisions()
        s.step(3)
        assert s.health()[0] == 0
        out = s.positions(), s.lambdas()
        s.close()
        return out

    a, b = run(G.JACOBI_GATHER, False), run(G.JACOBI_GATHER, False)
    np.testing.assert_array_equal(a[0], b[0])
    np.testing.assert_array_equal(a[1], b[1])
    # the order of at most a few dozen FP32 additions a vertex and iteration, as
    # between two runs of the atomics (which contacts use in both variants)
    for press in (False, True):
        d = run(G.JACOBI_GATHER, press)[0] - run(G.JACOBI_ATOMIC, press)[0]
        assert np.abs(d).max() <= 1e-5 * np.abs(X).max()
