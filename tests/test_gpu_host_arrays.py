"""Host arrays of the caller that are not aligned to their type (a field of a
packed record, a buffer at an odd offset): the device cannot read them itself,
so the host copies them."""
import numpy as np
import pytest

import xpbd_gb300 as G

pytestmark = pytest.mark.gpu


def _odd(a, offset):
    """a's values at `offset` bytes past an aligned address."""
    a = np.ascontiguousarray(a)
    buf = np.zeros(a.nbytes + 16, np.uint8)
    at = (-buf.ctypes.data) % 16 + offset
    v = buf[at:at + a.nbytes].view(a.dtype).reshape(a.shape)
    v[...] = a
    assert v.ctypes.data % a.itemsize == offset % a.itemsize
    return v


@pytest.mark.parametrize("offset", [1, 2, 4, 8])
def test_unaligned_rows_and_targets(lib, offset):
    """Offsets 4 and 8 are aligned floats (read by the device, not in 16-byte
    pieces); 1 and 2 are not."""
    X, tets, _ = G.grid_mesh(2, 2, 2, 0.1)
    s = G.XPBDSolver(X, tets, None, 3e3, 0.45, 1000.0)
    s.mlp_init(3)
    rng = np.random.default_rng(0)
    rows = rng.normal(size=(300, 16)).astype(np.float32)
    y = rng.normal(size=(300, 2)).astype(np.float32)
    out = s.mlp_forward(rows)
    np.testing.assert_array_equal(s.mlp_forward(_odd(rows, offset)), out)
    loss, grad = s.mlp_loss_grad(rows, y)
    for r, t in ((_odd(rows, offset), y), (rows, _odd(y, offset)), (_odd(rows, offset), _odd(y, offset))):
        l2, g2 = s.mlp_loss_grad(r, t)
        # the sums' order is the atomics'
        assert abs(l2 - loss) <= 1e-12 * abs(loss)
        assert np.abs(g2 - grad).max() <= 1e-5 * np.abs(grad).max()
    s.close()


@pytest.mark.parametrize("offset", [1, 2, 4])
def test_unaligned_positions_and_velocities(lib, offset):
    X, tets, _ = G.grid_mesh(3, 2, 2, 0.1)
    s = G.XPBDSolver(X, tets, None, 3e3, 0.45, 1000.0)
    s.fix_vertices(X[:, 2] == 0)
    x = X + 0.01 * np.random.default_rng(1).normal(size=X.shape)
    f = x.astype(np.float32)
    s.set_positions(_odd(x, offset))
    np.testing.assert_array_equal(s.positions(), f.astype(np.float64))
    s.set_positions_f32(_odd(f + np.float32(0.5), offset))
    out = _odd(np.zeros_like(f), offset)
    s.positions_f32(out=out)
    np.testing.assert_array_equal(out, f + np.float32(0.5))
    s.set_velocities(_odd(x, offset))
    np.testing.assert_array_equal(s.velocities(), f.astype(np.float64))
    s.close()
