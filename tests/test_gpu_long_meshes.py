"""Meshes and grids that are very long along one axis, where a kernel's blocks
pass the extent (65535) of a launch's y or z dimension.

The same beam of several hundred thousand elements along y and along x: 20 iterations of each CG form from zero,
which differ by rounding only (K x of a mesh with its axes exchanged; 1e-9 of the
largest displacement for FP64, 1e-4 for the FP32 iterations)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

N = 330000


def _iterate(hx, axis, **kw):
    dims = [1, 1, 1]
    dims[axis] = N
    bc = np.zeros((4 * (N + 1), 3), np.float32, order="F")
    f = np.zeros(12 * (N + 1))
    shape = tuple(d + 1 for d in dims[::-1])  # z, y, x
    first = [slice(None)] * 3
    first[2 - axis] = slice(0, 1)
    for c in range(3):
        bc[:, c].reshape(shape)[tuple(first)] = 1.0
    rng = np.random.default_rng(3)
    along = rng.uniform(0.5, 1.0, N + 1)
    load = f.reshape(shape + (3,))
    load[..., 2] = along.reshape([N + 1 if 2 - axis == a else 1 for a in range(3)])
    fac = rng.uniform(0.5, 1.0, N)
    with hx.Context(0) as ctx:
        ctx.set_grid(*dims)
        ctx.set_material(1.0, 0.3)
        ctx.set_bc(bc)
        u, rep = ctx.solve(f, fac, tol=1e-12, max_iter=20, ok=(0, 1), **kw)
    assert rep.status == 1 and rep.iterations == 20
    u = u.reshape(shape + (3,))
    # nodes as (position along the beam, across, z), components (along, across, z)
    if axis == 0:
        return u.transpose(2, 1, 0, 3)
    return u.transpose(1, 2, 0, 3)[..., [1, 0, 2]]


@pytest.mark.parametrize("kw,tol", [(dict(), 1e-9), (dict(precision=1), 1e-4)])
def test_a_long_beam_along_y(hx, kw, tol):
    ux, uy = _iterate(hx, 0, **kw), _iterate(hx, 1, **kw)
    assert np.abs(ux).max() > 0
    assert np.abs(ux - uy).max() <= tol * np.abs(ux).max()


def test_network_gradients_on_a_long_grid(hx):
    """A grid of 33000 nodes in z (8250 tiles for each of the layers' 8 uses) against its four
    quarters: dy is 0 but for the middle of each, 16 nodes (the reach of 8 layers and as much
    again) from the ends, so that the gradients are the sums of the quarters' (FP32 sums in
    another order: 1e-4 of the largest)."""
    import importlib
    learned = importlib.import_module("2025_12_09_hexat_v069_b200.learned")
    nz, q = 33000, 8250
    rng = np.random.default_rng(5)
    x0 = rng.standard_normal((nz, 2, 2, 16)).astype(np.float32)
    dy = np.zeros_like(x0)
    for i in range(4):
        dy[i * q + 16:(i + 1) * q - 16] = rng.standard_normal((q - 32, 2, 2, 16))
    with hx.Context(0) as ctx:
        ctx.set_grid(4, 4, 4)
        ctx.set_material(1.0, 0.3)
        ctx.net_set_params(learned.load_params())
        _, g = ctx.net_forward_backward((2, 2, nz), x0.reshape(-1, 16), dy.reshape(-1, 16))
        s = np.zeros_like(g)
        for i in range(4):
            cut = slice(i * q, (i + 1) * q)
            s += ctx.net_forward_backward((2, 2, q), x0[cut].reshape(-1, 16),
                                          dy[cut].reshape(-1, 16))[1]
    assert np.abs(g).max() > 0
    assert np.abs(g - s).max() <= 1e-4 * np.abs(g).max()
