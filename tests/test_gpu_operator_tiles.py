"""The structured operator at the edges of its tiles and chunks: one thread
block owns 31 x 7 node columns (FP64, K x), 31 x 5 (FP64, fused steps) or
31 x 7 (FP32, two element rows per thread), over a chunk of z-planes whose
length depends on the grid.

Tolerances: K x against the FP64 oracle to 1e-12 of its largest entry (the
same operator, other summation order); the fused steps through the solves
they carry: the FP64 and the mixed solution to 1e-8 at tol 1e-10 (contrast
<= 1e3 here, as in the parity tests).  The FP32 multigrid cycle is a symmetric operator up to
rounding: fewer than 100 dependent FP32 operations of amplification below 10
leave 100 x 10 x 6e-8 = 6e-5, tested at 1e-4."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EDGES = [(1, 1, 1), (1, 7, 2), (30, 6, 3), (31, 7, 4), (32, 8, 5), (62, 14, 9), (61, 13, 1),
         (2, 30, 40), (93, 4, 3)]


@pytest.mark.parametrize("nu", [0.3, 0.0, -0.2])
@pytest.mark.parametrize("h", [(1.0, 1.0, 1.0), (0.5, 0.5, 0.5), (1.3, 0.7, 2.1)])
def test_apply_at_tile_edges(ctx, hx, orc, h, nu):
    for dims in EDGES:
        nodes, el, _ = hx.mesh.generate_mesh(*dims)
        c0 = hx.mesh.connectivity0(el)
        ctx.set_grid(*dims, *h)
        ctx.set_material(1.0, nu)
        rng = np.random.default_rng(sum(dims))
        fac = rng.uniform(0.0, 1.0, c0.shape[0])
        fac[rng.uniform(size=fac.shape) < 0.2] = 0.0
        x = rng.standard_normal(3 * nodes.shape[0])
        yo = orc.apply_stiffness(c0, nodes.shape[0], orc.canonical_ke(*h, nu), fac, x)
        y = ctx.apply_stiffness(x, fac)
        assert np.abs(y - yo).max() <= 1e-12 * max(1.0, np.abs(yo).max()), dims


@pytest.mark.parametrize("h", [(1.0, 1.0, 1.0), (1.0, 0.8, 1.25)])
@pytest.mark.parametrize("dims", [(30, 6, 3), (31, 7, 8), (32, 8, 5), (62, 10, 4), (16, 16, 21)])
def test_fused_steps_at_tile_edges(ctx, hx, orc, dims, h):
    nodes, el, bc, f = hx.workloads.cantilever(*dims)
    c0 = hx.mesh.connectivity0(el)
    ctx.set_grid(*dims, *h)
    ctx.set_material(1.0, 0.3)
    ctx.set_bc(bc)
    fac = hx.workloads.simp(np.random.default_rng(3).uniform(0.1, 1.0, c0.shape[0]))
    ke, nN = orc.canonical_ke(*h, 0.3), nodes.shape[0]
    free = orc.free_mask_from(bc, orc.diagonal(c0, nN, ke, fac))
    uo, _, _, _ = orc.cg_solve(c0, nN, ke, fac, free, f * free, tol=1e-10)
    u, rep = ctx.solve(f, fac, tol=1e-10)
    um, rm = ctx.solve(f, fac, tol=1e-10, precision=1)
    assert np.abs(u - uo).max() <= 1e-8 * np.abs(uo).max()
    assert np.abs(um - uo).max() <= 1e-8 * np.abs(uo).max()
    assert np.all(u[free == 0] == 0.0) and np.all(um[free == 0] == 0.0)


@pytest.mark.parametrize("dims", [(64, 16, 16), (60, 28, 16)])
def test_multigrid_cycle_is_symmetric(ctx, hx, dims):
    import torch
    nodes, el, bc, f = hx.workloads.cantilever(*dims)
    ctx.set_grid(*dims)
    ctx.set_material(1.0, 0.3)
    ctx.set_bc(bc)
    fac = hx.workloads.simp(np.random.default_rng(4).uniform(0.1, 1.0, el.shape[0]))
    ctx.solve(f, fac, tol=1e-6, preconditioner=3)
    free = torch.from_numpy(bc.reshape(-1) == 0).cuda().double()
    g = torch.Generator(device="cuda").manual_seed(5)
    r = [torch.randn(f.size, generator=g, dtype=torch.float64, device="cuda") * free
         for _ in range(2)]
    z = [torch.empty_like(v) for v in r]
    torch.cuda.synchronize()
    for a, b in zip(r, z):
        ctx.gmg_apply(a.data_ptr(), b.data_ptr())
    for v in z:
        assert float((v * (1 - free)).abs().max()) == 0.0
    a, b = float(z[0] @ r[1]), float(z[1] @ r[0])
    assert abs(a - b) <= 1e-4 * float(z[0].norm() * r[1].norm())
    assert float(z[0] @ r[0]) > 0 and float(z[1] @ r[1]) > 0
