"""Multigrid cycles on the row lengths where the row-wise grid transfers and
the FP32 cycle vectors of the FP64 solve change form: rows shorter than a
warp, rows of more than one pass of a CTA (256 coarse DOFs in the restriction,
512 fine ones in the prolongation), odd DOF counts (every grid here has an odd
node count, so the 2-wide residual update ends in a scalar tail)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

DIMS = [(4, 10, 20), (20, 12, 4), (10, 14, 30), (84, 6, 8), (256, 4, 4), (260, 6, 4), (400, 4, 8)]


@pytest.mark.parametrize("dims", DIMS)
def test_cycle_is_symmetric_and_the_solve_matches_jacobi(ctx, hx, dims):
    """The restriction is the transpose of the prolongation, so the cycle stays
    symmetric up to FP32 rounding; with the shift at 1e-3 x max diag the
    condition number is below 5e3, so two solves to 1e-10 agree to 1e-6."""
    import torch
    nodes, el, bc, f = hx.workloads.cantilever(*dims)
    ctx.set_grid(*dims)
    ctx.set_material(1.0, 0.3)
    ctx.set_bc(bc)
    rng = np.random.default_rng(5)
    fac = hx.workloads.simp(rng.uniform(0.1, 1.0, el.shape[0]))
    kw = dict(tol=1e-10, shift_factor=1e-3, max_iter=20000)
    uj, rj = ctx.solve(f, fac, **kw)
    um, rm = ctx.solve(f, fac, preconditioner=3, **kw)
    assert rj.status == 0 and rm.status == 0 and rm.true_rel_res < 1e-9
    assert rm.iterations < rj.iterations
    assert np.linalg.norm(um - uj) <= 1e-6 * np.linalg.norm(uj)

    dev = torch.device("cuda", 0)
    free = torch.from_numpy(bc.reshape(-1) == 0).to(dev)
    g = torch.Generator(device="cpu").manual_seed(1)
    r = [torch.randn(f.size, generator=g, dtype=torch.float64).to(dev) * free for _ in range(2)]
    z = [torch.empty_like(v) for v in r]
    for v, out in zip(r, z):
        ctx.gmg_apply(v.data_ptr(), out.data_ptr())
    scale = np.sqrt(float(r[0] @ z[0]) * float(r[1] @ z[1]))
    assert abs(float(r[0] @ z[1]) - float(r[1] @ z[0])) <= 1e-5 * scale
    assert not torch.any(z[0][~free])


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("precision", [0, 1])
def test_host_inputs_copied_beside_the_set_up(ctx, hx, dtype, precision):
    """Host calls copy f and u beside the multigrid set-up: each call in a row with
    new loads, factors and initial guesses, in both types, matches the Jacobi
    solve of the same call.  Condition number below 5e3 and both solves to 1e-9:
    1e-5, which also covers the Float32 of inputs (the same for both) and results."""
    dims = (36, 20, 12)
    nodes, el, bc, f = hx.workloads.cantilever(*dims)
    ctx.set_grid(*dims)
    ctx.set_material(1.0, 0.3)
    ctx.set_bc(bc)
    rng = np.random.default_rng(11)
    kw = dict(tol=1e-9, shift_factor=1e-3, max_iter=20000)
    for call in range(4):
        fac = hx.workloads.simp(rng.uniform(0.1, 1.0, el.shape[0])).astype(dtype)
        load = (f * (call + 1) + rng.standard_normal(f.size) * (bc.reshape(-1) == 0)).astype(dtype)
        u0 = rng.standard_normal(f.size).astype(dtype) if call % 2 else None
        um, rm = ctx.solve(load, fac, u0=u0, preconditioner=3, precision=precision, **kw)
        uj, rj = ctx.solve(load, fac, **kw)
        assert rm.status == 0 and rj.status == 0
        d = um.astype(np.float64) - uj.astype(np.float64)
        assert np.linalg.norm(d) <= 1e-5 * np.linalg.norm(uj.astype(np.float64)), call
