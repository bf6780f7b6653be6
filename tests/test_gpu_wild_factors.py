"""Factors that are not numbers.  A node next to a NaN factor carries no
(positive) stiffness and is held fixed, and a factor among fixed nodes has no part
in any free row: the solve is that of the rest, in every form.

Against the oracle with the NaN elements' nodes fixed and all such factors 0, at the tolerances of
the other solve tests (tol 1e-10 for FP64: 1e-8; tol 1e-8 for the mixed forms: 1e-5)."""
import importlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

DIMS = (12, 6, 5)


def _system(hx, orc):
    nx, ny, nz = DIMS
    nodes, el, bc, f = hx.workloads.cantilever(*DIMS)
    c0 = hx.mesh.connectivity0(el)
    b = [bc[:, c].reshape(nz + 1, ny + 1, nx + 1) for c in range(3)]
    for a in b:
        a[:, :, 1] = 1.0  # the first layer of elements lies among fixed nodes
    fac = hx.workloads.simp(np.random.default_rng(9).uniform(0.3, 1.0, el.shape[0]))
    e = fac.reshape(nz, ny, nx)
    e[:, :, 0] = np.inf
    e[2, 1, 0] = np.nan
    e[2, 3, 6] = e[0, 0, 9] = np.nan
    clean = np.where(np.isfinite(fac), fac, 0.0)
    bo = bc.copy()
    bo[np.unique(c0[np.isnan(fac)])] = 1.0
    nN = nodes.shape[0]
    ke = orc.canonical_ke(1.0, 1.0, 1.0, 0.3)
    free = orc.free_mask_from(bo, orc.diagonal(c0, nN, ke, clean))
    u, _, _, _ = orc.cg_solve(c0, nN, ke, clean, free, f * free, tol=1e-11)
    return bc, f, fac, u


@pytest.mark.parametrize("precond", [0, 1, 3])
@pytest.mark.parametrize("precision", [0, 1])
def test_solves_of_the_rest(hx, orc, precond, precision):
    bc, f, fac, uo = _system(hx, orc)
    with hx.Context(0) as ctx:
        ctx.set_grid(*DIMS)
        ctx.set_material(1.0, 0.3)
        ctx.set_bc(bc)
        if precond == 1:
            importlib.import_module("2025_12_09_hexat_v069_b200.learned").load_into(ctx)
        u, rep = ctx.solve(f, fac, tol=1e-8 if precision else 1e-10, preconditioner=precond,
                           precision=precision)
    assert rep.status == 0
    assert np.abs(u - uo).max() <= (1e-5 if precision else 1e-8) * np.abs(uo).max()


def test_device_arrays_keep_the_callers_factors(hx, orc):
    import torch
    bc, f, fac, uo = _system(hx, orc)
    with hx.Context(0) as ctx:
        ctx.set_grid(*DIMS)
        ctx.set_material(1.0, 0.3)
        ctx.set_bc(bc)
        fd, facd = torch.from_numpy(f).cuda(), torch.from_numpy(fac).cuda()
        ud = torch.zeros_like(fd)
        snaps = torch.zeros((400, f.size), dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        ctx.solve_device(fd.data_ptr(), facd.data_ptr(), ud.data_ptr(), tol=1e-10)
        n = ctx.pcg_snapshots(fd.data_ptr(), facd.data_ptr(), 2, 400, 1e-10, snaps.data_ptr())
        assert np.array_equal(facd.cpu().numpy(), fac, equal_nan=True)
        assert np.abs(ud.cpu().numpy() - uo).max() <= 1e-8 * np.abs(uo).max()
        assert 0 < n < 400
        assert np.abs(snaps[n - 1].cpu().numpy() - uo).max() <= 1e-4 * np.abs(uo).max()
        # and then a system without any
        ok = torch.where(torch.isfinite(facd), facd, 0.5)
        torch.cuda.synchronize()
        rep = ctx.solve_device(fd.data_ptr(), ok.data_ptr(), ud.data_ptr(), tol=1e-10)
    assert rep.status == 0 and rep.true_rel_res < 1e-9
