"""Wall-clock limit of a solve: HX_NOT_CONVERGED stands for a solution that is
not converged, and the work after the limit is at most the batch of iterations
in flight when it passed."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FORMS = [dict(), dict(precision=1), dict(preconditioner=3), dict(preconditioner=3, precision=1)]


def _beam(ctx, hx, dims):
    nodes, el, bc, f = hx.workloads.cantilever(*dims)
    ctx.set_grid(*dims)
    ctx.set_material(1.0, 0.3)
    ctx.set_bc(bc)
    return f, hx.workloads.simp(np.full(el.shape[0], 1.0))


@pytest.mark.parametrize("form", FORMS)
def test_a_converged_solve_is_not_reported_as_timed_out(ctx, hx, form):
    f, fac = _beam(ctx, hx, (8, 4, 4))
    tol = 1e-4
    full = ctx.solve(f, fac, tol=tol, **form)[1]
    assert full.status == 0
    # a batch of two thirds of the iterations: converged in the second one
    batch = full.iterations * 2 // 3 // 2 * 2
    for limit in (1e-6, 0.05, 0.1, 0.2, 0.4, 0.8, 1.6, 3.2):
        rep = ctx.solve(f, fac, tol=tol, wall_limit_ms=limit, check_every=batch, ok=(0, 1),
                        **form)[1]
        assert (rep.status == 0) == (rep.true_rel_res < tol), (limit, rep.as_dict())


def test_limit_ends_the_solve_after_the_batch_in_flight(ctx, hx):
    f, fac = _beam(ctx, hx, (60, 20, 20))
    rep = ctx.solve(f, fac, tol=1e-10, wall_limit_ms=1e-6, check_every=16, ok=(0, 1))[1]
    assert rep.status == 1 and rep.iterations == 16
