"""The snapshot of the best iterate (hx_solve with ref_retry = 1, keep_best =
1), taken inside the fused step of the next iteration and, for the last
iteration, after the loop.  The solve is deterministic, so a run stopped at
m iterations without snapshots returns x_m of the longer run; the stalled
run's answer has to be the x_m of lowest residual (up to the contraction of
x + alpha p in the two kernels that form it, 1e-12)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

DIMS = (40, 2, 2)
STALLED = 2


def _setup(ctx, hx):
    nodes, el, bc, f = hx.workloads.cantilever(*DIMS)
    fac = np.ones(el.shape[0])
    ctx.set_grid(*DIMS)
    ctx.set_material(1.0, 0.3)
    ctx.set_bc(bc)
    return f, fac


# The residual of this beam has a local minimum at 137 and at 143: there the best
# iterate lies one or two iterations before the last one; elsewhere it is the last.
# Odd and even ends use either of the two direction buffers.
@pytest.mark.parametrize("max_iter", [136, 137, 138, 139, 140, 143, 144, 145])
def test_stalled_solve_returns_the_iterate_of_lowest_residual(ctx, hx, max_iter):
    f, fac = _setup(ctx, hx)
    kw = dict(tol=1e-12, shift_factor=1e-9, check_every=1, ok=range(10))
    runs = [ctx.solve(f, fac, max_iter=m, ref_retry=0, keep_best=0, **kw)
            for m in range(130, max_iter + 1)]
    best = min(runs, key=lambda r: r[1].rel_res)
    u, rep = ctx.solve(f, fac, max_iter=max_iter, ref_retry=1, keep_best=1, **kw)
    assert rep.status == STALLED and rep.attempts == 1
    assert np.linalg.norm(u - best[0]) <= 1e-12 * np.linalg.norm(best[0])
