"""opts.check_every, the host poll period in iterations, in the learned forms:
a graph launch holds that many iterations, so a solve launches whole multiples
of their kernels."""
import importlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [0, 1])
def test_poll_period_of_the_learned_forms(hx, precision):
    learned = importlib.import_module("2025_12_09_hexat_v069_b200.learned")
    nodes, el, bc, f = hx.workloads.cantilever(24, 12, 12)
    fac = hx.workloads.simp(np.random.default_rng(8).uniform(0.3, 1.0, el.shape[0]))
    with hx.Context(0) as ctx:
        ctx.set_grid(24, 12, 12)
        ctx.set_material(1.0, 0.3)
        ctx.set_bc(bc)
        learned.load_into(ctx)
        kw = dict(tol=1e-8, precision=precision, preconditioner=1, learned_no_fallback=1)
        reps = {p: ctx.solve(f, fac, check_every=p, **kw)[1] for p in (0, 2, 20, 600)}
    its = {p: r.iterations for p, r in reps.items()}
    n = {p: r.kernel_launches for p, r in reps.items()}
    assert all(r.status == 0 for r in reps.values())
    assert len(set(its.values())) == 1  # the same iterations
    per = n[2] / its[2]                 # kernels per iteration, about
    assert its[2] < 600
    assert n[600] >= 600 * 0.8 * per
    assert n[0] == n[2] < n[20] < n[600]
