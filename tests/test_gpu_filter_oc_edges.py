"""The filter's step at the edges of its 32 x 8 tiles and z-chunks, and the OC
bisection taken several steps per pass.

Tolerances: the filter runs the oracle's CG in another summation order; at
the iteration counts used here (<= 40, equal to the oracle's) rounding stays below
1e-10 absolute for densities in [0, 1], as in the parity tests.  The OC update
takes the oracle's decisions, so lambda and the step count are equal and
x_new differs by rounding only (1e-12)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("compat", [0, 1])
@pytest.mark.parametrize("dims", [(1, 1, 1), (31, 7, 3), (32, 8, 1), (30, 6, 9), (33, 15, 4),
                                  (63, 2, 40), (4, 40, 5)])
def test_filter_at_tile_edges(ctx, hx, orc, dims, compat):
    ctx.set_grid(*dims)
    nodes, el, _ = hx.mesh.generate_mesh(*dims)
    n = el.shape[0]
    rho = np.random.default_rng(n).uniform(0.0, 1.0, n)
    f, rep = ctx.filter(rho, 1.7, compat)
    fo, ito, _ = orc.helmholtz_filter(hx.mesh.connectivity0(el), nodes.shape[0], rho, 1.0, 1.0, 1.0,
                                      1.7, compat)
    assert rep.iterations == ito
    assert np.abs(f - fo).max() <= 1e-10


def test_filter_of_zeros_returns_the_input(ctx, hx):
    ctx.set_grid(9, 5, 4)
    f, rep = ctx.filter(np.zeros(180), 2.0, 0)
    assert rep.status == 0 and np.all(f == 0.0)


@pytest.mark.parametrize("n,volfrac", [(1, 0.3), (255, 0.3), (257, 0.05), (100000, 0.6)])
def test_oc_steps_match_the_oracle(ctx, hx, orc, n, volfrac):
    ctx.set_grid(n, 1, 1)
    rng = np.random.default_rng(n)
    x = rng.uniform(0.0, 1.0, n)
    dc = -rng.uniform(0.0, 1.0, n) ** 3
    dc[rng.uniform(size=n) < 0.1] = 0.0
    dv = rng.uniform(0.5, 1.0, n)
    for v in (dv, np.ones(n)):
        xn, lam, steps = ctx.oc_update(x, dc, v, volfrac, 0.2)
        xo, lamo, stepso = orc.oc_update(x, dc, v, volfrac, 0.2)
        assert steps == stepso and abs(lam - lamo) <= 1e-12 * lamo
        assert np.abs(xn - xo).max() <= 1e-12
