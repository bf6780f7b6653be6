"""Filters on few, long rows of nodes, whose vector kernels cut the rows into
segments of a multiple of 32 nodes.

Tolerance as in test_gpu_filter_oc_edges: the oracle's CG in another summation
order, equal iteration counts, 1e-10 absolute for densities in [0, 1]."""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(127, 1, 1), (128, 1, 1), (129, 2, 1), (1000, 1, 1),
                                  (1, 1000, 1), (321, 3, 5), (2000, 5, 2)])
def test_filter_of_long_rows(ctx, hx, orc, dims):
    ctx.set_grid(*dims)
    nodes, el, _ = hx.mesh.generate_mesh(*dims)
    n = el.shape[0]
    rho = np.random.default_rng(n).uniform(0.0, 1.0, n)
    f, rep = ctx.filter(rho, 1.7, 0)
    fo, ito, _ = orc.helmholtz_filter(hx.mesh.connectivity0(el), nodes.shape[0], rho, 1.0, 1.0, 1.0,
                                      1.7, 0)
    assert rep.iterations == ito
    assert np.abs(f - fo).max() <= 1e-10


def test_a_long_row_is_not_one_warps_work(ctx):
    """100000 x 1 x 1 elements: 0.8 ms with the row cut, 20 ms by one warp per row."""
    import torch
    n = 100000
    rho = torch.rand(n, dtype=torch.float64, device="cuda")
    out = torch.empty_like(rho)
    torch.cuda.synchronize()
    ctx.set_grid(n, 1, 1)
    best = 1e9
    for _ in range(6):
        t = time.perf_counter()
        ctx.filter_device(rho.data_ptr(), out.data_ptr(), 1.5)
        best = min(best, time.perf_counter() - t)
    assert best < 5e-3
