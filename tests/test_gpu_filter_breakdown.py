"""A filter whose CG breaks down in its first iteration (p.q underflows while
r.r does not) returns zeros: the iterate is still 0, and the direction buffer
that iteration 0 does not write has no part in the result, whatever an earlier
call or the allocator left in it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

BREAKDOWN = 3
TINY = 5e-324  # the smallest subnormal


def _filter(ctx, rho, radius):
    import torch
    d = torch.from_numpy(np.asarray(rho, np.float64)).cuda()
    out = torch.full_like(d, 7.0)
    torch.cuda.synchronize()
    with pytest.raises(Exception) as e:
        ctx.filter_device(d.data_ptr(), out.data_ptr(), radius)
    assert e.value.status == BREAKDOWN
    return out.cpu().numpy()


def test_breakdown_in_the_first_iteration_gives_zeros(hx):
    with hx.Context(0) as ctx:
        ctx.set_grid(3, 1, 1)
        # Leaves NaN in the direction of iteration 1.  r = a (1, -1, -1, 1) along x and
        # A ~ R^2 diag(1, 2, 2, 1) / 3: the terms of r.D^-1 r are 3 and 1.5 times a^2 / R^2,
        # those of p.Ap 3.375 and 1.6875 times; with a^2 / R^2 = 0.157 TINY all of the
        # former are below half of TINY and vanish, some of the latter are not:
        # alpha = 0, beta = 0 / 0.
        R = 1e7
        a = R * np.sqrt(0.157) * np.sqrt(TINY)
        _filter(ctx, 8 * a * np.array([1.0, -2.0, 1.0]), R)
        # r ~ 1e-150 and A ~ 1e26: r.r is 1e-300, p.q underflows in iteration 0
        out = _filter(ctx, np.full(3, 1e-150), 1e13)
    assert np.all(out == 0.0)
