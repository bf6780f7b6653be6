"""Which grids the allocation-free operator takes: it launches K x alone, with
one partial sum per thread block of 31 x 7 node columns, and refuses grids of
more than 16384 of them (about 1880 x 1880 nodes per plane).

Without a device an accepted grid ends with HX_CUDA_ERROR when the scratch
array's address is asked for, a refused one with HX_BAD_ARG before that."""
import ctypes
import time

import numpy as np
import pytest

BAD_ARG, CUDA_ERROR = 6, 7


def _call(hx, dims, x, fac, y, xkx, stream=None):
    return hx.load().hx_apply_stiffness_noalloc(*dims, 1.0, 1.0, 1.0, 0.3, x, fac, y, xkx, stream)


@pytest.mark.parametrize("dims,want", [
    ((16, 8, 8), CUDA_ERROR),
    ((750, 650, 400), CUDA_ERROR),    # 25 x 93 columns, each one chunk long
    ((1000, 450, 400), CUDA_ERROR),
    ((1700, 1700, 8), CUDA_ERROR),    # 55 x 243 = 13365
    ((1875, 1875, 1), CUDA_ERROR),    # 61 x 268 = 16348
    ((1876, 1876, 1), BAD_ARG),       # 61 x 269 = 16409
    ((100000, 10000, 1), BAD_ARG),
])
def test_grids_taken_without_a_device(hx, dims, want):
    import torch
    if torch.cuda.is_available():
        pytest.skip("a GPU is present: the call would run")
    a = np.zeros(8)
    p = a.ctypes.data + (-a.ctypes.data) % 16
    assert _call(hx, dims, p, p, p, p) == want


def test_blocks_of_a_tall_grid_are_counted_quickly(hx):
    """A million planes: 25 us over the useful chunk lengths, 3.5 ms over all of them."""
    import torch
    if torch.cuda.is_available():
        pytest.skip("a GPU is present: the call would run")
    a = np.zeros(8)
    p = a.ctypes.data + (-a.ctypes.data) % 16
    best = 1e9
    for _ in range(10):
        t = time.perf_counter()
        assert _call(hx, (1, 1, 1000000), p, p, p, p) == CUDA_ERROR
        best = min(best, time.perf_counter() - t)
    assert best < 1e-3


@pytest.mark.gpu
def test_most_partial_sums(hx, ctx):
    """13365 blocks: y as the context's operator gives it (the same kernel), x.y by its own sum
    (both to rounding: 1e-12 of the sum of magnitudes)."""
    import torch
    dims = (1700, 1700, 1)
    n, ne = 3 * 1701 * 1701 * 2, 1700 * 1700
    g = torch.Generator(device="cuda").manual_seed(6)
    kw = dict(dtype=torch.float64, device="cuda")
    x, fac = torch.randn(n, generator=g, **kw), torch.rand(ne, generator=g, **kw)
    y, s = torch.empty(n, **kw), torch.empty(1, **kw)
    st = _call(hx, dims, x.data_ptr(), fac.data_ptr(), y.data_ptr(), s.data_ptr(),
               ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert st == 0
    torch.cuda.synchronize()
    ctx.set_grid(*dims)
    ctx.set_material(1.0, 0.3)
    yr = ctx.apply_stiffness(x.cpu().numpy(), fac.cpu().numpy())
    assert np.array_equal(y.cpu().numpy(), yr)
    assert abs(float(s) - float(x @ y)) <= 1e-12 * float((x * y).abs().sum())
