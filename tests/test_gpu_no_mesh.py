"""Calls that bring their own grid as the first ones of a context, before any
mesh is set: the reference-shaped filter and the density update.  Run in a child
process (a crash there is a failure here) and compared with a context that has a
mesh: the same kernels on the same grids, so bit for bit."""
import subprocess
import sys

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

CHILD = r"""
import importlib
import numpy as np
hx = importlib.import_module("2025_12_09_hexat_v069_b200")
api = importlib.import_module("2025_12_09_hexat_v069_b200.api")
dims = (15, 6, 7)
n = 15 * 6 * 7
rng = np.random.default_rng(1)
rho, l1, orig = (rng.uniform(0.1, 1.0, n).astype(np.float32) for _ in range(3))
prot = rng.uniform(size=n) < 0.1
cfg = {"geometry": {"nElem_x_computed": 15, "nElem_y_computed": 6, "nElem_z_computed": 7,
                    "dx_computed": 1.0, "dy_computed": 1.0, "dz_computed": 1.0,
                    "max_domain_dim": 15.0},
       "optimization_parameters": {"filter_R_init_perc": 8.0, "filter_R_interm_perc": 5.0,
                                   "filter_R_final_perc": 3.0},
       "solver_parameters": {"filter_tolerance": 1e-5}}

def run(ctx):
    f = api.apply_gpu_filter(rho, *dims, 1.0, 1.0, 1.0, 1.2, ctx=ctx)
    d = rho.copy()
    u = api.update_density(d, l1.copy(), prot, 1.0, 1.0, 7, 40, orig, 1e-3, 1.0, cfg, ctx=ctx)
    return f[0], f[2], d, u[0], u[4]

def update_first(ctx):
    d = rho.copy()
    api.update_density(d, l1.copy(), prot, 1.0, 1.0, 7, 40, orig, 1e-3, 1.0, cfg, ctx=ctx)
    return d

with hx.Context(0) as a, hx.Context(0) as b, hx.Context(0) as c:
    b.set_grid(40, 9, 9)
    ra, rb = run(a), run(b)
    assert ra[0].size == n and ra[1] > 0
    for x, y in zip(ra, rb):
        assert np.array_equal(x, y)
    assert np.array_equal(update_first(c), ra[2])
print("done")
"""


def test_filter_and_update_before_any_mesh():
    out = subprocess.run([sys.executable, "-c", CHILD], cwd=ROOT, timeout=300,
                         capture_output=True, text=True)
    assert out.returncode == 0 and "done" in out.stdout, (out.returncode, out.stderr)
