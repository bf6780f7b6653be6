"""Device allocations of training steps and gradient checks: the first of a
context makes a few, later ones none.  Counted in a child process whose cudaMalloc is wrapped
by a small preloaded library."""
import os
import subprocess
import sys

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

WRAP = r"""
#define _GNU_SOURCE
#include <dlfcn.h>
#include <stddef.h>
static int n;
int cudaMalloc(void **p, size_t s) {
  static int (*real)(void **, size_t);
  if (!real) real = (int (*)(void **, size_t))dlsym(RTLD_NEXT, "cudaMalloc");
  ++n;
  return real(p, s);
}
int cuda_mallocs(void) { return n; }
"""

CHILD = r"""
import ctypes, importlib, sys
import numpy as np
import torch
hx = importlib.import_module("2025_12_09_hexat_v069_b200")
learned = importlib.import_module("2025_12_09_hexat_v069_b200.learned")
count = ctypes.CDLL(sys.argv[1]).cuda_mallocs
dims = (32, 16, 16)
n, ne = 3 * 33 * 17 * 17, 32 * 16 * 16
kw = dict(dtype=torch.float64, device="cuda")
fac, e, r = torch.ones(ne, **kw), torch.randn(n, **kw), torch.randn(n, **kw)
torch.cuda.synchronize()
with hx.Context(0) as ctx:
    ctx.set_grid(*dims)
    ctx.set_material(1.0, 0.3)
    ctx.net_set_params(learned.load_params())
    ctx.net_prepare(fac.data_ptr())
    c = [count()]
    for _ in range(2):
        ctx.net_train_batch([r.data_ptr()], [e.data_ptr()], 1e-4)
        c.append(count())
    a = np.random.default_rng(0).standard_normal((9 * 9 * 9, 16)).astype(np.float32)
    y, grads = ctx.net_forward_backward((9, 9, 9), a, a)
    c.append(count())
    y2, grads2 = ctx.net_forward_backward((9, 9, 9), a, a)
    assert np.array_equal(y, y2) and np.array_equal(grads, grads2)
    c.append(count())
    # a training step after it places its buffers anew
    p = learned.load_params()
    out = []
    for fb in (False, True):
        ctx.net_set_params(p)
        if fb:
            ctx.net_forward_backward((9, 9, 9), a, a)
        ctx.net_train_batch([r.data_ptr()], [e.data_ptr()], 1e-4)
        out.append(ctx.net_get_params())
    assert np.array_equal(*out)
print("allocations", c[0], *(b - a for a, b in zip(c, c[1:])))
"""


def test_allocations_of_training_steps(tmp_path):
    src, lib = tmp_path / "wrap.c", tmp_path / "wrap.so"
    src.write_text(WRAP)
    subprocess.run(["gcc", "-shared", "-fPIC", "-o", str(lib), str(src), "-ldl"], check=True)
    env = dict(os.environ, LD_PRELOAD=str(lib), PYTHONPATH=ROOT)
    out = subprocess.run([sys.executable, "-c", CHILD, str(lib)], env=env, cwd=ROOT, timeout=300,
                         capture_output=True, text=True)
    assert out.returncode == 0, out.stderr
    before, first, second, fb, fb2 = map(int, out.stdout.split("allocations")[1].split())
    assert before > 0  # the wrapper is in place
    # vectors of the mesh and one block for the networks' training buffers
    assert first <= 12 and second == 0, (first, second)
    # the gradient check on given data uses that block
    assert fb <= 1 and fb2 == 0, (fb, fb2)
