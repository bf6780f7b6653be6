"""The work that a user of this library has it do, as measurable cases.

listed() names the cases, draw() gives more of the same ranges, prepare()
makes what a program has in hand before the call, run() makes one pass
through the public entry points, work() says what a pass cannot do without,
and exact() computes the result in 64 bits with plain torch.

Kinds of pass:
  apply   K(f) x and x.K x on device arrays without allocation: the operator
          of a z-slab of a decomposed solve (hx_apply_stiffness_noalloc)
  grid    the reference-shaped drop-in solve with pruning on the device
          (api.solve_system_grid): Float32 host arrays, shift 1e-6, voids
  solve   hx_solve on pinned Float32 host arrays, in each solver form
  design  the design part of a GPU-resident optimisation iteration: filter,
          SIMP, compliance, sensitivities, their filter, the OC update
  stress  the reference's outer iteration after the solve: stress field and
          stress-ratio density update (Float32 host arrays)
  train   one Adam step of the learned preconditioner on residual / error
          pairs (forward and backward through all networks)
"""
import ctypes
import importlib

import numpy as np
import torch

hx = importlib.import_module("2025_12_09_hexat_v069_b200")
api = importlib.import_module("2025_12_09_hexat_v069_b200.api")
learned = importlib.import_module("2025_12_09_hexat_v069_b200.learned")
_lib = importlib.import_module("2025_12_09_hexat_v069_b200._lib")

NU = 0.3
PRECOND = {"jacobi": _lib.HX_PC_JACOBI, "learned": _lib.HX_PC_LEARNED,
           "multigrid": _lib.HX_PC_MULTIGRID}
PRECISION = {"fp64": _lib.HX_PREC_FP64, "mixed": _lib.HX_PREC_MIXED32}


# --------------------------------------------------------------------------
# cases
# --------------------------------------------------------------------------
def _solve(name, dims, precond, precision, support="cantilever", shift=0.0, warm=False):
    c = {"kind": "solve", "nx": dims[0], "ny": dims[1], "nz": dims[2], "precond": precond,
         "precision": precision, "support": support, "shift": shift, "warm": warm}
    return dict(c, name=name) if name else c


def _other(kind, name, dims, **kw):
    c = {"kind": kind, "nx": dims[0], "ny": dims[1], "nz": dims[2], **kw}
    return dict(c, name=name) if name else c


def listed():
    return [
        # the smallest call: the operator on a thin slab, all launch latency
        _other("apply", "apply_16x8x8", (16, 8, 8), h=1.0),
        # the operator at the scale workload's size (8.2M elements)
        _other("apply", "apply_320x160x160", (320, 160, 160), h=1.0),
        # the first mesh a user tries, through the drop-in call
        _other("grid", "dropin_60x20x20", (60, 20, 20)),
        # an odd, ragged mesh with the mixed-precision Jacobi form
        _solve("mixed_jacobi_97x45x51", (97, 45, 51), "jacobi", "mixed"),
        # the plain solve, the library's default, at 1.8M elements
        _solve("fp64_jacobi_192x96x96", (192, 96, 96), "jacobi", "fp64"),
        # the learned form on the grid its networks were trained on
        _solve("learned_128x64x64", (128, 64, 64), "learned", "mixed"),
        # the headline: the learned form on the scale workload
        _solve("learned_320x160x160", (320, 160, 160), "learned", "mixed"),
        # the fastest form on the scale workload
        _solve("multigrid_320x160x160", (320, 160, 160), "multigrid", "fp64"),
        # an optimisation loop's solve: near-0/1 design, warm start, free
        # rigid mode held by the shift
        _solve("mg_mbb_warm_240x80x80", (240, 80, 80), "multigrid", "mixed", "mbb", 1e-6, True),
        # the rest of that loop's iteration
        _other("design", "design_160x80x80", (160, 80, 80), radius=2.5),
        # the reference's own outer iteration on host arrays
        _other("stress", "stress_update_120x40x40", (120, 40, 40), radius=3.0),
        # fine-tuning the networks on the current design
        _other("train", "train_96x48x48", (96, 48, 48), batch=4),
    ]


def draw(rng):
    kind = rng.choice(["apply", "grid", "solve", "solve", "solve", "solve", "design", "stress",
                       "train"])

    def dims(lo, hi):  # element counts lo .. hi, spread over the logarithm; sides near 2:1:1
        ne = lo * (hi / lo) ** rng.random()
        a, b = rng.uniform(1.0, 3.0), rng.uniform(0.7, 1.4)
        ny = (ne / (a * b)) ** (1.0 / 3.0)
        return max(4, round(a * ny)), max(4, round(ny)), max(4, round(b * ny))

    if kind == "apply":
        return _other(kind, None, dims(600, 8e6), h=rng.choice([1.0, 0.5, 2.0]))
    if kind == "grid":
        return _other(kind, None, dims(3e3, 2e5))
    if kind == "design":
        return _other(kind, None, dims(2e4, 2e6), radius=rng.choice([1.5, 2.5, 3.0]))
    if kind == "stress":
        return _other(kind, None, dims(2e4, 4e5), radius=rng.choice([2.0, 3.0]))
    if kind == "train":
        return _other(kind, None, dims(2e4, 3e5), batch=rng.choice([1, 2, 4]))
    precond = rng.choice(["jacobi", "learned", "multigrid"])
    d = dims(1e4, 1.5e6)
    support, shift, warm = "cantilever", 0.0, False
    if precond == "multigrid":  # sides the hierarchy can halve a few times, or not
        m = rng.choice([16, 8, 2, 1])
        d = tuple(max(m, 4, m * round(x / m)) for x in d)
        if rng.random() < 0.4:
            support, shift, warm = "mbb", 1e-6, True
    return _solve(None, d, precond, rng.choice(["fp64", "mixed"]), support, shift, warm)


# --------------------------------------------------------------------------
# inputs, from the seed alone
# --------------------------------------------------------------------------
def _dims(case):
    return case["nx"], case["ny"], case["nz"]


def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _smooth(dims, seed):
    """i.i.d. uniform noise smoothed over about three elements, mapped to [0, 1]."""
    nx, ny, nz = dims
    t = torch.rand((1, 1, nz, ny, nx), generator=_gen(seed), dtype=torch.float64, device="cuda")
    for _ in range(2):
        t = torch.nn.functional.avg_pool3d(t, 5, 1, 2, count_include_pad=False)
    t = t.reshape(-1)
    return (t - t.min()) / (t.max() - t.min())


def _design(dims, seed):
    """A near-0/1 density as an optimisation leaves it."""
    t = _smooth(dims, seed)
    return 1e-3 + (1.0 - 1e-3) / (1.0 + torch.exp(-12.0 * (t - 0.5)))


def _simp(rho):
    return 1e-9 + rho ** 3 * (1.0 - 1e-9)


def _boundary(dims, support):
    """(bc nN x 3 Float32 column-major, f 3nN Float64) as the workloads have them: a cantilever
    clamped at x = 0 with a line load at x = nx, or the half MBB beam."""
    nx, ny, nz = dims
    n = (nx + 1) * (ny + 1) * (nz + 1)
    bc = np.zeros((n, 3), np.float32, order="F")
    b = [bc[:, c].reshape(nz + 1, ny + 1, nx + 1) for c in range(3)]
    f = np.zeros(3 * n)
    fy = f.reshape(nz + 1, ny + 1, nx + 1, 3)[..., 1]
    if support == "mbb":
        b[0][:, :, 0] = 1.0
        b[1][:, 0, nx] = 1.0
        fy[:, ny, 0] = -1.0 / (nz + 1)
    else:
        for c in b:
            c[:, :, 0] = 1.0
        fy[nz // 2, :, nx] = -1.0 / (ny + 1)
    return bc, f


def _beam(dims, seed):
    """A cantilever's bending displacement with a little noise (FP64, interleaved)."""
    nx, ny, nz = dims
    x = torch.arange(nx + 1, dtype=torch.float64, device="cuda") / nx
    y = torch.arange(ny + 1, dtype=torch.float64, device="cuda") / ny - 0.5
    u = torch.zeros((nz + 1, ny + 1, nx + 1, 3), dtype=torch.float64, device="cuda")
    u[..., 1] = -(x * x * (3.0 - x))
    u[..., 0] = (3.0 * x * (2.0 - x)) * (y * ny / nx)[:, None]
    u += 1e-3 * torch.randn(u.shape, generator=_gen(seed), dtype=torch.float64, device="cuda")
    u[:, :, 0] = 0.0
    return u.reshape(-1)


def _pinned(t):
    p = torch.empty(t.shape, dtype=torch.float32, pin_memory=True)
    p.copy_(t)
    return p


def _grid(case, h=1.0):
    ctx = hx.Context(0)
    ctx.set_grid(*_dims(case), h, h, h)
    ctx.set_material(1.0, NU)
    return ctx


def _solve_inputs(case, seed):
    """fac (Float32 device), shared by prepare and exact."""
    dims = _dims(case)
    if case["support"] == "mbb":
        return _simp(_design(dims, seed)).float()
    return _simp(1e-3 + (1.0 - 1e-3) * _smooth(dims, seed)).float()


def _grid_density(case, seed):
    """Float32 density with a share of voids below the pruning threshold."""
    return ((_smooth(_dims(case), seed) - 0.25) / 0.5).clamp(0.0, 1.0).float()


_STRESS_CONFIG = {
    "solver_parameters": {"filter_tolerance": 1e-5},
    "optimization_parameters": {"stress_regularization_ratio": 1.5, "filter_R_interm_iter_perc": 50.0,
                                "final_density_threshold": 0.95, "max_culling_ratio": 0.1},
}


def prepare(case, seed):
    kind, dims = case["kind"], _dims(case)
    nx, ny, nz = dims
    ne, n = nx * ny * nz, 3 * (nx + 1) * (ny + 1) * (nz + 1)
    s = {"case": case}
    if kind == "apply":
        s["x"] = torch.randn(n, generator=_gen(seed), dtype=torch.float64, device="cuda")
        s["fac"] = _simp(1e-3 + (1.0 - 1e-3) * torch.rand(
            ne, generator=_gen(seed + 1), dtype=torch.float64, device="cuda"))
        s["y"] = torch.empty_like(s["x"])
        s["xkx"] = torch.empty(1, dtype=torch.float64, device="cuda")
        s["lib"] = hx.load()
        return s
    if kind == "grid":
        bc, f = _boundary(dims, "cantilever")
        s.update(ctx=hx.Context(0), bc=bc, f=f.astype(np.float32),
                 density=_grid_density(case, seed).cpu().numpy())
        return s
    if kind == "stress":
        cfg = {k: dict(v) for k, v in _STRESS_CONFIG.items()}
        cfg["geometry"] = {"nElem_x_computed": nx, "nElem_y_computed": ny, "nElem_z_computed": nz,
                           "dx_computed": 1.0, "dy_computed": 1.0, "dz_computed": 1.0,
                           "max_domain_dim": float(nx)}
        perc = 100.0 * 2.5 * case["radius"] / nx
        cfg["optimization_parameters"].update(filter_R_init_perc=perc, filter_R_interm_perc=perc,
                                              filter_R_final_perc=perc)
        rho = _design(dims, seed).float().cpu().numpy()
        prot = np.zeros(ne, bool)
        prot.reshape(nz, ny, nx)[:, :, -2:] = True
        s.update(ctx=_grid(case), cfg=cfg, rho=rho, prot=prot,
                 u=_beam(dims, seed).float().cpu().numpy())
        return s
    ctx = s["ctx"] = _grid(case)
    support = case.get("support", "cantilever")
    bc, f = _boundary(dims, support)
    ctx.set_bc(bc)
    if kind == "solve":
        s["f"], s["fac"] = _pinned(torch.from_numpy(f)), _pinned(_solve_inputs(case, seed))
        s["u"] = torch.zeros(n, dtype=torch.float32, pin_memory=True)
        if case["warm"]:
            s["u0"] = _pinned(_warm_guess(case, seed))
        if case["precond"] == "learned":
            learned.load_into(ctx)
        s["opts"] = hx.default_opts(
            tol=1e-6, preconditioner=PRECOND[case["precond"]],
            precision=PRECISION[case["precision"]], shift_factor=case["shift"], max_iter=100000,
            warm_start=int(case["warm"]))
        return s
    if kind == "design":
        f64 = dict(dtype=torch.float64, device="cuda")
        s.update(x=_design(dims, seed), u=_beam(dims, seed + 1), f=torch.from_numpy(f).cuda())
        for k in ("rho", "fac", "dc", "dcf", "xn"):
            s[k] = torch.empty(ne, **f64)
        return s
    # train
    fac = _simp(1e-3 + (1.0 - 1e-3) * _smooth(dims, seed))
    free = _free(case, torch.ones_like(fac), bc)
    s["params"] = learned.load_params()
    s["fac"], s["r"], s["e"] = fac, [], []
    ke = _ke(1.0)
    for b in range(case["batch"]):
        e = (_beam(dims, seed + 10 + b) * free)
        s["e"].append(e)
        s["r"].append(_apply(ke, fac, e, dims) * free)
    ctx.net_set_params(s["params"])
    torch.cuda.synchronize()
    ctx.net_prepare(fac.data_ptr())
    return s


def _warm_guess(case, seed):
    """A displacement of the right size and shape to start from: the half beam's deflection."""
    nx, ny, nz = _dims(case)
    x = torch.arange(nx + 1, dtype=torch.float64) / nx
    y = torch.arange(ny + 1, dtype=torch.float64) / ny - 0.5
    c = 8.0 * nx ** 3 / (nz * ny ** 3)
    u = torch.zeros((nz + 1, ny + 1, nx + 1, 3), dtype=torch.float64)
    u[..., 1] = -c * (1.0 - 1.5 * x * x + 0.5 * x ** 3)
    u[..., 0] = -c * (3.0 * x - 1.5 * x * x) * (y * ny / nx)[:, None]
    return u.reshape(-1)


# --------------------------------------------------------------------------
# one pass
# --------------------------------------------------------------------------
def _ptr(t):
    return ctypes.c_void_p(t.data_ptr())


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "apply":
        h = case["h"]
        st = s["lib"].hx_apply_stiffness_noalloc(
            *_dims(case), h, h, h, NU, _ptr(s["x"]), _ptr(s["fac"]), _ptr(s["y"]), _ptr(s["xkx"]),
            ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
        if st != 0:
            raise RuntimeError(f"hx_apply_stiffness_noalloc: status {st}")
        return {"y": s["y"], "xkx": s["xkx"]}
    ctx = s["ctx"]
    if kind == "grid":
        x, _, _ = api.solve_system_grid(_dims(case), (1.0, 1.0, 1.0), 1.0, NU, s["bc"], s["f"],
                                        s["density"], ctx=ctx)
        return x
    if kind == "solve":
        if case["warm"]:
            s["u"].copy_(s["u0"])
        rep = _lib.SolveReport()
        st = ctx.lib.hx_solve(ctx.h, _lib.HX_F32, _ptr(s["f"]), _ptr(s["fac"]), _ptr(s["u"]),
                              ctypes.byref(s["opts"]), ctypes.byref(rep))
        ctx.check(st, "hx_solve")
        return s["u"]
    if kind == "design":
        d = {k: s[k].data_ptr() for k in ("x", "u", "f", "rho", "fac", "dc", "dcf", "xn")}
        ctx.filter_device(d["x"], d["rho"], case["radius"])
        ctx.simp_device(d["rho"], d["fac"])
        c = ctx.compliance_device(d["f"], d["u"])
        ctx.sensitivity_device(d["rho"], d["u"], d["dc"])
        ctx.filter_device(d["dc"], d["dcf"], case["radius"])
        ctx.oc_update_device(d["x"], d["dcf"], d["xn"], 0.4, 0.2)
        return {"rho": s["rho"], "fac": s["fac"], "dc": s["dc"], "dcf": s["dcf"], "xn": s["xn"],
                "c": c}
    if kind == "stress":
        pr, vm, vo, l1, dr = ctx.stress(s["u"], s["rho"], 1.0, NU)
        dens, l1n = s["rho"].copy(), l1.copy()
        api.update_density(dens, l1n, s["prot"], 1.0, 0.05, 20, 100, s["rho"], 1e-3, 1.0, s["cfg"],
                           ctx=ctx)
        return {"principal": pr, "von_mises": vm, "voigt": vo, "l1": l1, "dir": dr,
                "density": dens, "l1_filtered": l1n}
    ctx.net_set_params(s["params"])
    loss = ctx.net_train_batch([r.data_ptr() for r in s["r"]], [e.data_ptr() for e in s["e"]], 1e-4)
    return {"params": ctx.net_get_params(), "loss": loss}


# --------------------------------------------------------------------------
# what a pass cannot do without: inputs read once, outputs written once
# --------------------------------------------------------------------------
def work(case):
    kind = case["kind"]
    nx, ny, nz = _dims(case)
    ne, n = nx * ny * nz, 3 * (nx + 1) * (ny + 1) * (nz + 1)
    op = 280.0 * ne  # one operator product: about 140 multiply-adds per element
    if kind == "apply":
        return {"bytes": 16.0 * n + 8.0 * ne, "flops": op}
    if kind == "grid":
        return {"bytes": 12.0 * n + 4.0 * ne, "flops": op}
    if kind == "solve":
        return {"bytes": (12.0 if case["warm"] else 8.0) * n + 4.0 * ne, "flops": op}
    if kind == "design":
        return {"bytes": 16.0 * n + 48.0 * ne, "flops": op}
    if kind == "stress":
        return {"bytes": 4.0 * n + 4.0 * 14 * ne + 17.0 * ne, "flops": 300.0 * ne}
    return {"bytes": case["batch"] * 16.0 * n + 8.0 * ne + 8.0 * hx.Context.NET_PARAMS,
            "flops": case["batch"] * 24 * 2 * 27 * 256 * (ne / 64.0)}


# --------------------------------------------------------------------------
# 64-bit results with plain torch
# --------------------------------------------------------------------------
def _ke(h):
    """24 x 24 stiffness of a cube element of unit modulus by 2 x 2 x 2 Gauss points; corner
    b = bx + 2 by + 4 bz, DOF 3 b + c."""
    c1, c2, c3 = 1.0 - NU, NU, (1.0 - 2.0 * NU) / 2.0
    D = np.zeros((6, 6))
    D[:3, :3] = c2
    D[[0, 1, 2], [0, 1, 2]] = c1
    D[[3, 4, 5], [3, 4, 5]] = c3
    D /= (1.0 + NU) * (1.0 - 2.0 * NU)
    s = np.array([[2 * (b & 1) - 1, 2 * ((b >> 1) & 1) - 1, 2 * (b >> 2) - 1] for b in range(8)])
    K = np.zeros((24, 24))
    p = 1.0 / np.sqrt(3.0)
    for gx in (-p, p):
        for gy in (-p, p):
            for gz in (-p, p):
                t = 1.0 + s * np.array([gx, gy, gz])
                d = s * np.stack([t[:, 1] * t[:, 2], t[:, 0] * t[:, 2], t[:, 0] * t[:, 1]], 1)
                d = d / 8.0 * (2.0 / h)
                B = np.zeros((6, 24))
                B[0, 0::3], B[1, 1::3], B[2, 2::3] = d[:, 0], d[:, 1], d[:, 2]
                B[3, 0::3], B[3, 1::3] = d[:, 1], d[:, 0]
                B[4, 1::3], B[4, 2::3] = d[:, 2], d[:, 1]
                B[5, 0::3], B[5, 2::3] = d[:, 2], d[:, 0]
                K += B.T @ D @ B * (h / 2.0) ** 3
    return torch.from_numpy(K).cuda()


def _corner(b, dims):
    nx, ny, nz = dims
    x, y, z = b & 1, (b >> 1) & 1, b >> 2
    return slice(z, z + nz), slice(y, y + ny), slice(x, x + nx)


def _apply(ke, fac, u, dims):
    nx, ny, nz = dims
    u = u.view(nz + 1, ny + 1, nx + 1, 3)
    v = torch.cat([u[_corner(b, dims)] for b in range(8)], -1) @ ke
    v *= fac.view(nz, ny, nx, 1)
    y = torch.zeros_like(u)
    for b in range(8):
        y[_corner(b, dims)] += v[..., 3 * b:3 * b + 3]
    return y.reshape(-1)


def _node_sum(fac, dims):
    nx, ny, nz = dims
    s = torch.zeros((nz + 1, ny + 1, nx + 1), dtype=torch.float64, device="cuda")
    for b in range(8):
        s[_corner(b, dims)] += fac.view(nz, ny, nx)
    return s.reshape(-1)


def _free(case, fac, bc):
    """1 on the DOFs that are solved for: free ones with stiffness."""
    fixed = torch.from_numpy(np.ascontiguousarray(bc)).cuda() > 0
    return (~fixed & (_node_sum(fac, _dims(case)) > 0)[:, None]).double().reshape(-1)


def _cg(case, fac, bc, f, shift_factor):
    """Jacobi-preconditioned conjugate gradients to 1e-10; None after 12000 steps."""
    dims, ke = _dims(case), _ke(1.0)
    free = _free(case, fac, bc)
    diag = (_node_sum(fac, dims)[:, None] * torch.diagonal(ke)[:3]).reshape(-1)
    shift = shift_factor * float((diag * free).max())
    m = torch.where(free > 0, 1.0 / (diag + shift).clamp_min(1e-300), 0.0)
    r = torch.from_numpy(np.asarray(f, np.float64)).cuda() * free
    x, bn = torch.zeros_like(r), float(r.norm())
    z = m * r
    p, rz = z.clone(), torch.dot(r, z)
    for it in range(12000):
        q = (_apply(ke, fac, p, dims) + shift * p) * free
        a = rz / torch.dot(p, q)
        x += a * p
        r -= a * q
        if it % 50 == 49 and float(r.norm()) < 1e-10 * bn:
            return x
        z = m * r
        new = torch.dot(r, z)
        p = z + (new / rz) * p
        rz = new
    return None


def exact(case, seed):
    kind, dims = case["kind"], _dims(case)
    nx, ny, nz = dims
    if kind == "apply":
        s = prepare(case, seed)
        y = _apply(_ke(case["h"]), s["fac"], s["x"], dims)
        return {"y": y, "xkx": torch.dot(s["x"], y).reshape(1)}
    if kind in ("grid", "solve") and nx * ny * nz <= 2_000_000:
        bc, f = _boundary(dims, case.get("support", "cantilever"))
        f = f.astype(np.float32)
        if kind == "grid":
            d = _grid_density(case, seed)
            return _cg(case, torch.where(d >= 1e-3, d, 0.0).double(), bc, f, 1e-6)
        return _cg(case, _solve_inputs(case, seed).double(), bc, f, case["shift"])
    return None
