"""The work a user of this framework has it do, as cases that can be timed and
checked: loop steps of a tissue at the sizes of the benchmark configurations
and around them, batches of tissues, gradients through the loop, the
cell-model and linear-solver plugin calls of a host program, and steps through
host buffers.

``exact`` restates the same mathematics in plain torch FP64 (cell models,
diffusion operator, a conjugate-gradient solve run to rounding), with
gradients by torch autograd.
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

S_PER_M = 1e-3      # S/m -> mS/um
DX = 100.0          # um
DT = 0.02           # ms


# ---- the cases -----------------------------------------------------------------

def listed():
    return [
        # One cable, the smallest tissue in use (single-fibre propagation, unit
        # tests, parameter fits): a few blocks per kernel, so launches, grid
        # reductions and latency are all there is.  FP64, one dump interval.
        dict(name="cable_400_tt2006_fp64", kind="tissue", model="tt2006", precision="fp64", form="iso",
             nx=400, ny=1, nz=1, steps=50),
        # The plain-method configuration: 1.0 x 1.0 x 0.2 cm cuboid, FP64.
        dict(name="cuboid_200k_tt2006_fp64", kind="tissue", model="tt2006", precision="fp64", form="iso",
             nx=100, ny=100, nz=20, steps=10),
        # The precision configuration: 2 x 2 x 0.5 cm slab with 20 % diffuse
        # fibrosis (removed cells), fibres along x, mixed precision.
        dict(name="slab_2m_fibrosis_torord_mixed", kind="tissue", model="torord", precision="mixed", form="fibrosis",
             nx=200, ny=200, nz=50, steps=5),
        # The batching configuration: 128 cables and 128 sheets in one atlas,
        # conductance scalings per tissue, activation tracking, mixed precision.
        dict(name="batch_256_tt2006_mixed", kind="batch", precision="mixed", cables=128, sheets=128,
             cable_lo=100, cable_hi=400, sheet_lo=64, sheet_hi=256, steps=5),
        # The scale configuration, the largest run: 5 x 5 x 1 cm slab,
        # transmural cell types, rotating fibres (27-point rows), mixed precision.
        dict(name="slab_25m_rotating_torord_mixed", kind="tissue", model="torord", precision="mixed", form="rotating",
             nx=500, ny=500, nz=100, steps=2),
        # The same physics in FP64 (the reference precision) on a slab whose
        # sides are no multiple of any tile.
        dict(name="slab_3m_rotating_torord_fp64", kind="tissue", model="torord", precision="fp64", form="rotating",
             nx=254, ny=187, nz=61, steps=2),
        # The differentiation configuration's sheet: traces at 64 sensors and
        # the gradient with respect to conductivity and gKr, FP64.
        dict(name="gradient_256_tt2006_fp64", kind="gradient", precision="fp64", nx=256, ny=256, sensors=64,
             nsteps=100, sample_every=10, checkpoint_every=50),
        # The same with the mixed forward, on a smaller sheet of odd sides.
        dict(name="gradient_97x131_tt2006_mixed", kind="gradient", precision="mixed", nx=97, ny=131, sensors=32,
             nsteps=100, sample_every=10, checkpoint_every=50),
        # A population of uncoupled cells (cell-model studies): 2 ms of the
        # ToRORd model per call, the whole state read back.
        dict(name="population_20k_torord_mixed", kind="population", model="torord", precision="mixed", cells=20000,
             substeps=100),
        # The cell-model plugin call of a host program that owns the loop:
        # stimulus from host memory every step, FP64 state kept on the device.
        dict(name="plugin_200k_torord_fp64", kind="plugin", model="torord", precision="fp64", cells=200000),
        # A step through host buffers (stimulus in, V out, pinned memory), the
        # reference-host mode, on a slab of odd sides.
        dict(name="host_step_1m_tt2006_mixed", kind="host", model="tt2006", precision="mixed", form="iso",
             nx=173, ny=211, nz=37),
        # The linear-solver plugin call: a general CSR matrix kept on the
        # device, right-hand side and solution in host memory.
        dict(name="csr_200k_fp64", kind="csr", nx=100, ny=100, nz=20),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["tissue", "tissue", "tissue", "tissue", "tissue", "batch", "gradient", "population", "plugin",
                       "host", "csr"])
    precision = rng.choice(["fp64", "mixed"])
    model = rng.choice(["tt2006", "torord"])
    if kind in ("tissue", "host"):
        form = rng.choice(["iso", "fibrosis", "rotating"])
        shape = rng.choice(["cable", "sheet", "slab", "slab"])
        most = 4_000_000 if kind == "tissue" else 1_500_000
        if shape == "cable" and form != "rotating":
            nx, ny, nz = _log(rng, 100, 4000), 1, 1
        elif shape == "sheet" and form != "rotating":
            nx, ny, nz = _log(rng, 32, 1200), _log(rng, 32, 1200), 1
        else:
            nz = _log(rng, 8, 100)
            nx = _log(rng, 40, 400)
            ny = max(17, min(_log(rng, 40, 400), most // (nx * nz)))
        case = dict(kind=kind, model=model, precision=precision, form=form, nx=nx, ny=ny, nz=nz)
        if kind == "tissue":
            case["steps"] = rng.randint(1, 4) if nx * ny * nz > 500_000 else rng.randint(4, 40)
        return case
    if kind == "batch":
        lo = rng.randint(20, 90)
        return dict(kind=kind, precision=precision, cables=rng.randint(1, 128), sheets=rng.randint(1, 64),
                    cable_lo=100, cable_hi=400, sheet_lo=lo, sheet_hi=lo + rng.randint(10, 150),
                    steps=rng.randint(2, 8))
    if kind == "gradient":
        every = rng.choice([5, 10, 20])
        return dict(kind=kind, precision=precision, nx=_log(rng, 24, 256), ny=_log(rng, 24, 256),
                    sensors=rng.randint(4, 64), nsteps=every * rng.randint(2, 5), sample_every=every,
                    checkpoint_every=rng.choice([20, 30, 50]))
    if kind == "population":
        return dict(kind=kind, model=model, precision=precision, cells=_log(rng, 64, 40000),
                    substeps=rng.choice([25, 50, 100]))
    if kind == "plugin":
        return dict(kind=kind, model=model, precision="fp64", cells=_log(rng, 500, 800_000))
    return dict(kind="csr", nx=_log(rng, 20, 130), ny=_log(rng, 20, 130), nz=_log(rng, 1, 20))


# ---- inputs, from the seed alone --------------------------------------------------

def _rng(seed):
    return np.random.Generator(np.random.Philox(int(seed)))


def _blobs(r, nx, ny, nz, share=0.06):
    """Stimulus boxes covering about `share` of the grid (a paced tissue has
    several activated regions, each with its own border)."""
    m = np.zeros((nz, ny, nx), dtype=np.uint8)
    for _ in range(4):
        s = [max(1, int(round(n * (share / 4) ** (1.0 / max(1, sum(k > 1 for k in (nx, ny, nz))))
                              * r.uniform(0.8, 1.25)))) if n > 1 else 1 for n in (nx, ny, nz)]
        o = [int(r.integers(0, n - w + 1)) for n, w in zip((nx, ny, nz), s)]
        m[o[2]:o[2] + s[2], o[1]:o[1] + s[1], o[0]:o[0] + s[0]] = 1
    return m.reshape(-1)


def _tissue_inputs(case, seed):
    """Keywords of the tissue: two stimulus regions (the configurations' planar
    one and boxes), removed cells, fibre angles, cell types."""
    r = _rng(seed)
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    n = nx * ny * nz
    kw = dict(model=case["model"], precision=case["precision"])
    active = None
    if case["form"] == "fibrosis":
        active = (r.random(n) >= 0.2).astype(np.uint8)
        kw.update(assembly="anisotropic", sigma_l=0.2 * S_PER_M, sigma_t=0.05 * S_PER_M, sigma_n=0.05 * S_PER_M,
                  active=active)
    elif case["form"] == "rotating":
        z = (np.arange(nz) + 0.5) / nz
        kw.update(assembly="anisotropic", sigma_l=0.2 * S_PER_M, sigma_t=0.04 * S_PER_M, sigma_n=0.04 * S_PER_M,
                  fibre_angle_z=np.deg2rad(60.0 - 120.0 * z + r.uniform(-10.0, 10.0)))
    else:
        kw.update(assembly="homogeneous", sigma=(float(r.uniform(0.1, 0.16)) * S_PER_M,) * 3)
    if case["model"] == "torord" and nz >= 3:
        third = np.minimum(2, (3 * np.arange(nz)) // nz).astype(np.uint8)
        kw["celltype"] = np.broadcast_to(third[:, None, None], (nz, ny, nx)).reshape(-1).copy()
    kw["x_limit"] = float(r.uniform(450.0, 650.0))
    kw["current"] = float(r.uniform(-56.0, -50.0))
    kw["mask"] = _blobs(r, nx, ny, nz)
    return kw


def _stims(kw):
    from monoalg3d_c_b200 import Stim
    return [Stim(kind="x_less_than", start=0.0, duration=2.0, current=kw.pop("current"), x_limit=kw.pop("x_limit")),
            Stim(kind="cell_mask", start=0.0, duration=1.0, current=-53.0, cell_mask=kw.pop("mask"))]


def _batch_inputs(case, seed):
    # the tissues belong to the study; the parameters are drawn
    q, r = _rng(2002), _rng(seed)
    sizes = [(int(c), 1) for c in q.integers(case["cable_lo"], case["cable_hi"] + 1, case["cables"])]
    sizes += [(int(s), int(s)) for s in q.integers(case["sheet_lo"], case["sheet_hi"] + 1, case["sheets"])]
    return sizes, np.exp(0.2 * r.standard_normal((len(sizes), 5))), float(r.uniform(-56.0, -50.0))


def _gradient_inputs(case, seed):
    r = _rng(seed)
    nx, ny = case["nx"], case["ny"]
    n = nx * ny
    w = r.standard_normal((ny, nx))
    kx, ky = np.fft.fftfreq(nx)[None, :], np.fft.fftfreq(ny)[:, None]
    f = np.real(np.fft.ifft2(np.fft.fft2(w) * np.exp(-np.pi ** 2 * 100.0 * (kx ** 2 + ky ** 2))))
    sigma = 0.13 * S_PER_M * np.exp(0.3 * (f / f.std()).reshape(-1))
    gkr = np.exp(0.1 * r.standard_normal(n))
    # sensors and paced spots belong to the study, conductivity and data are drawn
    q = _rng(3004)
    sensors = q.choice(n, size=case["sensors"], replace=False).astype(np.int64)
    mask = np.zeros((ny, nx), dtype=np.uint8)
    for s in sensors[::2]:
        j, i = divmod(int(s), nx)
        mask[max(0, j - 3):j + 2, max(0, i - 4):i + 1] = 1
    samples = case["nsteps"] // case["sample_every"]
    data = -80.0 + 5.0 * r.standard_normal((samples, case["sensors"]))
    return sigma, gkr, sensors, mask.reshape(-1), data


def _cells_inputs(case, seed):
    """Cell types, a spread of initial states and the stimulus of each cell."""
    r = _rng(seed)
    n = case["cells"]
    tor = case["model"] == "torord"
    ct = r.integers(0, 3, n).astype(np.uint8) if tor else None
    base = np.array(TORORD_STATE)[ct].T if tor else np.tile(np.array(TT2006_STATE)[:, None], (1, n))
    state = base * (1.0 + 0.005 * r.standard_normal(base.shape))
    state[0] = base[0] + r.uniform(0.0, 6.0, n)
    if tor:
        state[10:33] = np.clip(state[10:33], 0.0, 1.0)
    else:
        state[1:13] = np.clip(state[1:13], 0.0, 1.0)
    stim = np.where(r.random(n) < 0.5, r.uniform(-53.0, -20.0, n), 0.0)
    return ct, np.ascontiguousarray(state), stim


def _csr_inputs(case, seed):
    """The 7-point operator of a cuboid with varying conductivity as a general
    CSR matrix, b = alpha V of a tissue with fronts, x0 = V a step earlier."""
    r = _rng(seed)
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    n = nx * ny * nz
    sig = 0.13 * S_PER_M * np.exp(0.2 * r.standard_normal((nz, ny, nx)))
    idx = np.arange(n, dtype=np.int64).reshape(nz, ny, nx)
    alpha = 0.14 / DT * 1e-8 * DX ** 3
    rows, cols, vals = [], [], []
    diag = np.full(n, alpha)
    for ax in range(3):
        lo = [slice(None)] * 3
        hi = [slice(None)] * 3
        lo[ax], hi[ax] = slice(0, -1), slice(1, None)
        a, b = idx[tuple(lo)].reshape(-1), idx[tuple(hi)].reshape(-1)
        sa, sb = sig[tuple(lo)].reshape(-1), sig[tuple(hi)].reshape(-1)
        c = 2.0 * sa * sb / (sa + sb) * DX
        np.add.at(diag, a, c)
        np.add.at(diag, b, c)
        rows += [a, b]
        cols += [b, a]
        vals += [-c, -c]
    rows = np.concatenate(rows + [np.arange(n)])
    cols = np.concatenate(cols + [np.arange(n)])
    vals = np.concatenate(vals + [diag])
    o = np.lexsort((cols, rows))
    rows, cols, vals = rows[o], cols[o], vals[o]
    ptr = np.zeros(n + 1, dtype=np.int32)
    np.cumsum(np.bincount(rows, minlength=n), out=ptr[1:])
    v = -85.0 + 110.0 * _blobs(r, nx, ny, nz, 0.3).astype(np.float64) + 0.5 * r.standard_normal(n)
    return ptr, cols.astype(np.int32), vals, alpha * v, v + 0.3 * r.standard_normal(n)


# ---- what a program holds, and one pass ------------------------------------------

class _DeviceArray:
    def __init__(self, ptr, shape, strides, owner):
        self.__cuda_array_interface__ = {"shape": shape, "strides": strides, "typestr": "<f8", "data": (ptr, False),
                                         "version": 3}
        self.owner = owner


def _device_tensor(ptr, shape, strides, owner):
    return torch.as_tensor(_DeviceArray(ptr, shape, strides, owner), device="cuda")


def prepare(case, seed):
    import monoalg3d_c_b200 as mb
    from monoalg3d_c_b200._lib import check
    from monoalg3d_c_b200.batch import Batch
    kind = case["kind"]
    if kind in ("tissue", "host"):
        kw = _tissue_inputs(case, seed)
        n = case["nx"] * case["ny"] * case["nz"]
        if kind == "host":
            mask = kw.pop("mask")
            kw.pop("x_limit")
            cur = kw.pop("current")
            a = kw.get("active")
            on = mask if a is None else mask[a != 0]
            t = mb.Tissue(case["nx"], case["ny"], case["nz"], **kw)
            stim = torch.zeros(on.size, dtype=torch.float64).pin_memory()
            stim.numpy()[:] = cur * on
            quiet = torch.zeros(on.size, dtype=torch.float64).pin_memory()
            v = torch.zeros(n, dtype=torch.float64).pin_memory()
            return dict(case=case, t=t, stim=stim.numpy(), quiet=quiet.numpy(), v=v.numpy(), done=0,
                        keep=(stim, quiet, v))
        t = mb.Tissue(case["nx"], case["ny"], case["nz"], stims=_stims(kw), **kw)
        return dict(case=case, t=t, v=_device_tensor(t.device_v()[0], (n,), None, t))
    if kind == "batch":
        sizes, scales, cur = _batch_inputs(case, seed)
        b = Batch(sizes, scales, mb.Stim(kind="x_less_than", start=0.0, duration=2.0, current=cur, x_limit=100.0),
                  model="tt2006", precision=case["precision"], assembly="homogeneous",
                  sigma=(0.13 * S_PER_M,) * 3, track_activation=True)
        return dict(case=case, t=b, v=_device_tensor(b.tissue.device_v()[0], (b.atlas[0] * b.atlas[1],), None, b))
    if kind == "gradient":
        from monoalg3d_c_b200.adjoint import Adjoint
        sigma, gkr, sensors, mask, data = _gradient_inputs(case, seed)
        adj = Adjoint(case["nx"], case["ny"], 1, sigma, gkr, sensors, case["nsteps"], case["sample_every"],
                      case["checkpoint_every"], precision=case["precision"],
                      stims=[mb.Stim(kind="cell_mask", start=0.0, duration=2.0, current=-53.0, cell_mask=mask)])
        return dict(case=case, adj=adj, sigma=torch.tensor(sigma, device="cuda", requires_grad=True),
                    gkr=torch.tensor(gkr, device="cuda", requires_grad=True), data=torch.tensor(data, device="cuda"))
    if kind in ("population", "plugin"):
        ct, state, stim = _cells_inputs(case, seed)
        o = mb.OdeSolver(case["model"], case["cells"], DT, case.get("substeps", 1), precision=case["precision"])
        o.set_model_initial_conditions_gpu(celltype=ct)
        o.set_state(state)
        s = dict(case=case, o=o, stim=stim, quiet=np.zeros_like(stim), time=0.0)
        if kind == "plugin":
            sv, pitch = C.c_void_p(), C.c_size_t()
            check(mb.lib.mb_ode_device_state(o._h, C.byref(sv), C.byref(pitch)))
            s["sv"] = _device_tensor(sv.value, (o.neq, case["cells"]), (pitch.value, 8), o)
        return s
    ptr, col, val, b, x0 = _csr_inputs(case, seed)
    h = C.c_void_p()
    check(mb.lib.mb_csr_create(C.byref(h), b.size, ptr.ctypes.data, col.ctypes.data, val.ctypes.data))
    return dict(case=case, h=_Csr(h, mb.lib), b=b, x0=x0)


class _Csr:
    def __init__(self, h, lib):
        self.h, self.lib = h, lib

    def __del__(self):
        self.lib.mb_csr_destroy(self.h)


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind in ("tissue", "batch"):
        s["t"].step(case["steps"])
        return s["v"]
    if kind == "host":
        # stimulus during the first 2 ms of a 1000 ms cycle
        s["t"].step_host(s["stim"] if s["done"] % 50000 < 100 else s["quiet"], s["v"])
        s["done"] += 1
        return s["v"]
    if kind == "gradient":
        from monoalg3d_c_b200 import adjoint
        s["sigma"].grad = s["gkr"].grad = None
        tr = adjoint.traces(s["sigma"], s["gkr"], s["adj"])
        loss = 0.5 * ((tr - s["data"]) ** 2).sum()
        loss.backward()
        return {"traces": tr.detach(), "grad_sigma": s["sigma"].grad, "grad_gkr": s["gkr"].grad}
    if kind in ("population", "plugin"):
        on = s["time"] % 1000.0 < 1.99
        s["o"].solve_model_odes_gpu(s["time"], s["stim"] if on else s["quiet"])
        s["time"] += DT * case.get("substeps", 1)
        return s["sv"] if kind == "plugin" else s["o"].state()
    from monoalg3d_c_b200._lib import check, lib
    x = s["x0"].copy()
    its, err = C.c_uint32(), C.c_double()
    check(lib.mb_csr_solve(s["h"].h, s["b"].ctypes.data, x.ctypes.data, 1e-16, 200, 1, C.byref(its), C.byref(err)))
    return x


# ---- cost and tolerance --------------------------------------------------------------

def _state_bytes(model, precision):
    """State of a cell, read and written once, and V in and V* out."""
    if model == "tt2006":
        return 2 * (18 * 8 if precision == "fp64" else 5 * 8 + 13 * 4) + 16
    return 2 * (42 * 8 if precision == "fp64" else 8 * 8 + 34 * 4) + 16


# operations of one cell step (adds, multiplies, divisions, and 10 for an exponential)
_OPS = {"tt2006": 1200, "torord": 2200}


def _step_cost(cells, model, precision, its=15, points=7):
    """One loop step: the cell model's rows once, and a conjugate-gradient
    solve of `its` iterations that reads and writes x, r and p once each (FP64
    x, FP32 r and p in the mixed form, with two FP64 residuals)."""
    cg = 8 * (6 * its + 3) if precision == "fp64" else 32 * its + 24 * 2
    return cells * (_state_bytes(model, precision) + cg), cells * (_OPS[model] + its * (2 * points + 12))


def work(case):
    kind = case["kind"]
    if kind in ("tissue", "host"):
        n = case["nx"] * case["ny"] * case["nz"]
        cells = n * (0.8 if case["form"] == "fibrosis" else 1.0)
        b, f = _step_cost(cells, case["model"], case["precision"], points=19 if case["form"] == "rotating" else 7)
        if kind == "host":
            return {"bytes": b + 16 * n, "flops": f}
        return {"bytes": case["steps"] * b, "flops": case["steps"] * f}
    if kind == "batch":
        sizes, _, _ = _batch_inputs(case, 0)
        cells = sum(a * b for a, b in sizes)
        b, f = _step_cost(cells, "tt2006", case["precision"], points=5)
        return {"bytes": case["steps"] * (b + cells * 32), "flops": case["steps"] * f}
    if kind == "gradient":
        cells = case["nx"] * case["ny"]
        b, f = _step_cost(cells, "tt2006", case["precision"], points=5)
        # forward, recomputation, and a backward step of about twice a step's work
        return {"bytes": case["nsteps"] * 4 * b, "flops": case["nsteps"] * 4 * f}
    if kind in ("population", "plugin"):
        steps = case.get("substeps", 1)
        neq = 19 if case["model"] == "tt2006" else 43
        b = _state_bytes(case["model"], case["precision"]) + 8 + (neq * 8 if kind == "population" else 0)
        return {"bytes": case["cells"] * b, "flops": case["cells"] * steps * _OPS[case["model"]]}
    n = case["nx"] * case["ny"] * case["nz"]
    nnz = 7 * n
    return {"bytes": 15 * (12 * nnz + 4 * n + 8 * 6 * n) + 24 * n, "flops": 15 * (2 * nnz + 12 * n)}


def tolerance(case):
    """About four times what the same path shows against ``exact`` or, where
    that is more, what its stopping rule allows (r.r <= 1e-16: the last
    iteration may fall on either side)."""
    kind = case["kind"]
    if kind == "csr":
        return {"rel": 1e-10, "max": 1e-8}
    fp64 = case["precision"] == "fp64"
    if kind == "gradient":
        return {"rel": 2e-8, "max": 2e-6} if fp64 else {"rel": 5e-5, "max": 2e-2}
    if kind in ("population", "plugin"):
        return {"rel": 1e-12, "max": 1e-9} if fp64 else {"rel": 2e-7, "max": 1e-4}
    return {"rel": 1e-8, "max": 1e-6} if fp64 else {"rel": 2e-7, "max": 2e-5}


# ---- the same in plain torch, 64 bits ---------------------------------------------------

def _f(x):
    """A literal that the model library holds as a float."""
    return float(np.float32(x))


TT2006_STATE = [_f(x) for x in (-85.23, 0.00621, 0.4712, 0.0095, 0.00172, 0.7444, 0.7045, 3.373e-5, 0.7888, 0.9755,
                                0.9953, 0.999998, 2.42e-8, 0.000126, 3.64, 0.00036, 0.9073, 8.604, 136.89)]

# steady states of the endo, mid and epi cells
TORORD_STATE = [
    [-8.890585e+01, 1.107642e-02, 6.504164e-05, 1.210818e+01, 1.210851e+01, 1.426206e+02, 1.426205e+02, 1.530373e+00,
     1.528032e+00, 7.455488e-05, 7.814592e-04, 8.313839e-01, 8.311938e-01, 6.752873e-01, 8.308255e-01, 1.585610e-04,
     5.294475e-01, 2.896996e-01, 9.419166e-04, 9.996194e-01, 5.938602e-01, 4.799180e-04, 9.996194e-01, 6.543754e-01,
     -2.898677e-33, 1.000000e+00, 9.389659e-01, 1.000000e+00, 9.999003e-01, 9.999773e-01, 1.000000e+00, 1.000000e+00,
     4.920606e-04, 8.337021e-04, 6.962775e-04, 8.425453e-04, 9.980807e-01, 1.289824e-05, 3.675442e-04, 2.471690e-01,
     1.742987e-04, 5.421027e-24, 6.407933e-23],
    [-8.924177e+01, 1.922391e-02, 6.585066e-05, 1.503347e+01, 1.503401e+01, 1.434407e+02, 1.434406e+02, 1.959747e+00,
     1.963459e+00, 8.177438e-05, 7.269124e-04, 8.379059e-01, 8.377164e-01, 6.860578e-01, 8.372100e-01, 1.487602e-04,
     5.350003e-01, 2.851164e-01, 9.208259e-04, 9.996411e-01, 5.673539e-01, 4.691672e-04, 9.996412e-01, 6.265825e-01,
     -4.922960e-40, 1.000000e+00, 9.200354e-01, 1.000000e+00, 9.997888e-01, 9.999665e-01, 1.000000e+00, 1.000000e+00,
     5.161178e-04, 1.189422e-03, 6.917041e-04, 8.225453e-04, 9.979358e-01, 1.835276e-05, 5.316232e-04, 2.650323e-01,
     1.678628e-04, 2.091039e-25, 2.438403e-23],
    [-8.917755e+01, 1.288116e-02, 5.767956e-05, 1.284260e+01, 1.284291e+01, 1.429114e+02, 1.429113e+02, 1.812268e+00,
     1.810520e+00, 6.631866e-05, 7.370422e-04, 8.366816e-01, 8.366012e-01, 6.840260e-01, 8.363958e-01, 1.505860e-04,
     5.412669e-01, 3.043382e-01, 9.248184e-04, 9.996371e-01, 9.996342e-01, 4.712023e-04, 9.996371e-01, 9.996366e-01,
     4.333129e-43, 1.000000e+00, 9.485160e-01, 1.000000e+00, 9.999339e-01, 9.999822e-01, 1.000000e+00, 1.000000e+00,
     3.086885e-04, 5.303737e-04, 6.775197e-04, 8.264829e-04, 9.982135e-01, 9.433146e-06, 2.730221e-04, 2.308784e-01,
     1.690386e-04, -1.103286e-23, -6.177055e-22]]


def _tt2006_step(y, stim, dt, scale=(1.0, 1.0, 1.0, 1.0, 1.0)):
    """One Rush-Larsen step of ten Tusscher & Panfilov 2006 (epicardial);
    scale: gNa, gKr, gKs, gCaL, gK1."""
    e, w = torch.exp, torch.where
    V, xr1, xr2, xs, m, h, j, d, f, f2, fc, s, r, cai, casr, cass, rp, nai, ki = y
    F, R, T = _f(96485.3415), 8314.472, 310.0
    RT, RTF = R * T, R * T / F
    EK = RTF * torch.log(5.4 / ki)
    EKs = RTF * torch.log((5.4 + 0.03 * 140.0) / (ki + 0.03 * nai))
    ENa = RTF * torch.log(140.0 / nai)
    ECa = 0.5 * RTF * torch.log(2.0 / cai)
    vk = V - EK
    bk = (3.0 * e(_f(0.0002) * (vk + 100.0)) + e(_f(0.1) * (vk - 10.0))) / (1.0 + e(-0.5 * vk))
    ak = _f(0.1) / (1.0 + e(_f(0.06) * (vk - 200.0)))
    IK1 = 5.405 * scale[4] * ak / (ak + bk) * vk
    Ito = 0.294 * r * s * vk
    IKr = 0.153 * scale[1] * xr1 * xr2 * vk * math.sqrt(5.4 / _f(5.4))
    IKs = 0.098 * scale[2] * xs * xs * (V - EKs)
    IpK = 0.0146 * vk / (1.0 + e((25.0 - V) / _f(5.98)))
    v15 = V - 15.0
    near = v15.abs() < 1e-5
    v15 = w(near, torch.full_like(v15, 1.0), v15)
    ea = 2.0 * v15 * F / RT
    ICaL = 3.98e-05 * scale[3] * d * f * f2 * fc * 4.0 * v15 * F * F / RT * (0.25 * cass * e(ea) - 2.0) / torch.expm1(ea)
    ICaL = w(near, 3.98e-05 * scale[3] * d * f * f2 * fc * 2.0 * F * (0.25 * cass - 2.0), ICaL)
    IbCa = 0.000592 * (V - ECa)
    IpCa = 0.1238 * cai / (cai + 0.0005)
    INaK = 2.724 * 5.4 / (5.4 + 1.0) * nai / (nai + 40.0) / (
        1.0 + _f(0.1245) * e(_f(-0.1) * V * F / RT) + _f(0.0353) * e(-V * F / RT))
    INa = 14.838 * scale[0] * m * m * m * h * j * (V - ENa)
    IbNa = 0.00029 * (V - ENa)
    eg = e((0.35 - 1.0) * V * F / RT)
    INaCa = 1000.0 * (e(0.35 * V * F / RT) * nai ** 3 * 2.0 - eg * 140.0 ** 3 * cai * 2.5) / (
        (87.5 ** 3 + 140.0 ** 3) * (1.38 + 2.0) * (1.0 + 0.1 * eg))

    def sg(x):
        return 1.0 / (1.0 + e(x))

    xr1i, txr1 = sg((-26.0 - V) / 7.0), 450.0 * sg((-45.0 - V) / 10.0) * 6.0 * sg((V + 30.0) / 11.5)
    xr2i, txr2 = sg((V + 88.0) / 24.0), 3.0 * sg((-60.0 - V) / 20.0) * _f(1.12) * sg((V - 60.0) / 20.0)
    xsi = sg((-5.0 - V) / 14.0)
    txs = 1400.0 / torch.sqrt(1.0 + e((5.0 - V) / 6.0)) * sg((V - 35.0) / 15.0) + 80.0
    mi = sg((_f(-56.86) - V) / _f(9.03)) ** 2
    tm = sg((-60.0 - V) / 5.0) * (_f(0.1) * sg((V + 35.0) / 5.0) + _f(0.1) * sg((V - 50.0) / 200.0))
    hi = sg((V + _f(71.55)) / _f(7.43)) ** 2
    low = V < -40.0
    Vl, Vh = w(low, V, torch.full_like(V, -60.0)), w(low, torch.full_like(V, 0.0), V)
    ah = w(low, _f(0.057) * e(-(Vl + 80.0) / _f(6.8)), torch.zeros_like(V))
    bh = w(low, _f(2.7) * e(_f(0.079) * Vl) + 310000.0 * e(_f(0.3485) * Vl),
           _f(0.77) / (_f(0.13) * (1.0 + e((Vh + _f(10.66)) / _f(-11.1)))))
    aj = w(low, (-25428.0 * e(_f(0.2444) * Vl) - _f(6.948e-06) * e(_f(-0.04391) * Vl)) * (Vl + _f(37.78))
           / (1.0 + e(_f(0.311) * (Vl + _f(79.23)))), torch.zeros_like(V))
    bj = w(low, _f(0.02424) * e(_f(-0.01052) * Vl) / (1.0 + e(_f(-0.1378) * (Vl + _f(40.14)))),
           _f(0.6) * e(_f(0.057) * Vh) / (1.0 + e(_f(-0.1) * (Vh + 32.0))))
    th, tj = 1.0 / (ah + bh), 1.0 / (aj + bj)
    di = sg((-8.0 - V) / 7.5)
    td = (_f(1.4) * sg((-35.0 - V) / 13.0) + 0.25) * _f(1.4) * sg((V + 5.0) / 5.0) + sg((50.0 - V) / 20.0)
    e30 = e((V + 30.0) / 10.0)
    fi = sg((V + 20.0) / 7.0)
    tf = 1102.5 * e(-(V + 27.0) ** 2 / 225.0) + 200.0 * sg((13.0 - V) / 10.0) + 180.0 / (1.0 + e30) + 20.0
    f2i = _f(0.67) * sg((V + 35.0) / 7.0) + _f(0.33)
    tf2 = 562.0 * e(-(V + 27.0) ** 2 / 240.0) + 31.0 * sg((25.0 - V) / 10.0) + 80.0 / (1.0 + e30)
    cr = (cass / _f(0.05)) ** 2
    fci, tfc = _f(0.6) / (1.0 + cr) + _f(0.4), 80.0 / (1.0 + cr) + 2.0
    si = sg((V + 20.0) / 5.0)
    ts = 85.0 * e(-(V + 45.0) ** 2 / 320.0) + 5.0 * sg((V - 20.0) / 5.0) + 3.0
    ri = sg((20.0 - V) / 6.0)
    tr = 9.5 * e(-(V + 40.0) ** 2 / 1800.0) + _f(0.8)
    kc = 2.5 - 1.5 / (1.0 + (1.5 / casr) ** 2)
    k1 = 0.15 / kc
    O = k1 * cass * cass * rp / (0.06 + k1 * cass * cass)
    Irel = 0.102 * O * (casr - cass)
    iup = 0.006375 / (1.0 + 0.00025 ** 2 / (cai * cai))
    ileak = _f(0.00036) * (casr - cai)
    ixf = _f(0.0038) * (cass - cai)
    bi = 1.0 / (1.0 + _f(0.2) * _f(0.001) / (cai + _f(0.001)) ** 2)
    bsr = 1.0 / (1.0 + 10.0 * _f(0.3) / (casr + _f(0.3)) ** 2)
    bss = 1.0 / (1.0 + _f(0.4) * _f(0.00025) / (cass + _f(0.00025)) ** 2)
    Vc, Vsr, Vss, Cm = 0.016404, _f(0.001094), _f(5.468e-05), 0.185
    dV = -(IK1 + Ito + IKr + IKs + ICaL + INaK + INa + IbNa + INaCa + IbCa + IpK + IpCa + stim)
    drp = -_f(0.045) * kc * cass * rp + _f(0.005) * (1.0 - rp)
    dcai = bi * ((ileak - iup) * Vsr / Vc + ixf - (IbCa + IpCa - 2.0 * INaCa) * Cm / (2.0 * Vc * F))
    dcasr = bsr * (iup - (Irel + ileak))
    dcass = bss * (-ICaL * Cm / (2.0 * Vss * F) + Irel * Vsr / Vss - ixf * Vc / Vss)
    dnai = -(INa + IbNa + 3.0 * INaK + 3.0 * INaCa) / (Vc * F) * Cm
    dki = -(IK1 + Ito + IKr + IKs + IpK + stim - 2.0 * INaK) / (Vc * F) * Cm

    def g(x, inf, tau):
        return inf + (x - inf) * e(-dt / tau)

    return [V + dt * dV, g(xr1, xr1i, txr1), g(xr2, xr2i, txr2), g(xs, xsi, txs), g(m, mi, tm), g(h, hi, th),
            g(j, hi, tj), g(d, di, td), g(f, fi, tf), g(f2, f2i, tf2), g(fc, fci, tfc), g(s, si, ts), g(r, ri, tr),
            cai + dt * dcai, casr + dt * dcasr, cass + dt * dcass, rp + dt * drp, nai + dt * dnai, ki + dt * dki]


def _torord_step(y, stim, dt, ct):
    """One step of ToRORd-fkatp (Tomek et al. 2019): gates by the linearised
    update (Euler where |1/tau| < 1), the rest by Euler.  ct: 0 endo, 1 mid, 2 epi."""
    e, w = torch.exp, torch.where
    (v, CaMKt, cass, nai, nass, ki, kss, cansr, cajsr, cai, m, h, j, hp, jp, mL, hL, hLp, a, iF, iS, ap, iFp, iSp, d,
     ff, fs, fcaf, fcas, jca, ffp, fcafp, nca, ncai, c0, c1, c2, I, o, xs1, xs2, Jnp, Jp) = y
    epi, mid = ct == 2, ct == 1
    one = torch.ones_like(v)

    def by(endo, m_, p):
        return w(epi, p * one, w(mid, m_ * one, endo * one))

    def sg(x):
        return 1.0 / (1.0 + e(x))

    nao, cao, ko, cli, clo = 140.0, 1.8, 5.0, 24.0, 150.0
    R, T, F = 8314.0, 310.0, 96485.0
    L, rad = 0.01, 0.0011
    vcell = 1000 * 3.14 * rad * rad * L
    Acap = 2 * (2 * 3.14 * rad * rad + 2 * 3.14 * rad * L)
    vmyo, vnsr, vjsr, vss = 0.68 * vcell, 0.0552 * vcell, 0.0048 * vcell, 0.02 * vcell
    CaMKb = 0.05 * (1.0 - CaMKt) / (1.0 + 0.0015 / cass)
    CaMKa = CaMKb + CaMKt
    dCaMKt = 0.05 * CaMKb * CaMKa - 0.00068 * CaMKt
    RTF = R * T / F
    ENa, EK = RTF * torch.log(nao / nai), RTF * torch.log(ko / ki)
    EKs = RTF * torch.log((ko + 0.01833 * nao) / (ki + 0.01833 * nai))
    vf = v * F / (R * T)
    vff = vf * F
    ph = 1.0 / (1.0 + 0.15 / CaMKa)
    # sodium
    mss = sg(-(56.86 + v) / 9.03) ** 2
    tm = 0.1292 * e(-((v + 45.79) / 15.54) ** 2) + 0.06487 * e(-((v - 4.823) / 51.12) ** 2)
    up = v >= -40.0
    vl, vh = w(up, -60.0 * one, v), w(up, v, 0.0 * one)
    ah = w(up, 0.0 * one, 0.057 * e(-(vl + 80.0) / 6.8))
    bh = w(up, 0.77 / (0.13 * (1.0 + e(-(vh + 10.66) / 11.1))), 2.7 * e(0.079 * vl) + 3.1e5 * e(0.3485 * vl))
    aj = w(up, 0.0 * one, (-2.5428e4 * e(0.2444 * vl) - 6.948e-6 * e(-0.04391 * vl)) * (vl + 37.78)
           / (1.0 + e(0.311 * (vl + 79.23))))
    bj = w(up, 0.6 * e(0.057 * vh) / (1.0 + e(-0.1 * (vh + 32.0))),
           0.02424 * e(-0.01052 * vl) / (1.0 + e(-0.1378 * (vl + 40.14))))
    th, tj = 1.0 / (ah + bh), 1.0 / (aj + bj)
    hss, hssp = sg((v + 71.55) / 7.43) ** 2, sg((v + 77.55) / 7.43) ** 2
    INa = 11.7802 * (v - ENa) * m ** 3 * ((1.0 - ph) * h * j + ph * hp * jp)
    mLss = sg(-(v + 42.85) / 5.264)
    hLss, hLssp = sg((v + 87.61) / 7.488), sg((v + 93.81) / 7.488)
    INaL = 0.0279 * by(1.0, 1.0, 0.6) * (v - ENa) * mL * ((1.0 - ph) * hL + ph * hLp)
    # transient outward
    ass = sg(-(v - 14.34) / 14.82)
    ta = 1.0515 / (1.0 / (1.2089 * (1.0 + e(-(v - 18.4099) / 29.3814))) + 3.5 * sg((v + 100.0) / 29.3814))
    iss = sg((v + 43.94) / 5.711)
    de = w(epi, 1.0 - 0.95 * sg((v + 70.0) / 5.0), one)
    tiF = (4.562 + 1.0 / (0.3933 * e(-(v + 100.0) / 100.0) + 0.08004 * e((v + 50.0) / 16.59))) * de
    tiS = (23.62 + 1.0 / (0.001416 * e(-(v + 96.52) / 59.05) + 1.780e-8 * e((v + 114.1) / 8.079))) * de
    AiF = sg((v - 213.6) / 151.2)
    ii, ip = AiF * iF + (1.0 - AiF) * iS, AiF * iFp + (1.0 - AiF) * iSp
    assp = sg(-(v - 24.34) / 14.82)
    dti = (1.354 + 1.0e-4 / (e((v - 167.4) / 15.89) + e(-(v - 12.23) / 0.2154))) * (1.0 - 0.5 * sg((v + 70.0) / 20.0))
    Ito = 0.16 * by(1.0, 2.0, 2.0) * (v - EK) * ((1.0 - ph) * a * ii + ph * ap * ip)
    # L-type calcium
    dss = w(v > 31.4978, one, 1.0763 * e(-1.0070 * e(-0.0829 * v)))
    td = 0.6 + 1.0 / (e(-0.05 * (v + 6.0)) + e(0.09 * (v + 14.0)))
    fss = sg((v + 19.58) / 3.696)
    tff = 7.0 + 1.0 / (0.0045 * e(-(v + 20.0) / 10.0) + 0.0045 * e((v + 20.0) / 10.0))
    tfs = 1000.0 + 1.0 / (0.000035 * e(-(v + 5.0) / 4.0) + 0.000035 * e((v + 5.0) / 6.0))
    f = 0.6 * ff + 0.4 * fs
    tfcaf = 7.0 + 1.0 / (0.04 * e(-(v - 4.0) / 7.0) + 0.04 * e((v - 4.0) / 7.0))
    tfcas = 100.0 + 1.0 / (0.00012 * e(-v / 3.0) + 0.00012 * e(v / 7.0))
    Af = 0.3 + 0.6 * sg((v - 10.0) / 10.0)
    fca, fcap = Af * fcaf + (1.0 - Af) * fcas, Af * fcafp + (1.0 - Af) * fcas
    fp = 0.6 * ffp + 0.4 * fs
    jcass = sg((v + 18.08) / 2.7916)
    dnca = 500.0 / (500.0 / jca + (1.0 + 0.002 / cass) ** 4) - nca * jca
    dncai = 500.0 / (500.0 / jca + (1.0 + 0.002 / cai) ** 4) - ncai * jca
    A = 1.82e6 * (74.0 * 310.0) ** -1.5

    def gam(z2, ion):
        s = ion ** 0.5
        return -A * z2 * (s / (1.0 + s) - 0.3 * ion)

    Io = 0.5 * (nao + ko + clo + 4.0 * cao) / 1000.0
    gcao, gmo = math.exp(gam(4.0, Io)), math.exp(gam(1.0, Io))
    e1, e2 = e(vf), e(2.0 * vf)
    phi = []
    for na, k, ca in ((nass, kss, cass), (nai, ki, cai)):
        ion = 0.5 * (na + k + cli + 4.0 * ca) / 1000.0
        gca, gm = e(gam(4.0, ion)), e(gam(1.0, ion))
        phi.append((4.0 * vff * (gca * ca * e2 - gcao * cao) / (e2 - 1.0), vff * (gm * na * e1 - gmo * nao) / (e1 - 1.0),
                    vff * (gm * k * e1 - gmo * ko) / (e1 - 1.0)))
    gcai = gca
    PCa = 8.3757e-05 * by(1.0, 2.0, 1.2)
    oss = d * ((1.0 - ph) * (f * (1.0 - nca) + jca * fca * nca) + 1.1 * ph * (fp * (1.0 - nca) + jca * fcap * nca))
    osi = d * ((1.0 - ph) * (f * (1.0 - ncai) + jca * fca * ncai) + 1.1 * ph * (fp * (1.0 - ncai) + jca * fcap * ncai))
    ICaLs, ICaNas, ICaKs = 0.8 * PCa * phi[0][0] * oss, 0.8 * 0.00125 * PCa * phi[0][1] * oss, 0.8 * 3.574e-4 * PCa * phi[0][2] * oss
    fi = 1.0 - 0.8
    ICaLi, ICaNai, ICaKi = fi * PCa * phi[1][0] * osi, fi * 0.00125 * PCa * phi[1][1] * osi, fi * 3.574e-4 * PCa * phi[1][2] * osi
    ICaL = ICaLs + ICaLi
    # rapid delayed rectifier
    al, be = 0.1161 * e(0.2990 * vf), 0.2442 * e(-1.604 * vf)
    al1, be1 = 1.25 * 0.1235, 0.1911
    al2, be2 = 0.0578 * e(0.9710 * vf), 0.349e-3 * e(-1.062 * vf)
    ali, bei = 0.2533 * e(0.5953 * vf), 1.25 * 0.0522 * e(-0.8209 * vf)
    aci = 0.52e-4 * e(1.525 * vf)
    bic = be2 * bei * aci / (al2 * ali)
    dc0 = c1 * be - c0 * al
    dc1 = c0 * al + c2 * be1 - c1 * (be + al1)
    dc2 = c1 * al1 + o * be2 + I * bic - c2 * (be1 + al2 + aci)
    do = c2 * al2 + I * bei - o * (be2 + ali)
    dI = c2 * aci + o * ali - I * (bic + bei)
    IKr = 0.0321 * math.sqrt(ko / 5.0) * by(1.0, 0.8, 1.3) * o * (v - EK)
    # slow delayed and inward rectifiers
    xss = sg(-(v + 11.60) / 8.932)
    tx1 = 817.3 + 1.0 / (2.326e-4 * e((v + 48.28) / 17.80) + 0.001292 * e(-(v + 210.0) / 230.0))
    tx2 = 1.0 / (0.01 * e((v - 50.0) / 20.0) + 0.0193 * e(-(v + 66.54) / 31.0))
    IKs = 0.0011 * by(1.0, 1.0, 1.4) * (1.0 + 0.6 / (1.0 + (3.8e-5 / cai) ** 1.4)) * xs1 * xs2 * (v - EKs)
    vk = v - EK
    ak = 4.094 / (1.0 + e(0.1217 * (vk - 49.934)))
    bk = (15.72 * e(0.0674 * (vk - 3.257)) + e(0.0618 * (vk - 594.31))) / (1.0 + e(-0.1629 * (vk + 14.207)))
    IK1 = 0.6992 * by(1.0, 1.3, 1.2) * math.sqrt(ko / 5.0) * ak / (ak + bk) * vk
    # sodium-calcium exchange
    hca, hna = e(0.1670 * vf), e(0.5224 * vf)

    def ncx(na, ca):
        h1 = 1.0 + na / 88.12 * (1.0 + hna)
        h2, h3 = na * hna / (88.12 * h1), 1.0 / h1
        h4 = 1.0 + na / 15.0 * (1.0 + na / 5.0)
        h5, h6 = na * na / (h4 * 15.0 * 5.0), 1.0 / h4
        h7 = 1.0 + nao / 88.12 * (1.0 + 1.0 / hna)
        h8, h9 = nao / (88.12 * hna * h7), 1.0 / h7
        h10 = 12.5 + 1.0 + nao / 15.0 * (1.0 + nao / 5.0)
        h11, h12 = nao * nao / (h10 * 15.0 * 5.0), 1.0 / h10
        k1, k2 = h12 * cao * 1.5e6, 5.0e3
        k3p, k3q = h9 * 6.0e4, h8 * 5.0e3
        k3 = k3p + k3q
        k4p, k4q = h3 * 6.0e4 / hca, h2 * 5.0e3
        k4, k5, k6 = k4p + k4q, 5.0e3, h6 * ca * 1.5e6
        k7, k8 = h5 * h2 * 6.0e4, h8 * h11 * 6.0e4
        x1 = k2 * k4 * (k7 + k6) + k5 * k7 * (k2 + k3)
        x2 = k1 * k7 * (k4 + k5) + k4 * k6 * (k1 + k8)
        x3 = k1 * k3 * (k7 + k6) + k8 * k6 * (k2 + k3)
        x4 = k2 * k8 * (k4 + k5) + k3 * k5 * (k1 + k8)
        s = x1 + x2 + x3 + x4
        E1, E2, E3, E4 = x1 / s, x2 / s, x3 / s, x4 / s
        al_ = 1.0 / (1.0 + (150.0e-6 / ca) ** 2)
        return al_ * (3.0 * (E4 * k7 - E1 * k8) + E3 * k4q - E2 * k3q + 2.0 * (E2 * k2 - E1 * k1))

    G = 0.0034 * by(1.0, 1.4, 1.1)
    INCi, INCs = (1.0 - 0.35) * G * ncx(nai, cai), 0.35 * G * ncx(nass, cass)
    # sodium-potassium pump
    kn = 9.073 * e(-0.1550 * vf / 3.0)
    kno = 27.78 * e((1.0 + 0.1550) * vf / 3.0)
    P = 4.2 / (1.0 + 1.0e-7 / 1.698e-7 + nai / 224.0 + ki / 292.0)
    Di = (1.0 + nai / kn) ** 3 + (1.0 + ki / 0.5) ** 2 - 1.0
    Do = (1.0 + nao / kno) ** 3 + (1.0 + ko / 0.3582) ** 2 - 1.0
    am = 9.8 / 1.698e-7
    a1, b1 = 949.5 * (nai / kn) ** 3 / Di, 182.4 * 0.05
    a2, b2 = 687.2, 39.4 * (nao / kno) ** 3 / Do
    a3, b3 = 1899.0 * (ko / 0.3582) ** 2 / Do, 79300.0 * P * 1.0e-7 / (1.0 + am)
    a4, b4 = 639.0 * am / (1.0 + am), 40.0 * (ki / 0.5) ** 2 / Di
    x1 = a4 * a1 * a2 + b2 * b4 * b3 + a2 * b4 * b3 + b3 * a1 * a2
    x2 = b2 * b1 * b4 + a1 * a2 * a3 + a3 * b1 * b4 + a2 * a3 * b4
    x3 = a2 * a3 * a4 + b3 * b2 * b1 + b2 * b1 * a4 + a3 * a4 * b1
    x4 = b4 * b3 * b2 + a3 * a4 * a1 + b2 * a4 * a1 + b3 * b2 * a1
    xs = x1 + x2 + x3 + x4
    INaK = 15.4509 * by(1.0, 1.0, 0.9) * (3.0 * (x1 * a3 - x2 * b3) + 2.0 * (x4 * b1 - x3 * a1)) / xs
    # background, pump, chloride
    IKb = 0.0189 * by(1.0, 1.0, 0.6) * sg(-(v - 10.8968) / 23.9871) * (v - EK)
    INab = 1.9239e-09 * vff * (nai * e1 - nao) / (e1 - 1.0)
    ICab = 5.9194e-08 * 4.0 * vff * (gcai * cai * e2 - gcao * cao) / (e2 - 1.0)
    IpCa = 5e-04 * cai / (0.0005 + cai)
    ECl = RTF * math.log(cli / clo)
    ICl = 0.2843 / (1.0 + 0.1 / cass) * (v - ECl)
    IClb = 1.98e-3 * (v - ECl)
    # sarcoplasmic reticulum
    jr8 = (1.7 / cajsr) ** 8
    rel = by(1.0, 1.7, 1.0)
    Ji = 0.5 * 4.75 * (-ICaL) / (1.0 + jr8) * rel
    Jip = 0.5 * 1.25 * 4.75 * (-ICaL) / (1.0 + jr8) * rel
    tr = torch.clamp(4.75 / (1.0 + 0.0123 / cajsr), min=0.001)
    trp = torch.clamp(1.25 * 4.75 / (1.0 + 0.0123 / cajsr), min=0.001)
    Jrel = 1.5378 * ((1.0 - ph) * Jnp + ph * Jp)
    ups = by(1.0, 1.0, 1.3)
    Jup = (1.0 - ph) * ups * 0.005425 * cai / (cai + 0.00092) + ph * ups * 2.75 * 0.005425 * cai / (
        cai + 0.00092 - 0.00017) - 0.0048825 * cansr / 15.0
    Jtr = (cansr - cajsr) / 60.0
    dv = -(INa + INaL + Ito + ICaL + (ICaNas + ICaNai) + (ICaKs + ICaKi) + IKr + IKs + IK1 + INCi + INCs + INaK + INab
           + IKb + IpCa + ICab + ICl + IClb + stim)
    JdNa, JdK, Jd = (nass - nai) / 2.0, (kss - ki) / 2.0, (cass - cai) / 0.2
    dnai = -(ICaNai + INa + INaL + 3.0 * INCi + 3.0 * INaK + INab) * Acap / (F * vmyo) + JdNa * vss / vmyo
    dnass = -(ICaNas + 3.0 * INCs) * Acap / (F * vss) - JdNa
    dki = -(ICaKi + Ito + IKr + IKs + IK1 + IKb + stim - 2.0 * INaK) * Acap / (F * vmyo) + JdK * vss / vmyo
    dkss = -ICaKs * Acap / (F * vss) - JdK
    Bi = 1.0 / (1.0 + 0.05 * by(1.0, 1.0, 1.3) * 0.00238 / (0.00238 + cai) ** 2 + 0.07 * 0.0005 / (0.0005 + cai) ** 2)
    dcai = Bi * (-(ICaLi + IpCa + ICab - 2.0 * INCi) * Acap / (2.0 * F * vmyo) - Jup * vnsr / vmyo + Jd * vss / vmyo)
    Bs = 1.0 / (1.0 + 0.047 * 0.00087 / (0.00087 + cass) ** 2 + 1.124 * 0.0087 / (0.0087 + cass) ** 2)
    dcass = Bs * (-(ICaLs - 2.0 * INCs) * Acap / (2.0 * F * vss) + Jrel * vjsr / vss - Jd)
    dcansr = Jup - Jtr * vjsr / vnsr
    dcajsr = (Jtr - Jrel) / (1.0 + 10.0 * 0.8 / (0.8 + cajsr) ** 2)

    def g(x, tau, inf):
        tau = tau * one
        dec = -dt / tau
        return w(tau > 1.0, x + dt * (inf - x) / tau, inf + (x - inf) * e(dec))

    def eu(x, dx):
        return x + dt * dx

    return [eu(v, dv), eu(CaMKt, dCaMKt), eu(cass, dcass), eu(nai, dnai), eu(nass, dnass), eu(ki, dki), eu(kss, dkss),
            eu(cansr, dcansr), eu(cajsr, dcajsr), eu(cai, dcai), g(m, tm, mss), g(h, th, hss), g(j, tj, hss),
            g(hp, th, hssp), g(jp, 1.46 * tj, hss), g(mL, tm, mLss), g(hL, 200.0, hLss), g(hLp, 600.0, hLssp),
            g(a, ta, ass), g(iF, tiF, iss), g(iS, tiS, iss), g(ap, ta, assp), g(iFp, dti * tiF, iss),
            g(iSp, dti * tiS, iss), g(d, td, dss), g(ff, tff, fss), g(fs, tfs, fss), g(fcaf, tfcaf, fss),
            g(fcas, tfcas, fss), g(jca, 75.0, jcass), g(ffp, 2.5 * tff, fss), g(fcafp, 2.5 * tfcaf, fss),
            eu(nca, dnca), eu(ncai, dncai), eu(c0, dc0), eu(c1, dc1), eu(c2, dc2), eu(I, dI), eu(o, do),
            g(xs1, tx1, xss), g(xs2, tx2, xss), g(Jnp, tr, Ji), g(Jp, trp, Jip)]


def _advance(model, y, stim, dt, ct, scale, chunk=1 << 21):
    """y: (neq, n) state, advanced in place, a chunk of cells at a time."""
    for lo in range(0, y.shape[1], chunk):
        c = slice(lo, lo + chunk)
        st = stim[c] if torch.is_tensor(stim) else stim
        cols = [r[c] for r in y]
        if model == "tt2006":
            new = _tt2006_step(cols, st, dt, (1.0,) * 5 if scale is None else [q[c] for q in scale])
        else:
            new = _torord_step(cols, st, dt, ct[c])
        y[:, c] = torch.stack(new)


ALPHA = 0.14 * 1.0 / DT * _f(1e-8) * DX ** 3


def _faces(shape, cx, cy, cz, active):
    """Couplings of the 7-point operator across the three face families, zero
    at removed cells; cx, cy, cz: numbers or tensors of the face shapes."""
    out = []
    for ax, c in ((2, cx), (1, cy), (0, cz)):
        s = list(shape)
        s[ax] -= 1
        k = torch.zeros(s, dtype=torch.float64, device=active.device) + c
        n = shape[ax]
        out.append((ax, k * active.narrow(ax, 0, n - 1) * active.narrow(ax, 1, n - 1)))
    return out


def _seven_point(faces, alpha, active):
    def mul(x):
        y = alpha * x * active
        for ax, k in faces:
            if k.numel() == 0:
                continue
            n = x.shape[ax]
            flux = k * (x.narrow(ax, 0, n - 1) - x.narrow(ax, 1, n - 1))
            y.narrow(ax, 0, n - 1).add_(flux)
            y.narrow(ax, 1, n - 1).sub_(flux)
        return y

    diag = torch.full_like(active, alpha)
    for ax, k in faces:
        if k.numel():
            n = active.shape[ax]
            diag.narrow(ax, 0, n - 1).add_(k)
            diag.narrow(ax, 1, n - 1).add_(k)
    return mul, diag


def _rotating(nx, ny, nz, angles, sl, st, alpha, device):
    """The anisotropic operator with in-plane fibres turning through the
    planes: face conductivities averaged over the two cells, and the cross
    conductivity of a face averaged over the pairs of cells beside it that
    exist (divided by their number once more), on the rows of each plane for
    the 3 x 3 kinds of cell (first, inner and last in x and y)."""
    D = [(st + (sl - st) * math.cos(t) ** 2, st + (sl - st) * math.sin(t) ** 2, (sl - st) * math.cos(t) * math.sin(t), st)
         for t in angles]
    rows = np.zeros((nz, 3, 3, 3, 3, 3))          # plane, y kind, x kind, offsets z, y, x
    for k in range(nz):
        for jy in range(3):
            for jx in range(3):
                def ok(x, y, z):
                    return (0 <= k + z < nz and not (x < 0 and jx == 0) and not (x > 0 and jx == 2)
                            and not (y < 0 and jy == 0) and not (y > 0 and jy == 2))
                r = np.zeros((3, 3, 3))           # offsets z, y, x
                r[1, 1, 1] = alpha
                for x, y, z, q in ((1, 0, 0, 0), (-1, 0, 0, 0), (0, 1, 0, 1), (0, -1, 0, 1), (0, 0, 1, 3), (0, 0, -1, 3)):
                    if ok(x, y, z):
                        c = 0.5 * (D[k][q] + D[k + z][q]) * DX
                        r[1, 1, 1] += c
                        r[1 + z, 1 + y, 1 + x] -= c

                def cross(face):                  # face: +-1 in x (0) or in y (1)
                    ax, sgn = face
                    if not ok(*((sgn, 0, 0) if ax == 0 else (0, sgn, 0))):
                        return 0.0
                    tot, cnt = 0.0, 0
                    for z in (0, 1, -1):
                        for t in (0, sgn):
                            p, m = ((t, 1, z), (t, -1, z)) if ax == 0 else ((1, t, z), (-1, t, z))
                            if ok(*p) and ok(*m):
                                tot += 2.0 * D[k + z][2]
                                cnt += 2
                    return tot / cnt / cnt if cnt else 0.0

                right, left, top, down = cross((0, 1)), cross((0, -1)), cross((1, 1)), cross((1, -1))
                for z in (-1, 0, 1):
                    for x, c in ((-1, left), (0, left - right), (1, -right)):
                        if ok(x, 1, z) and ok(x, -1, z):
                            r[1 + z, 2, 1 + x] += c * DX
                            r[1 + z, 0, 1 + x] -= c * DX
                    for y, c in ((-1, down), (0, down - top), (1, -top)):
                        if ok(1, y, z) and ok(-1, y, z):
                            r[1 + z, 1 + y, 2] += c * DX
                            r[1 + z, 1 + y, 0] -= c * DX
                rows[k, jy, jx] = r
    rows = torch.tensor(rows, device=device)
    kx = torch.ones(nx, dtype=torch.long, device=device)
    ky = torch.ones(ny, dtype=torch.long, device=device)
    kx[0], kx[-1], ky[0], ky[-1] = 0, 2, 0, 2

    def coef(z, y, x):
        return rows[:, :, :, z, y, x][:, ky][:, :, kx]

    used = [(z, y, x) for z in range(3) for y in range(3) for x in range(3) if bool((rows[:, :, :, z, y, x] != 0).any())]
    big = nx * ny * nz > 6_000_000
    stored = {} if big else {q: coef(*q) for q in used}

    def mul(v):
        p = torch.nn.functional.pad(v, (1, 1, 1, 1, 1, 1))
        out = torch.zeros_like(v)
        for q in used:
            c = coef(*q) if big else stored[q]
            out.addcmul_(c, p[q[0]:q[0] + nz, q[1]:q[1] + ny, q[2]:q[2] + nx])
        return out

    return mul, coef(1, 1, 1)


def _cg(mul, diag, b, x0, rel2=1e-30, most=300):
    """Jacobi-preconditioned conjugate gradients to rounding."""
    x = x0.clone()
    r = b - mul(x)
    stop = rel2 * float((b * b).sum())
    z = r / diag
    p = z.clone()
    rz = (r * z).sum()
    last = math.inf
    for _ in range(most):
        rr = float((r * r).sum())
        if rr <= stop or (rr >= last and rr <= 1e4 * stop):
            break
        last = rr
        q = mul(p)
        al = rz / (p * q).sum()
        x += al * p
        r -= al * q
        z = r / diag
        rz, old = (r * z).sum(), rz
        p = z + (rz / old) * p
    return x


def _loop(case, kw, shape, stim_of, steps, scale=None):
    """The operator-split loop from rest; stim_of(step): the merged stimulus of
    the active cells."""
    dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
    nz, ny, nx = shape
    n = nx * ny * nz
    act = torch.ones(n, dtype=torch.float64, device=dev)
    if kw.get("active") is not None:
        act = torch.tensor(kw["active"], device=dev).double()
    cells = torch.nonzero(act).reshape(-1)
    a3 = act.reshape(shape)
    ct = None
    if kw["model"] == "torord":
        types = np.zeros(n, dtype=np.int64) if kw.get("celltype") is None else kw["celltype"].astype(np.int64)
        ct = torch.tensor(types, device=dev)[cells]
        y = torch.tensor(TORORD_STATE, dtype=torch.float64, device=dev).T[:, ct].contiguous()
        v0 = -88.763800
    else:
        y = torch.tensor(TT2006_STATE, dtype=torch.float64, device=dev)[:, None].repeat(1, cells.numel())
        v0 = _f(-85.23)
    if kw.get("fibre_angle_z") is not None:
        mul, diag = _rotating(nx, ny, nz, kw["fibre_angle_z"], kw["sigma_l"], kw["sigma_t"], ALPHA, dev)
    else:
        c = [kw["sigma_l"], kw["sigma_t"], kw["sigma_t"]] if kw["assembly"] == "anisotropic" else list(kw["sigma"])
        mul, diag = _seven_point(_faces(shape, *[q * DX for q in c], a3), ALPHA, a3)
    v = (v0 * act).reshape(shape)
    for k in range(steps):
        _advance(kw["model"], y, stim_of(k, cells), DT, ct, scale)
        vs = torch.zeros(n, dtype=torch.float64, device=dev)
        vs[cells] = y[0]
        v = _cg(mul, diag, ALPHA * vs.reshape(shape), v)
        y[0] = v.reshape(-1)[cells]
    return v.reshape(-1)


def _windows(steps):
    """Loop times by repeated addition, as the loop clock has them."""
    t, out = 0.0, []
    for _ in range(steps):
        out.append(t)
        t += DT
    return out


def exact(case, seed):
    kind = case["kind"]
    dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
    if kind in ("tissue", "host"):
        kw = _tissue_inputs(case, seed)
        nx, ny, nz = case["nx"], case["ny"], case["nz"]
        steps = case.get("steps", 1)
        times = _windows(steps)
        mask = torch.tensor(kw["mask"], device=dev).double()
        if kind == "host":
            stim = kw["current"] * mask
            v = _loop(case, kw, (nz, ny, nx), lambda k, cells: stim[cells], steps)
            if kw.get("active") is not None:
                v = v.clone()
                v[torch.tensor(kw["active"], device=dev) == 0] = 0.0
            return v.cpu().numpy()
        x = (torch.arange(nx, dtype=torch.float64, device=dev) + 0.5) * DX < kw["x_limit"]
        plane = kw["current"] * x.double().repeat(ny * nz)

        def stim_of(k, cells):
            return (plane + (-53.0 * mask if times[k] <= 1.0 else 0.0))[cells] if times[k] <= 2.0 else 0.0
        return _loop(case, kw, (nz, ny, nx), stim_of, steps)
    if kind == "batch":
        from monoalg3d_c_b200.batch import pack        # where each tissue's cells lie in the atlas
        sizes, scales, cur = _batch_inputs(case, seed)
        W, H, x0, y0 = pack(sizes)
        active = np.zeros((H, W), dtype=np.uint8)
        sc = np.ones((5, H, W))
        edge = np.zeros((H, W))
        for q, (a, b) in enumerate(sizes):
            s = (slice(y0[q], y0[q] + b), slice(x0[q], x0[q] + a))
            active[s] = 1
            sc[(slice(None),) + s] = scales[q].astype(np.float32)[:, None, None]
            edge[s[0], x0[q]] = cur
        kw = dict(model="tt2006", assembly="homogeneous", sigma=(0.13 * S_PER_M,) * 3, active=active.reshape(-1))
        on = active.reshape(-1) != 0
        scale = torch.tensor(sc.reshape(5, -1)[:, on], device=dev)
        stim = torch.tensor(edge.reshape(-1), device=dev)
        return _loop(case, kw, (1, H, W), lambda k, cells: stim[cells], case["steps"], scale)
    if kind == "gradient":
        return _exact_gradient(case, seed, dev)
    if kind in ("population", "plugin"):
        ct, state, stim = _cells_inputs(case, seed)
        y = torch.tensor(state, device=dev)
        c = None if ct is None else torch.tensor(ct.astype(np.int64), device=dev)
        if case["precision"] == "mixed":
            y = _as_mixed(case["model"], y)
        s = torch.tensor(stim, device=dev)
        for _ in range(case.get("substeps", 1)):
            _advance(case["model"], y, s, DT, c, None)
        return y if kind == "plugin" else y.cpu().numpy()
    ptr, col, val, b, x0 = _csr_inputs(case, seed)
    n = b.size
    a = torch.sparse_csr_tensor(torch.tensor(ptr.astype(np.int64)), torch.tensor(col.astype(np.int64)), torch.tensor(val),
                                size=(n, n)).to(dev)
    rows = np.repeat(np.arange(n), np.diff(ptr))
    diag = torch.tensor(val[rows == col], device=dev)
    return _cg(lambda x: a @ x, diag, torch.tensor(b, device=dev), torch.tensor(x0, device=dev)).cpu().numpy()


def _as_mixed(model, y):
    """The states that the mixed form holds as floats, as it is given them."""
    keep = {0, 13, 14, 15, 17, 18} if model == "tt2006" else {0} | set(range(2, 10))
    out = y.clone()
    for s in range(y.shape[0]):
        if s not in keep:
            out[s] = y[s].float().double()
    return out


class _Solve(torch.autograd.Function):
    """v = A(sigma)^-1 (alpha v*), with the adjoint of the solve."""

    @staticmethod
    def forward(ctx, vs, sigma, guess):
        op = _sheet_operator(sigma)
        v = _cg(op[0], op[1], ALPHA * vs, guess)
        ctx.save_for_backward(sigma, v)
        return v

    @staticmethod
    def backward(ctx, lam):
        sigma, v = ctx.saved_tensors
        op = _sheet_operator(sigma)
        w = _cg(op[0], op[1], lam, torch.zeros_like(lam))
        with torch.enable_grad():
            s = sigma.detach().requires_grad_()
            form = sum((_face_sigma(s, ax) * DX * _diff(w, ax) * _diff(v, ax)).sum() for ax in (0, 1))
            gs, = torch.autograd.grad(-form, s)
        return ALPHA * w, gs, None


def _diff(x, ax):
    return x.narrow(ax, 0, x.shape[ax] - 1) - x.narrow(ax, 1, x.shape[ax] - 1)


def _face_sigma(s, ax):
    a, b = s.narrow(ax, 0, s.shape[ax] - 1), s.narrow(ax, 1, s.shape[ax] - 1)
    return 2.0 * a * b / (a + b)


def _sheet_operator(sigma):
    s = sigma.detach()
    active = torch.ones_like(s)
    return _seven_point([(1, _face_sigma(s, 1) * DX), (0, _face_sigma(s, 0) * DX)], ALPHA, active)


def _exact_gradient(case, seed, dev):
    sigma, gkr, sensors, mask, data = _gradient_inputs(case, seed)
    nx, ny = case["nx"], case["ny"]
    sig = torch.tensor(sigma.reshape(ny, nx), device=dev, requires_grad=True)
    g = torch.tensor(gkr, device=dev, requires_grad=True)
    one = torch.ones(nx * ny, dtype=torch.float64, device=dev)
    # scalings are held as floats; their gradient passes the rounding unchanged
    scale = (one, g + (g.detach().float().double() - g.detach()), one, one, one)
    y = [one * v for v in TT2006_STATE]
    stim = -53.0 * torch.tensor(mask, device=dev).double()
    times = _windows(case["nsteps"])
    sens = torch.tensor(sensors, device=dev)
    v = (one * _f(-85.23)).reshape(ny, nx)
    traces = []
    for k in range(case["nsteps"]):
        y = _tt2006_step(y, stim if times[k] <= 2.0 else 0.0, DT, scale)
        v = _Solve.apply(y[0].reshape(ny, nx), sig, v.detach())
        y[0] = v.reshape(-1)
        if (k + 1) % case["sample_every"] == 0:
            traces.append(y[0][sens])
    tr = torch.stack(traces)
    loss = 0.5 * ((tr - torch.tensor(data, device=dev)) ** 2).sum()
    loss.backward()
    return {"traces": tr.detach(), "grad_sigma": sig.grad.reshape(-1), "grad_gkr": g.grad}
