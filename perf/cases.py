"""The work that programs have this framework do, as cases that can be timed and compared.

A case is a dict of plain values; its "kind" says which public entry points it goes through:

  step      a basin advanced through GpuRun, its surface elevation and its 3-D state read back
  ensemble  several basins advanced together through ensemble.Ensemble
  solve     the stand-alone zeta solve on Purdue arrays (model.solve_zeta), host to host
  tridiag   batched column tridiagonals on device buffers (si3d_gpu_column_tridiag_noalloc)
  train     one gradient of the guess network (learn.Net: forward, loss, backward) on image crops
  infer     the guess network on a whole basin's image (learn.Net.forward)

listed() names the cases, draw() gives more of the same ranges, prepare() makes what a program holds
before the call, run() is one pass, work() the bytes and operations a pass cannot do without, and
exact() the result in 64 bits from plain torch where the work has one.
"""
import ctypes as C
import math
import tempfile

import numpy as np
import torch

from si3d_b200 import learn, native, synth
from si3d_b200.ensemble import Ensemble
from si3d_b200.model import GpuRun, solve_zeta

# Solver forms by name: precision, initial guess, whether the trained network is loaded.
FORMS = {
    "fp64": (native.SI3D_FP64, native.SI3D_X0_PREV, False),
    "mixed_ir": (native.SI3D_MIXED_IR, native.SI3D_X0_LAST, False),
    "mg": (native.SI3D_MIXED_MG, native.SI3D_X0_LAST, False),
    "learned_mg": (native.SI3D_MIXED_MG, native.SI3D_X0_LEARNED, True),
}


# ---------------------------------------------------------------------------- the cases
def _step(nx, ny, layers, form, steps, *, bowl=False, coupled=False, tuned=False, ntr=0, iturb=0):
    return {"kind": "step", "nx": nx, "ny": ny, "layers": layers, "form": form, "steps": steps, "bowl": bowl,
            "coupled": coupled, "tuned": tuned, "ntr": ntr, "iturb": iturb}


def listed():
    named = [
        # a small lake driven by a weather or ecology model that hands it new winds before every
        # step and reads the surface after it: the smallest steps, with the constructor's defaults
        ("bowl_coupled", _step(100, 50, 20, "fp64", 1, bowl=True, coupled=True)),
        # a medium lake of no round size, the learned guess in front of the multigrid solve
        ("basin_ragged", _step(517, 283, 23, "learned_mg", 10)),
        # the plain FP64 form (the reference's own algorithm) on the 1000 x 500 x 40 workload
        ("basin_fp64", _step(1000, 500, 40, "fp64", 4, tuned=True)),
        # the benchmark's workload and headline form, the largest
        ("basin_large", _step(2000, 1000, 60, "mg", 6, tuned=True)),
        # a water-quality run: conservative tracers carried along, refined FP32 solves
        ("tracers", _step(601, 307, 31, "mixed_ir", 4, ntr=5)),
        # a run with the Mellor-Yamada closure instead of constant eddy coefficients
        ("closure", _step(640, 360, 45, "mg", 5, iturb=1)),
        # a parameter or site study: several lakes of different sizes, one graph launch per step
        ("ensemble", {"kind": "ensemble", "members": 8, "nx": 400, "ny": 240, "layers": 40, "steps": 4}),
        # a Fortran host that replaces only its NSPCG call
        ("zeta_solve", {"kind": "solve", "nx": 300, "ny": 250, "precision": "fp64", "ratio": 120.0}),
        # a host model's own vertical solves on buffers that it owns
        ("column_tridiag", {"kind": "tridiag", "layers": 40, "columns": 20011}),
        # training the guess network: the batch and crop size of `learn train`
        ("net_train", {"kind": "train", "batch": 32, "height": 64, "width": 64}),
        # the network on the image of the 1000 x 500 workload
        ("net_image", {"kind": "infer", "batch": 1, "height": 1002, "width": 502}),
    ]
    return [dict(c, name=n) for n, c in named]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step"] * 6 + ["ensemble", "solve", "tridiag", "train", "infer"])
    if kind == "step":
        form = rng.choice(sorted(FORMS))
        nx, ny, layers = _log(rng, 60, 1300), _log(rng, 40, 700), rng.randint(8, 60)
        extra = rng.choice(["plain", "plain", "tracers", "closure", "coupled"])
        return _step(nx, ny, layers, form, rng.randint(1, 8), bowl=rng.random() < 0.2, coupled=extra == "coupled",
                     tuned=rng.random() < 0.5, ntr=rng.randint(1, 6) if extra == "tracers" else 0,
                     iturb=1 if extra == "closure" else 0)
    if kind == "ensemble":
        return {"kind": kind, "members": rng.randint(2, 12), "nx": _log(rng, 80, 500), "ny": _log(rng, 60, 300),
                "layers": rng.randint(12, 50), "steps": rng.randint(1, 6)}
    if kind == "solve":
        return {"kind": kind, "nx": _log(rng, 40, 600), "ny": _log(rng, 30, 400),
                "precision": rng.choice(["fp64", "mixed_ir"]), "ratio": rng.uniform(10.0, 200.0)}
    if kind == "tridiag":
        layers = rng.randint(3, 90)
        return {"kind": kind, "layers": layers, "columns": _log(rng, 100, native_columns(layers))}
    if kind == "train":
        side = rng.choice([32, 48, 64, 80])
        return {"kind": kind, "batch": rng.randint(4, 40), "height": side, "width": side}
    return {"kind": kind, "batch": 1, "height": _log(rng, 60, 2002), "width": _log(rng, 50, 1002)}


def native_columns(layers):
    """Columns of `layers` levels that one allocation-free tridiagonal call takes at most."""
    return (1 << 20) // layers


# ---------------------------------------------------------------------------- inputs
def _basin(nx, ny, layers, rng, *, bowl=False, ntr=0, iturb=0):
    """A lake of the synthetic workloads' generators: its bathymetry goes with its size (a program's
    lake stays the same from run to run), the wind field and the temperatures with the seed."""
    bed = 1000 * nx + 10 * ny + layers
    top, bottom = rng.uniform(16.0, 24.0), rng.uniform(6.0, 12.0)
    if bowl:
        depth = synth.bowl_bathymetry(nx, ny, 100.0, 100.0, hmax=float(layers))
        u = synth.wind_speed_for_stress(synth.stress_field(nx, ny, int(rng.integers(1 << 30)), rel=0.3, corr=10.0))
        dx, dt, ddz = 100.0, 60.0, 1.0
    else:
        ddz = min(1.5, 60.0 / layers)
        corr = min(20.0, max(4.0, min(nx, ny) / 8.0))
        depth = synth.random_bathymetry(nx, ny, bed, corr=corr, dmax=layers * ddz)
        u = synth.wind_speed_for_stress(synth.stress_field(nx, ny, int(rng.integers(1 << 30)), corr=corr))
        dx, dt = 50.0, 30.0
    return synth.Basin("lake", nx, ny, dx, dx, depth, layers, ddz, dt, 1000, dzmin=0.05 if bowl else 0.1, uair=u,
                       vair=0.2 * u, t_top=float(top), t_bottom=float(bottom), ntr=ntr, iturb=iturb)


def _pinned(n, dtype):
    return torch.empty(int(n), dtype=dtype, pin_memory=True)


def _frame_size(run, kind, arg):
    n = C.c_longlong(0)
    native.check(run.g.si3d_gpu_output_frame(run.gh, kind, arg, 0, None, 0, C.byref(n)))
    return n.value


def _outputs_of(run, case):
    """Page-locked buffers for what the program reads after a pass: the ptrack frame (hp, u, v, w
    and temperature of every wet cell), the tracers' frames, with the closure a plane (Av)."""
    frames = [("state", native.SI3D_OUT_PTRACK, 0)]
    frames += [(f"tracer{t}", native.SI3D_OUT_TRACER, t) for t in range(1, case.get("ntr", 0) + 1)]
    if case.get("iturb"):
        frames.append(("plane", native.SI3D_OUT_PLANE, 4))
    return [(n, k, a, _pinned(_frame_size(run, k, a), torch.float32)) for n, k, a in frames]


def _read(run, frames, zeta):
    g, out, tickets = run.g, {}, []
    native.check(g.si3d_gpu_fetch_field(run.gh, b"s", C.c_void_p(zeta.data_ptr())))
    for name, kind, arg, buf in frames:
        n, t = C.c_longlong(0), C.c_ulonglong(0)
        native.check(g.si3d_gpu_output_frame_async(run.gh, kind, arg, 0, C.c_void_p(buf.data_ptr()), buf.numel(),
                                                   C.byref(n), C.byref(t)))
        tickets.append(t.value)
        out[name] = buf.numpy()
    for t in tickets:
        native.check(g.si3d_gpu_output_wait(run.gh, t))
    native.check(g.si3d_gpu_copies_wait(run.gh))
    out["zeta"] = zeta.numpy()
    return out


def _prepare_step(case, rng):
    basin = _basin(case["nx"], case["ny"], case["layers"], rng, bowl=case["bowl"], ntr=case["ntr"], iturb=case["iturb"])
    precision, x0, net = FORMS[case["form"]]
    with tempfile.TemporaryDirectory(prefix="si3d_case_") as d:
        synth.write_run(basin, d)
        run = GpuRun(d, pcg_itmax=2000, precision=precision, x0_mode=x0)
    if net:
        run.set_net(learn.load_params())
    run.run(1)   # the start-up step, which differs from all later ones
    if case["tuned"]:
        run.autotune()
    st = {"run": run, "steps": case["steps"], "frames": _outputs_of(run, case), "zeta": _pinned(run.lm1, torch.float64)}
    if case["coupled"]:
        names = ("uair", "vair", "cdw")
        now = {k: run.get(k) for k in names}
        winds = []
        for gust in (1.0, 1.05):
            group = {k: _pinned(run.lm1, torch.float64) for k in names}
            for k in names:
                group[k].copy_(torch.from_numpy(now[k] * (1.0 if k == "cdw" else gust)))
            winds.append(group)
        st.update(winds=winds, turn=0)
    return st


def _run_step(st):
    run = st["run"]
    if "winds" in st:
        for k, w in st["winds"][st["turn"]].items():
            native.check(run.g.si3d_gpu_stage_field(run.gh, k.encode(), C.c_void_p(w.data_ptr())))
        native.check(run.g.si3d_gpu_stage_commit(run.gh))
        st["turn"] ^= 1
    native.check(run.h.si3d_host_run(run.hm, st["steps"], None))
    return _read(run, st["frames"], st["zeta"])


def _prepare_ensemble(case, rng):
    dirs = []
    with tempfile.TemporaryDirectory(prefix="si3d_case_") as root:
        for k in range(case["members"]):
            f = 1.0 - 0.7 * k / case["members"]   # from the full size down to about a third of it
            b = _basin(max(24, int(case["nx"] * f)), max(20, int(case["ny"] * f)), max(6, int(case["layers"] * f)), rng)
            dirs.append(synth.write_run(b, f"{root}/m{k}"))
        ens = Ensemble(dirs, autotune=True)
    ens.step(2)   # start-up, and the step that captures the graph
    return {"ens": ens, "steps": case["steps"], "frames": [_outputs_of(r, {}) for r in ens.runs],
            "zeta": [_pinned(r.lm1, torch.float64) for r in ens.runs]}


def _run_ensemble(st):
    st["ens"].step(st["steps"])
    return [_read(r, f, z) for r, f, z in zip(st["ens"].runs, st["frames"], st["zeta"])]


def _zeta_system(case, rng):
    """SolverSparse's five Purdue columns on a lake's wet cells, and a smooth solution of them."""
    nx, ny = case["nx"], case["ny"]
    depth = synth.random_bathymetry(nx, ny, 1000 * nx + ny, corr=min(20.0, min(nx, ny) / 8.0))
    wet = depth > 0
    lm = int(wet.sum())
    idx = np.zeros((nx + 2, ny + 2), dtype=np.int64)
    idx[1:-1, 1:-1][wet] = np.arange(1, lm + 1)
    dep = np.zeros((nx + 2, ny + 2))
    dep[1:-1, 1:-1] = np.where(wet, depth, 0.0)
    scale = case["ratio"] * rng.uniform(0.9, 1.1) / 4.0 / 60.0
    cx = scale * np.minimum(dep[:-1], dep[1:]) * (idx[:-1] > 0) * (idx[1:] > 0)           # east faces
    cy = scale * np.minimum(dep[:, :-1], dep[:, 1:]) * (idx[:, :-1] > 0) * (idx[:, 1:] > 0)
    at = np.nonzero(idx)
    i, j = at
    east, west, north, south = cx[i, j], cx[i - 1, j], cy[i, j], cy[i, j - 1]
    jcoef = np.stack([idx[i, j], idx[i - 1, j], idx[i, j - 1], idx[i, j + 1], idx[i + 1, j]], axis=1).astype(np.int32)
    coef = np.stack([1 + east + west + north + south, -west, -south, -north, -east], axis=1)
    x = np.zeros((nx + 2, ny + 2))
    x[1:-1, 1:-1] = 0.02 * synth.gaussian_field((nx, ny), min(nx, ny) / 6.0, rng)
    x *= idx > 0
    rhs = (coef[:, 0] * x[i, j] + coef[:, 1] * x[i - 1, j] + coef[:, 2] * x[i, j - 1] + coef[:, 3] * x[i, j + 1] +
           coef[:, 4] * x[i + 1, j])
    x0 = x[i, j] + 0.002 * rng.standard_normal(lm)
    return np.asfortranarray(coef), np.asfortranarray(jcoef), rhs, x0, x[i, j].copy()


def _tridiag_system(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    n, m = case["layers"], case["columns"]
    u = lambda: torch.rand(n, m, generator=g, device="cuda", dtype=torch.float64)  # noqa: E731
    a, c = -3.0 * u(), -3.0 * u()      # implicit vertical diffusion: negative off-diagonals
    a[0], c[-1] = 0.0, 0.0
    return a, 1.0 - a - c, c, u() - 0.5, 0.5 + u()


def _net_images(case, seed):
    """Images like the solver's features: smooth residual and increment, depth, the wet mask."""
    rng = np.random.Generator(np.random.PCG64(seed))
    b, h, w = case["batch"], case["height"], case["width"]
    corr = min(8.0, min(h, w) / 8.0)
    f = np.stack([synth.gaussian_field((h, w), corr, rng) for _ in range(4 * b)]).reshape(b, 4, h, w)
    wet = f[:, 3] > -0.5
    img = np.stack([f[:, 0] * wet, f[:, 1] * wet, np.clip(1.0 + 0.6 * f[:, 3], 0.0, 2.0) * wet, wet], axis=-1)
    to = lambda v: torch.from_numpy(np.ascontiguousarray(v, dtype=np.float32)).cuda()  # noqa: E731
    return to(img), to(f[:, 2] * wet), to(wet)


def _net_params(seed):
    """The trained parameters, moved a little by the seed (training starts and ends near them)."""
    rng = np.random.Generator(np.random.PCG64(seed))
    p = learn.load_params()
    return (p * (1.0 + 0.05 * rng.standard_normal(p.size))).astype(np.float32)


def prepare(case, seed):
    kind = case["kind"]
    rng = np.random.Generator(np.random.PCG64(seed))
    if kind == "step":
        return {"kind": kind, **_prepare_step(case, rng)}
    if kind == "ensemble":
        return {"kind": kind, **_prepare_ensemble(case, rng)}
    if kind == "solve":
        coef, jcoef, rhs, x0, _ = _zeta_system(case, rng)
        return {"kind": kind, "system": (coef, jcoef, rhs, x0), "precision": FORMS[case["precision"]][0]}
    if kind == "tridiag":
        t = _tridiag_system(case, seed)
        return {"kind": kind, "in": t, "out": (torch.empty_like(t[0]), torch.empty_like(t[0])), "lib": native.gpu()}
    feat, target, mask = _net_images(case, seed)
    net = learn.Net(case["batch"], case["height"], case["width"], _net_params(seed))
    return {"kind": kind, "net": net, "feat": feat, "target": target, "mask": mask}


# ---------------------------------------------------------------------------- one pass
def run(st):
    kind = st["kind"]
    if kind == "step":
        return _run_step(st)
    if kind == "ensemble":
        return _run_ensemble(st)
    if kind == "solve":
        x, _ = solve_zeta(*st["system"], itmax=4000, precision=st["precision"])
        return x
    if kind == "tridiag":
        n, m = st["in"][0].shape
        p = [C.c_void_p(t.data_ptr()) for t in st["in"] + st["out"]]
        native.check(st["lib"].si3d_gpu_column_tridiag_noalloc(n, m, *p, None))
        return {"ag": st["out"][0], "ar": st["out"][1]}
    net = st["net"]
    out = net.forward(st["feat"])
    if kind == "infer":
        return out
    net.loss_and_grad(st["feat"], st["target"], st["mask"])
    return {"out": out, "loss": net.loss[:1], "grad": net.grad}


# ---------------------------------------------------------------------------- what a pass needs
def _wet(nx, ny, layers, bowl):
    """Wet columns and wet cells of a basin of that size (the generators' averages)."""
    return (0.78 * nx * ny, 0.39 * nx * ny * layers) if bowl else (0.7 * nx * ny, 0.19 * nx * ny * layers)


def _step_bytes(nx, ny, layers, bowl=False, ntr=0, iturb=0):
    """One time step: three fd calls, each followed by a change of time levels.  A call reads 20
    3-D fields (velocities, transports and thicknesses at two levels, temperature, density, eddy
    coefficients, vertical velocity, heat), writes 7, and carries the 4 momentum solutions across
    the zeta solve; a change of levels reads 9 fields and writes 10.  The zeta system is read and
    its solution written once per call."""
    lm, n3 = _wet(nx, ny, layers, bowl)
    cells = 3 * (20 + 7 + 2 * 4 + 19) + ntr * 2 + (3 * 14 if iturb else 0)
    return 8 * (cells * n3 + 3 * 20 * lm)


def work(case):
    kind = case["kind"]
    if kind == "step":
        b = case["steps"] * _step_bytes(case["nx"], case["ny"], case["layers"], case["bowl"], case["ntr"], case["iturb"])
        lm, n3 = _wet(case["nx"], case["ny"], case["layers"], case["bowl"])
        return {"bytes": b + 4 * (5 + case["ntr"]) * n3 + 8 * lm, "flops": case["steps"] * 3 * 250 * n3}
    if kind == "ensemble":
        total, cells = 0.0, 0.0
        for k in range(case["members"]):
            f = 1.0 - 0.7 * k / case["members"]
            size = (case["nx"] * f, case["ny"] * f, case["layers"] * f)
            n3 = _wet(*size, False)[1]
            total += case["steps"] * _step_bytes(*size) + 20 * n3
            cells += n3
        return {"bytes": total, "flops": case["steps"] * 3 * 250 * cells}
    if kind == "solve":
        lm = 0.7 * case["nx"] * case["ny"]
        return {"bytes": lm * (5 * 8 + 5 * 4 + 3 * 8), "flops": 11 * lm}
    if kind == "tridiag":
        n = case["layers"] * case["columns"]
        return {"bytes": 7 * 8 * n, "flops": 13 * n}
    pixels = case["batch"] * case["height"] * case["width"]
    forward = 2 * pixels * 9 * (4 * 32 + 4 * 32 * 32 + 32)
    if kind == "infer":
        return {"bytes": pixels * 5 * 4, "flops": forward}
    return {"bytes": pixels * 7 * 4 + 8 * native.NET_NPARAM, "flops": 3 * forward}


# ---------------------------------------------------------------------------- 64-bit results
def _network64(p, feat):
    """The network in 64 bits: stem, four residual blocks, head, by plain convolutions."""
    x = feat.double().permute(0, 3, 1, 2)

    def conv(x, w, b, cin, cout):
        k = w.reshape(3, 3, cin, cout).permute(3, 2, 0, 1)
        return torch.nn.functional.conv2d(x, k, b, padding=1)

    sizes = [(4, 32)] + [(32, 32)] * 4 + [(32, 1)]
    layers, o = [], 0
    for cin, cout in sizes:
        layers.append((p[o:o + 9 * cin * cout], p[o + 9 * cin * cout:o + 9 * cin * cout + cout], cin, cout))
        o += 9 * cin * cout + cout
    x = torch.relu(conv(x, *layers[0]))
    for l in layers[1:5]:
        x = x + torch.relu(conv(x, *l))
    return conv(x, *layers[5])[:, 0]


def exact(case, seed):
    kind = case["kind"]
    if kind in ("step", "ensemble"):
        return None
    if kind == "solve":
        return _zeta_system(case, np.random.Generator(np.random.PCG64(seed)))[4]
    if kind == "tridiag":
        a, b, c, g, r = _tridiag_system(case, seed)
        den, gs, rs = [b[0]], [g[0]], [r[0]]
        for k in range(1, b.shape[0]):
            m = a[k] / den[-1]
            den.append(b[k] - m * c[k - 1])
            gs.append(g[k] - m * gs[-1])
            rs.append(r[k] - m * rs[-1])
        ag, ar = [gs[-1] / den[-1]], [rs[-1] / den[-1]]
        for k in range(b.shape[0] - 2, -1, -1):
            ag.append((gs[k] - c[k] * ag[-1]) / den[k])
            ar.append((rs[k] - c[k] * ar[-1]) / den[k])
        return {"ag": torch.stack(ag[::-1]), "ar": torch.stack(ar[::-1])}
    feat, target, mask = _net_images(case, seed)
    p = torch.from_numpy(_net_params(seed)).cuda().double()
    if kind == "infer":
        return _network64(p, feat)
    p.requires_grad_(True)
    out = _network64(p, feat)
    m = mask.double()
    loss = (m * (out - target.double()) ** 2).sum() / m.sum()
    loss.backward()
    return {"out": out.detach(), "loss": loss.detach().reshape(1), "grad": p.grad}
