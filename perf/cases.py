"""The calls of this library that its performance is measured on.

Five kinds of work, each through the entry points of the Python host layer on
torch device buffers (host arrays where the call takes host arrays):

  synthesis  MODE s of a control file: the model file's cubes -> MODEL, the
             Stokes synthesis, RSYN1D -> the profile file's payload
  jacobian   synthesis plus the node Jacobian of the columns, what one
             iteration of an inversion asks for
  response   MODE s with WRITE RESPONSE FUNCTION: responses to six parameters
             at every height, in the RF file's payload
  inversion  MODE i: the first iterations of the pixel-wise search from the
             default guess, model cubes and best profiles out
  lm_step    GET_PERTURBATION of a batch of pixels from host arrays, the call
             the Fortran host makes from its own loop
  guess      the warm-start network on a batch of observations
  training   one epoch of the warm-start network, weights out

Shapes are those of the benchmark (C1: 16x16x96, C2: 256x256x128, four lines:
NUMW 384 on 160 heights), of the reference's own test case (one blended region
of 500 points at 5 mA on 256 heights, with a line spread function), of the
inversion's last iterations (a few tens of columns) and ragged ones between.
Atmospheres have the distributions of firtez-dz_b200/atmos.py.
"""
import importlib.util
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _package():
    name = "firtez_dz_b200"
    if name not in sys.modules:
        d = os.path.join(ROOT, "firtez-dz_b200")
        spec = importlib.util.spec_from_file_location(name, os.path.join(d, "__init__.py"),
                                                      submodule_search_locations=[d])
        mod = importlib.util.module_from_spec(spec)
        sys.modules[name] = mod
        spec.loader.exec_module(mod)
    return sys.modules[name]


fz = _package()
from firtez_dz_b200 import v3io, warmstart  # noqa: E402

DEV = "cuda"

# Zeeman components of the database's lines 1..4 (J 2-2, 1-0, 1-1, 5-4)
COMPONENTS = {1: 13, 2: 3, 3: 7, 4: 27}
NET = (896, 1024, 1024, 512, 13)


def listed():
    return [
        # one pixel, as an interactive session or a single fitted profile asks for: latency
        {"name": "synthesis_one_column", "kind": "synthesis", "nx": 1, "ny": 1, "nz": 128, "lines": "two", "nw": 112,
         "he": 1, "lsf": 0.0},
        # C1: a small patch with its gas pressure given
        {"name": "synthesis_16x16", "kind": "synthesis", "nx": 16, "ny": 16, "nz": 96, "lines": "two", "nw": 112,
         "he": 0, "lsf": 0.0},
        # C2: a whole field in hydrostatic equilibrium, the throughput case
        {"name": "synthesis_256x256", "kind": "synthesis", "nx": 256, "ny": 256, "nz": 128, "lines": "two",
         "nw": 112, "he": 1, "lsf": 0.0},
        # the four-line set (visible and infrared) on a taller grid, ragged field
        {"name": "synthesis_four_lines", "kind": "synthesis", "nx": 61, "ny": 67, "nz": 160, "lines": "four",
         "nw": 96, "he": 1, "lsf": 0.0},
        # the reference's test case: a blended region of 500 points on 256 heights, instrument profile on
        {"name": "synthesis_blend_lsf", "kind": "synthesis", "nx": 24, "ny": 21, "nz": 256, "lines": "blend",
         "nw": 500, "he": 0, "lsf": 30.0},
        # the Jacobian of a full pool of an inversion (T 5 nodes, B and v_z 2 each)
        {"name": "jacobian_2048", "kind": "jacobian", "nx": 64, "ny": 32, "nz": 128, "lines": "two", "nw": 112,
         "he": 1, "nt": 5, "nb": 2, "nv": 2},
        # the same for the few pixels that an inversion's last iterations hold
        {"name": "jacobian_77", "kind": "jacobian", "nx": 7, "ny": 11, "nz": 128, "lines": "two", "nw": 112,
         "he": 1, "nt": 5, "nb": 2, "nv": 2},
        # response functions at every height of the small patch
        {"name": "response_16x16", "kind": "response", "nx": 16, "ny": 16, "nz": 96, "lines": "two", "nw": 112,
         "he": 1},
        # the first iterations of an inversion, where every pixel is still in the pool
        {"name": "inversion_64x32", "kind": "inversion", "nx": 64, "ny": 32, "nz": 128, "lines": "two", "nw": 112,
         "he": 1, "nt": 5, "nb": 2, "nv": 2, "maxit": 3},
        # the damped SVD step of a batch, called by a host that keeps its own loop
        {"name": "lm_step_1024", "kind": "lm_step", "npix": 1024, "np": 13, "nfreq": 896},
        # the learned initial guess of a tile of pixels
        {"name": "guess_16384", "kind": "guess", "n": 16384},
        # an epoch of its training
        {"name": "training_16384", "kind": "training", "n": 16384, "batch": 1024},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _field(rng, lo, hi):
    n = _log(rng, lo, hi)
    ny = max(1, int(round(math.sqrt(n) * rng.uniform(0.6, 1.0))))
    return max(1, n // ny), ny


def _grid(rng, nzmax):
    lines = rng.choice(["two", "two", "two", "four", "blend"])
    nw = {"two": rng.randint(31, 160), "four": rng.randint(31, 96), "blend": rng.randint(101, 500)}[lines]
    return lines, nw, rng.randint(48, nzmax)


def draw(rng):
    kind = rng.choice(["synthesis"] * 6 + ["jacobian"] * 4 + ["response", "inversion", "lm_step", "guess"])
    if kind == "synthesis":
        lines, nw, nz = _grid(rng, 256)
        numw = nw * _nreg(lines)
        nx, ny = _field(rng, 1, min(32768, 65536 * 128 * 224 // (nz * numw * (3 if lines == "four" else 1))))
        return {"kind": kind, "nx": nx, "ny": ny, "nz": nz, "lines": lines, "nw": nw, "he": rng.randint(0, 1),
                "lsf": rng.choice([0.0, 0.0, 30.0])}
    if kind == "jacobian":
        lines, nw, nz = _grid(rng, 160)
        nx, ny = _field(rng, 1, 3000)
        return {"kind": kind, "nx": nx, "ny": ny, "nz": nz, "lines": lines, "nw": nw, "he": rng.randint(0, 1),
                "nt": rng.randint(2, 5), "nb": rng.randint(1, 2), "nv": rng.randint(1, 2)}
    if kind == "response":
        nx, ny = _field(rng, 4, 300)
        return {"kind": kind, "nx": nx, "ny": ny, "nz": rng.randint(48, 128), "lines": "two",
                "nw": rng.randint(31, 112), "he": rng.randint(0, 1)}
    if kind == "inversion":
        nx, ny = _field(rng, 16, 2048)
        return {"kind": kind, "nx": nx, "ny": ny, "nz": rng.randint(64, 128), "lines": "two",
                "nw": rng.randint(64, 112), "he": 1, "nt": rng.randint(3, 5), "nb": rng.randint(1, 2),
                "nv": rng.randint(1, 2), "maxit": rng.randint(2, 3)}
    if kind == "lm_step":
        return {"kind": kind, "npix": _log(rng, 16, 1500), "np": rng.randint(4, 16), "nfreq": 4 * rng.randint(60, 240)}
    return {"kind": kind, "n": _log(rng, 100, 20000)}


# ------------------------------------------------------------------ inputs
def _nreg(lines):
    return {"two": 2, "four": 4, "blend": 1}[lines]


def _section(case):
    nw = case["nw"]
    if case["lines"] == "blend":   # both lines in one region that starts 700 mA before the first
        step = 2500.0 / nw
        return "1,2 %d -700.0 %.4f\n" % (nw, step)
    return fz.atmos.lines_section(_nreg(case["lines"]), nw)


def _context(case):
    lines = fz.lines_parse(fz.atmos.line_database_text())
    return fz.Synthesis(lines, fz.regions_from_lines_section(_section(case), lines), nz=case["nz"])


def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    return g


def _model(case, seed):
    """MODEL (npix, 13, nz) with the distributions of atmos.make_columns, drawn on the GPU."""
    n, nz, g = case["nx"] * case["ny"], case["nz"], _gen(seed)
    z = fz.atmos.z_grid(nz)
    cov = 150.0 ** 2 * (np.exp(-0.5 * ((z[:, None] - z[None, :]) / 100.0) ** 2) + 1e-9 * np.eye(nz))
    chol = torch.from_numpy(np.linalg.cholesky(cov)).to(DEV)
    zt = torch.from_numpy(z).to(DEV)
    f64 = {"dtype": torch.float64, "device": DEV, "generator": g}
    t = torch.from_numpy(fz.atmos.mean_temperature(z)).to(DEV)[None, :] + torch.randn((n, nz), **f64) @ chol.T
    t = t.clamp_min(3000.0)
    # ln Pg by the trapezoid rule, 1.2e5 dyn/cm^2 at z = 0
    dlnp = -1.3 * fz.atmos.MAMU * fz.atmos.GRAV / (fz.atmos.KBOL * t) * 1e5
    seg = 0.5 * (dlnp[:, 1:] + dlnp[:, :-1]) * (zt[1:] - zt[:-1])
    lnp = torch.cat([torch.zeros_like(t[:, :1]), seg.cumsum(1)], 1)
    k = int(np.clip(np.searchsorted(z, 0.0) - 1, 0, nz - 2))
    w = -z[k] / (z[k + 1] - z[k])
    pg = 1.2e5 * torch.exp(lnp - ((1 - w) * lnp[:, k] + w * lnp[:, k + 1])[:, None])
    b = torch.rand(n, **f64) * (4000.0 if case["lines"] == "four" else 2500.0)
    cosg = torch.rand(n, **f64) * 2.0 - 1.0
    phi = torch.rand(n, **f64) * math.pi
    v = torch.randn(n, **f64) * 2.0e5
    sing = (1.0 - cosg ** 2).sqrt()
    grad = 1.0 - 0.1 * (zt - zt[0]) / (zt[-1] - zt[0])
    m = torch.zeros((n, 13, nz), dtype=torch.float32, device=DEV)
    m[:, 0], m[:, 1] = t, pg
    for row, a in ((5, b * sing * phi.cos()), (6, b * sing * phi.sin()), (7, b * cosg), (10, v)):
        m[:, row] = a[:, None] * grad
    m[:, 12] = zt
    return m


def _observations(case, ctx, seed):
    """Profiles (nx, ny, NUMW, 4) as a telescope delivers them: two absorption lines of random depth, width and
    Doppler shift, Zeeman signals in the weak-field form, and noise of 1e-3 of the continuum."""
    n, g = case["nx"] * case["ny"], _gen(seed + 7)
    f64 = {"dtype": torch.float64, "device": DEV, "generator": g}
    depth = 0.55 + 0.15 * torch.rand((n, 1), **f64)
    width = 45.0 + 15.0 * torch.rand((n, 1), **f64)
    vel = 2.0 * torch.randn((n, 1), **f64)
    blos = (2.0 * torch.rand((n, 1), **f64) - 1.0) * 1500.0
    btr2 = (torch.rand((n, 1), **f64) * 1200.0) ** 2
    phi2 = 2.0 * math.pi * torch.rand((n, 1), **f64)
    rows = []
    for r, geff in zip(ctx.regions, (1.67, 2.5)):
        x = torch.arange(int(r["numwave"]), dtype=torch.float64, device=DEV) * float(r["dlambda"]) + float(r["wave_ini"])
        u = (x[None, :] - 21.0 * vel) / width
        line = depth * torch.exp(-u * u)
        di = 2.0 * u / width * line
        d2i = (2.0 - 4.0 * u * u) / width ** 2 * line
        zee = 4.67e-13 * 6302.0 ** 2 * 1e3 * geff   # mA per gauss
        lin = -0.25 * zee ** 2 * btr2 * d2i
        rows.append(torch.stack([1.0 - line, lin * phi2.cos(), lin * phi2.sin(), -zee * blos * di], -1))
    st = torch.cat(rows, 1)
    st = st + 1e-3 * torch.randn(st.shape, **f64)
    return st.float().reshape(case["nx"], case["ny"], -1, 4)


def _nodes(case):
    return {1: case["nt"], 4: case["nb"], 5: case["nb"], 6: case["nb"], 7: case["nv"]}


def _weights(seed):
    g = _gen(seed + 3)
    out = []
    for i, o in zip(NET[:-1], NET[1:]):
        out.append(((torch.rand((o, i), device=DEV, generator=g) * 2.0 - 1.0) * math.sqrt(6.0 / (i + o))).flatten())
        out.append(0.1 * torch.randn(o, device=DEV, generator=g))
    return torch.cat(out)


def _net_inputs(case, seed):
    g = _gen(seed)
    x = torch.randn((case["n"], NET[0]), device=DEV, generator=g)
    t = torch.randn((case["n"], NET[-1]), device=DEV, generator=g)
    return x, t


def _lm_inputs(case, seed):
    """Normalised Jacobians with singular values over one and a half decades, residuals and dampings."""
    g = _gen(seed)
    n, p, f = case["npix"], case["np"], case["nfreq"]
    mix = torch.randn((n, p, p), dtype=torch.float64, device=DEV, generator=g)
    q, _ = torch.linalg.qr(mix)
    scale = torch.logspace(0.0, -1.5, p, dtype=torch.float64, device=DEV) * 3.0
    jac = (q * scale[None, None, :]) @ torch.randn((n, p, f), dtype=torch.float64, device=DEV, generator=g)
    diff = torch.randn((n, f), dtype=torch.float64, device=DEV, generator=g)
    lam = 10.0 ** (4.0 * torch.rand(n, dtype=torch.float64, device=DEV, generator=g) - 3.0)
    return jac.float(), diff, lam


def _empty(*shape, dtype=torch.float32):
    return torch.empty(shape, dtype=dtype, device=DEV)


def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case}
    if kind in ("guess", "training"):
        s["net"] = warmstart.MLP(NET, seed=1)
        s["net"].set_params(_weights(seed).cpu().numpy())
        s["x"], s["t"] = _net_inputs(case, seed)
        s["y"] = _empty(case["n"], NET[-1])
        return s
    if kind == "lm_step":
        s["ctx"] = _context({"lines": "two", "nw": 112, "nz": 32})
        s["jac"], s["diff"], s["lam"] = (a.cpu().numpy() for a in _lm_inputs(case, seed))
        return s
    ctx = s["ctx"] = _context(case)
    nx, ny, nz, npix, nw = case["nx"], case["ny"], case["nz"], case["nx"] * case["ny"], ctx.numw
    s["xs"], s["ys"] = np.arange(nx) * 48.0, np.arange(ny) * 48.0
    s["syn"] = _empty(npix, 4, nw, dtype=torch.float64)
    s["stokes"] = _empty(nx, ny, nw, 4)
    s["out"] = _empty(npix, 13, nz)
    s["status"] = _empty(npix, dtype=torch.int32)
    if kind == "inversion":
        s["obs_file"] = _observations(case, ctx, seed)
        s["obs"] = _empty(npix, 4, nw, dtype=torch.float64)
        s["init"] = torch.from_numpy(warmstart.default_models(npix, nz)).to(DEV)
        s["chi2"] = _empty(npix, dtype=torch.float64)
        s["iters"] = _empty(npix, dtype=torch.int32)
        s["cubes"] = _empty(13, nx, ny, nz)
        s["opts"] = fz.LMOpts(maxit=case["maxit"], isigma=1e-3)
        ctx.rf_nodes(_nodes(case))
        return s
    s["cubes"] = v3io.cubes_from_model_device(_model(case, seed), nx, ny, s["xs"], s["ys"])
    s["model"] = _empty(npix, 13, nz)
    if kind == "jacobian":
        s["np"] = ctx.rf_nodes(_nodes(case))
        s["jac"] = _empty(npix, s["np"], 4 * nw)
    elif kind == "response":
        s["rf"] = _empty(npix, 6, nz, 4 * nw)
        s["payload"] = _empty(nx, ny, nz, nw, 4, 6)
    elif case["lsf"]:
        for r in range(_nreg(case["lines"])):
            ctx.lsf_gaussian(r, case["lsf"], 0.0)
    return s


# --------------------------------------------------------------------- run
def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "guess":
        s["net"].forward_device(case["n"], s["x"].data_ptr(), s["y"].data_ptr())
        return s["y"]
    if kind == "training":
        s["net"].train_device(case["n"], s["x"].data_ptr(), s["t"].data_ptr(), batch=case["batch"], epochs=1, lr=1e-3,
                              seed=5)
        return s["net"].get_params()
    if kind == "lm_step":
        return s["ctx"].lm_perturbation(s["jac"], s["diff"], s["lam"])
    ctx, nx, ny = s["ctx"], case["nx"], case["ny"]
    npix, he = nx * ny, bool(case["he"])
    if kind == "inversion":
        v3io.obs_from_stokes_device(s["obs_file"], out=s["obs"])
        ctx.invert_device(npix, s["obs"].data_ptr(), s["init"].data_ptr(), s["out"].data_ptr(), s["chi2"].data_ptr(),
                          s["iters"].data_ptr(), s["status"].data_ptr(), s["syn"].data_ptr(), hydrostatic=he,
                          opts=s["opts"])
        v3io.cubes_from_model_device(s["out"], nx, ny, s["xs"], s["ys"], out=s["cubes"])
        v3io.stokes_from_syn_device(s["syn"], nx, ny, out=s["stokes"])
        return {"cubes": s["cubes"], "stokes": s["stokes"], "iterations": s["iters"], "status": s["status"]}
    v3io.model_from_cubes_device(s["cubes"], out=s["model"])
    if kind == "jacobian":
        ctx.forward_rf_device(s["model"].data_ptr(), npix, s["syn"].data_ptr(), s["jac"].data_ptr(),
                              s["out"].data_ptr(), s["status"].data_ptr(), hydrostatic=he)
        v3io.stokes_from_syn_device(s["syn"], nx, ny, out=s["stokes"])
        return {"jacobian": s["jac"], "stokes": s["stokes"], "model": s["out"], "status": s["status"]}
    if kind == "response":
        ctx.forward_rf_full_device(s["model"].data_ptr(), npix, s["syn"].data_ptr(), s["rf"].data_ptr(),
                                   s["out"].data_ptr(), s["status"].data_ptr(), hydrostatic=he)
        v3io.stokes_from_syn_device(s["syn"], nx, ny, out=s["stokes"])
        v3io.rf_file_layout_device(s["rf"], nx, ny, out=s["payload"])
        return {"rf": s["payload"], "stokes": s["stokes"], "model": s["out"], "status": s["status"]}
    ctx.forward_device(s["model"].data_ptr(), npix, s["syn"].data_ptr(), s["out"].data_ptr(), s["status"].data_ptr(),
                       hydrostatic=he)
    v3io.stokes_from_syn_device(s["syn"], nx, ny, out=s["stokes"])
    return {"stokes": s["stokes"], "model": s["out"], "status": s["status"]}


# -------------------------------------------------------------------- work
def _synth_flops(case):
    """Chemistry chain (9.4e6 FP64 operations per 128 heights in hydrostatic mode, about a fifth of that with Pg
    given) and 145 operations per Zeeman component + 200 per (height, wavelength)."""
    chain = 9.4e6 * case["nz"] / 128 * (1.0 if case["he"] else 0.2)
    ids = {"two": (1, 2), "four": (1, 2, 3, 4), "blend": (1, 2)}[case["lines"]]
    comps = sum(COMPONENTS[i] for i in ids) * case["nw"]
    return chain + case["nz"] * (145.0 * comps + 200.0 * case["nw"] * _nreg(case["lines"]))


def work(case):
    kind = case["kind"]
    if kind in ("guess", "training"):
        w = sum(i * o for i, o in zip(NET[:-1], NET[1:]))
        n = case["n"]
        if kind == "guess":
            return {"bytes": 4.0 * n * (NET[0] + NET[-1]) + 4.0 * w, "flops": 2.0 * n * w}
        return {"bytes": 4.0 * n * (NET[0] + NET[-1]) + 7 * 4.0 * w, "flops": 6.0 * n * w}
    if kind == "lm_step":
        n, p, f = case["npix"], case["np"], case["nfreq"]
        return {"bytes": n * (4.0 * p * f + 8.0 * f + 8.0 * p), "flops": n * (2.0 * f * p * p + 2.0 * f * p + 20.0 * p ** 3)}
    npix, nz, numw = case["nx"] * case["ny"], case["nz"], case["nw"] * _nreg(case["lines"])
    model, prof = 4.0 * 13 * nz, 16.0 * numw
    if kind == "synthesis":
        return {"bytes": npix * (2 * model + prof), "flops": npix * _synth_flops(case)}
    if kind == "inversion":
        its = case["maxit"]
        np_ = case["nt"] + 3 * case["nb"] + case["nv"]
        return {"bytes": npix * (2 * model + 2 * prof),
                "flops": npix * (its * _synth_flops(case) + (its - 1) * (4400.0 * nz * numw + 8.0 * numw * np_ ** 2))}
    if kind == "jacobian":
        np_ = case["nt"] + 3 * case["nb"] + case["nv"]
        return {"bytes": npix * (2 * model + prof + prof * np_), "flops": npix * (_synth_flops(case) + 4400.0 * nz * numw)}
    return {"bytes": npix * (2 * model + prof + 6.0 * nz * prof), "flops": npix * (_synth_flops(case) + 4400.0 * nz * numw)}


# ------------------------------------------------------------------- exact
def exact(case, seed):
    """The damped SVD step and the network in 64 bits.  The synthesis and what
    builds on it have no 64-bit value in plain torch: they rest on the
    library's own tables (partition functions, cross sections, line data)."""
    if case["kind"] == "lm_step":
        jac, diff, lam = _lm_inputs(case, seed)
        j = jac.double()
        h = j @ j.transpose(1, 2)
        a = h + torch.diag_embed(torch.diagonal(h, dim1=1, dim2=2) * lam[:, None])
        g = (j @ diff[:, :, None])[:, :, 0]
        u, w, vt = torch.linalg.svd(a)
        inv = torch.where(w > 1e-4 * w[:, :1], 1.0 / w, torch.zeros_like(w))
        return (vt.transpose(1, 2) @ (inv * (u.transpose(1, 2) @ g[:, :, None])[:, :, 0])[:, :, None])[:, :, 0].cpu()
    if case["kind"] == "guess":
        x, p, o = _net_inputs(case, seed)[0].double(), _weights(seed).double(), 0
        for k, (i, n) in enumerate(zip(NET[:-1], NET[1:])):
            x = x @ p[o:o + i * n].reshape(n, i).T + p[o + i * n:o + i * n + n]
            o += i * n + n
            if k + 2 < len(NET):
                x = torch.nn.functional.gelu(x)
        return x.cpu()
    return None
