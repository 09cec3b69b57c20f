"""Performance cases of the lattice Boltzmann engine.

Each case is one pass of work that a user's program does through the public
entry points (``LBMBox``, ``LBMBatch``, ``LBMServer`` and the C ABI under
them), over the sizes, precisions, boundaries and routes that the engine
offers:

  steps       time steps of one box through the fused ``step``, then the
              populations in the reference's memory order into page-locked
              memory, as a host program that holds var_inc's arrays takes them
  coupled     the same with the upload in front: populations in, steps,
              populations out
  routines    the reference's main loop, one subroutine per call
  prerelax    the density pre-relaxation of a new run
  statistics  the spectra, moments and diagnostics of one output interval
  ensemble    many boxes of uneven sizes in concurrent batches
  serving     a burst of channel solves through the request loop

A case is a dict of plain values; ``listed`` gives the standing ones,
``draw`` more of the same ranges.  The initial velocity is a seeded
solenoidal Gaussian field, E(k) ~ k^4 exp(-2 (k/k0)^2); spheres are placed by
the reference's ``initpartpos`` and released at rest.
"""

from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

from multiphase_flow_codes_gb300 import _capi as capi
from multiphase_flow_codes_gb300 import ensemble, serving
from multiphase_flow_codes_gb300.engine import LBMBatch, LBMBox

FORCING = {"stochastic": capi.LBM_FORCING_STOCHASTIC, "constant": capi.LBM_FORCING_CONSTANT,
           "none": capi.LBM_FORCING_NONE}


def _box_case(name, kind, shape, npart, steps, prec="f64", walls=False, forcing="stochastic",
              rad=4.0, rho=2.5, k0=4.0, u_rms=0.03, watch=False):
    nx, ny, nz = shape
    return {"name": name, "kind": kind, "nx": nx, "ny": ny, "nz": nz, "npart": npart,
            "steps": steps, "prec": prec, "walls": walls, "forcing": forcing, "rad": rad,
            "rho": rho, "k0": k0, "u_rms": u_rms, "watch": watch}


def listed():
    return [
        # the smallest boxes, advanced a step at a time with the spheres read
        # back after each: a member of a small ensemble in FP32 ...
        _box_case("f32_box32_p5_watched", "steps", (32, 32, 32), 5, 10, "f32", rad=3.0, watch=True),
        # ... and the 64^3 configuration with 16 spheres in FP64
        _box_case("f64_box64_p16_watched", "steps", (64, 64, 64), 16, 10, rad=4.5, rho=5.0,
                  watch=True),
        # forced turbulence at 256^3 with 1000 spheres, the largest standing
        # configuration, in both precisions
        _box_case("f64_box256_p1000", "steps", (256, 256, 256), 1000, 30, k0=8.0, u_rms=0.04),
        _box_case("f32_box256_p1000", "steps", (256, 256, 256), 1000, 40, "f32", k0=8.0,
                  u_rms=0.04),
        # channels with walls and spheres: a ragged FP32 grid (nx no multiple
        # of 4, odd ny and nz) and a plain FP64 one
        _box_case("f32_channel_ragged_p150", "steps", (130, 95, 121), 150, 40, "f32", walls=True,
                  forcing="constant", rho=1.0),
        _box_case("f64_channel_p60", "steps", (96, 128, 80), 60, 30, walls=True,
                  forcing="constant", rho=1.0),
        # a decaying single-phase box whose populations go in and out on
        # every coupling interval of a host program
        _box_case("f64_coupled_fluid", "coupled", (150, 120, 100), 0, 20, forcing="none"),
        # the reference's own main loop, subroutine by subroutine
        _box_case("f64_routines_box128_p150", "routines", (128, 128, 128), 150, 8, rho=2.5),
        # the start of every new run: density pre-relaxation (30 iterations)
        _box_case("f64_prerelax_box128", "prerelax", (128, 128, 128), 0, 30),
        # what a run prints at each output interval
        _box_case("f64_statistics_box192", "statistics", (192, 192, 192), 0, 0, k0=8.0),
        # independent boxes of uneven sizes in two concurrent batches
        {"name": "f32_ensemble12", "kind": "ensemble", "boxes": 12, "spec_seed": 3003, "steps": 48},
        # a burst of channel solves through the request loop
        {"name": "f32_serving_burst6", "kind": "serving", "requests": 6, "max_x": 128, "max_y": 96,
         "max_z": 128, "max_part": 120, "steps": 200},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _draw_shape(rng, lo, hi, aligned):
    n = _log_int(rng, lo, hi)
    shape = [max(lo, min(hi, int(n * rng.uniform(0.7, 1.3)))) for _ in range(3)]
    if aligned:
        shape[0] = max(lo, shape[0] // 4 * 4)
    return shape


def draw(rng):
    kind = rng.choices(("steps", "coupled", "routines", "prerelax", "statistics", "ensemble",
                        "serving"), (12, 2, 2, 2, 1, 1, 1))[0]
    if kind == "ensemble":
        return {"kind": kind, "boxes": rng.randrange(4, 13), "spec_seed": rng.randrange(1, 10000),
                "steps": 6 * rng.randrange(4, 9)}
    if kind == "serving":
        return {"kind": kind, "requests": rng.randrange(3, 8), "max_x": 8 * rng.randrange(10, 17),
                "max_y": 8 * rng.randrange(9, 13), "max_z": 8 * rng.randrange(10, 17),
                "max_part": rng.randrange(20, 121), "steps": rng.randrange(100, 201)}
    prec = "f32" if kind == "steps" and rng.random() < 0.5 else "f64"
    hi = {"steps": 200, "coupled": 150, "routines": 128, "prerelax": 128, "statistics": 192}[kind]
    shape = _draw_shape(rng, 32, hi, rng.random() < 0.6)
    N = shape[0] * shape[1] * shape[2]
    walls = kind in ("steps", "coupled") and rng.random() < 0.4
    rad = round(rng.uniform(3.0, 6.0), 2)
    most = int(0.08 * N / (4.0 / 3.0 * math.pi * rad ** 3))
    npart = 0
    if kind in ("steps", "routines") and rng.random() < 0.8:
        npart = min(most, _log_int(rng, 1, 400))
    if walls:
        forcing = "constant"
    elif kind in ("coupled", "prerelax") or (npart == 0 and rng.random() < 0.6):
        forcing = "none"
    else:
        forcing = "stochastic"
    steps = {"statistics": 0, "routines": 6, "prerelax": rng.randrange(10, 31)}.get(
        kind, max(8, min(30, int(1.5e8 / N))))
    c = _box_case("", kind, shape, npart, steps, prec, walls, forcing, rad,
                  1.0 if walls else round(rng.uniform(1.5, 5.0), 2),
                  watch=kind == "steps" and rng.random() < 0.3)
    del c["name"]
    return c


# ---- inputs ---------------------------------------------------------------

def _velocity(nx, ny, nz, k0, u_rms, seed):
    """Seeded solenoidal Gaussian velocity (3, nz, ny, nx) on the GPU."""
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    v = torch.fft.rfftn(torch.randn((3, nz, ny, nx), generator=gen, device="cuda",
                                    dtype=torch.float64), dim=(1, 2, 3))
    k = torch.stack(torch.meshgrid(*[torch.fft.fftfreq(n, 1.0 / n, device="cuda",
                                                       dtype=torch.float64) for n in (nz, ny)],
                                   torch.fft.rfftfreq(nx, 1.0 / nx, device="cuda",
                                                      dtype=torch.float64),
                                   indexing="ij")).flip(0)  # kx, ky, kz
    k2 = (k * k).sum(0)
    k2s = torch.where(k2 == 0, torch.ones_like(k2), k2)
    v = v - k * ((k * v).sum(0) / k2s)
    kk = torch.sqrt(k2)
    v = v * torch.where(k2 == 0, torch.zeros_like(k2), kk * torch.exp(-(kk / k0) ** 2))
    u = torch.fft.irfftn(v, s=(nz, ny, nx), dim=(1, 2, 3))
    u = u - u.mean(dim=(1, 2, 3), keepdim=True)
    return u * (u_rms / torch.sqrt((u * u).sum(0).mean() / 3.0))


def _config(c):
    preset = capi.LBM_PRESET_CHANNEL if c["walls"] else capi.LBM_PRESET_BOX
    cfg = capi.config_init(preset, c["nx"], c["ny"], c["nz"], c["npart"], c["rad"], c["rho"])
    cfg.precision = capi.LBM_PREC_F32 if c["prec"] == "f32" else capi.LBM_PREC_F64
    cfg.forcing = FORCING[c["forcing"]]
    cfg.mrt_type = 1
    return cfg


def _page_locked(n):
    return torch.empty(n, dtype=torch.float64, pin_memory=True)


def _doubles(t):
    return C.cast(C.c_void_p(t.data_ptr()), C.POINTER(C.c_double))


def _check(rc, what):
    if rc != capi.LBM_OK:
        raise capi.LBMError(rc, what)


def _download(box, out):
    """lbm_download_f into a page-locked tensor, as (nz, ny, nx, 19)."""
    _check(capi.lib().lbm_download_f(box.handle, _doubles(out)), "download_f")
    return out.view(box.nz, box.ny, box.nx, 19)


def _prepare_box(c, seed):
    box = LBMBox(_config(c))
    u = _velocity(c["nx"], c["ny"], c["nz"], c["k0"], c["u_rms"], seed)
    box.initpop(*u.cpu().numpy())
    if c["kind"] != "prerelax":
        box.macrovar()
    if c["npart"]:
        box.init_particles(c["npart"], 1 + int(seed) % 1000003)
    box.synchronize()
    return box


def _prepare_ensemble(c, seed):
    boxes = []
    for i, (n, npart, rad, _, _) in enumerate(ensemble.specs(c["boxes"], c["spec_seed"])):
        cfg = capi.config_init(capi.LBM_PRESET_BOX, n, n, n, npart, rad, 2.5)
        cfg.precision = capi.LBM_PREC_F32
        b = LBMBox(cfg)
        b.init_spectral(4.0, 0.03, int(seed) * 64 + i)
        b.macrovar()
        if npart:
            b.init_particles(npart, 1 + (int(seed) * 64 + i) % 1000003)
        boxes.append(b)
    groups = ensemble.split(ensemble.specs(c["boxes"], c["spec_seed"]), 2)
    batches = [LBMBatch([boxes[i] for i in g]) for g in groups]
    streams = [torch.cuda.Stream() for _ in batches]
    for b, s in zip(batches, streams):
        b.autotune(3)
        b.set_stream(s.cuda_stream)
    return {"case": c, "boxes": boxes, "batches": batches, "streams": streams,
            "out": [_page_locked(19 * b.N) for b in boxes]}


def _prepare_serving(c, seed):
    rng = np.random.default_rng(int(seed))
    reqs = []
    for i in range(c["requests"]):
        # sizes spread over the case's range, the same for every seed
        t = (i + 1) / c["requests"]
        x, y, z = (8 * max(8, int(c[k] * s) // 8) for k, s in
                   (("max_x", t), ("max_y", 1.0 - 0.3 * t), ("max_z", 0.5 + 0.5 * t)))
        cap = int(0.1 * x * y * z / (4.0 / 3.0 * math.pi * 4.0 ** 3))
        reqs.append(serving.request(x, y, z, c["steps"] - 10 * i, wall_axis=1,
                                    npart=min(int(c["max_part"] * t), cap),
                                    seed=int(rng.integers(1, 1 << 40)), keep_state=True,
                                    mrt_type=serving.SERVING_MRT))
    return {"case": c, "server": serving.LBMServer(32 << 30), "requests": reqs}


def prepare(case, seed):
    if case["kind"] == "ensemble":
        return _prepare_ensemble(case, seed)
    if case["kind"] == "serving":
        return _prepare_serving(case, seed)
    box = _prepare_box(case, seed)
    state = {"case": case, "box": box}
    if case["kind"] != "statistics":
        state["out"] = _page_locked(19 * box.N)
    if case["kind"] == "coupled":
        state["in"] = _page_locked(19 * box.N)
        _download(box, state["in"])
    return state


# ---- one pass ----------------------------------------------------------------

def _run_serving(state):
    srv = state["server"]
    ids = [srv.submit(r) for r in state["requests"]]
    out = []
    for rid in ids:
        res = srv.wait(rid)
        if res.state != serving.REQ_DONE:
            raise capi.LBMError(res.error, "request failed")
        with srv.take(rid) as box:
            out.append({"summary": np.array(res.summary[:]), "particles": box.get_particles()})
    return out


def _output_interval(stats, rms, diag):
    """statistc's spectra and totals, rmsstat's row and diag's maxima; a row's
    means of zero-mean fields are rounding, so it stays one array."""
    totals = [stats[k] for k in ("energy", "dissipation", "skewness", "flatness", "uprime")]
    rms = dict(rms)
    return {"ek": stats["ek"], "dk": stats["dk"], "totals": np.array(totals), "nf": rms.pop("nf"),
            "rms": np.array(list(rms.values())), "diag": np.array(list(diag.values()))}


def run(state):
    c = state["case"]
    if c["kind"] == "serving":
        return _run_serving(state)
    if c["kind"] == "ensemble":
        for _ in range(c["steps"] // 6):
            for b in state["batches"]:
                b.step(6)
        for b in state["batches"]:
            b.synchronize()
        return [_download(b, o) for b, o in zip(state["boxes"], state["out"])]
    box = state["box"]
    if c["kind"] == "prerelax":
        iters, err = box.prerelax(0.0, c["steps"])
        return {"iterations": iters, "err": err, "f": _download(box, state["out"])}
    if c["kind"] == "statistics":
        box.macrovar()
        return _output_interval(box.statistics(), box.rmsstat(), box.diag())
    if c["kind"] == "coupled":
        _check(capi.lib().lbm_upload_f(box.handle, _doubles(state["in"])), "upload_f")
        box.macrovar()
    if c["kind"] == "routines":
        box.step_unfused(c["steps"])
    elif c["watch"]:
        for _ in range(c["steps"]):
            box.step(1)
            box.get_particles()
    else:
        box.step(c["steps"])
    return {"f": _download(box, state["out"]), "particles": box.get_particles()}


# ---- what a pass cannot do without ---------------------------------------------

def work(case):
    kind = case["kind"]
    if kind == "ensemble":
        sizes = [(s[0] ** 3, case["steps"]) for s in ensemble.specs(case["boxes"], case["spec_seed"])]
        return {"bytes": sum(n * (152.0 * k + 19 * 8) for n, k in sizes),
                "flops": sum(300.0 * n * k for n, k in sizes)}
    if kind == "serving":
        st = []
        for i in range(case["requests"]):
            t = (i + 1) / case["requests"]
            x, y, z = (8 * max(8, int(case[k] * s) // 8) for k, s in
                       (("max_x", t), ("max_y", 1.0 - 0.3 * t), ("max_z", 0.5 + 0.5 * t)))
            st.append(x * y * z * (case["steps"] - 10 * i))
        return {"bytes": 152.0 * sum(st), "flops": 300.0 * sum(st)}
    N = case["nx"] * case["ny"] * case["nz"]
    es = 8 if case["prec"] == "f64" else 4
    if kind == "statistics":
        # populations to velocity, the three velocity components and their
        # derivative and vorticity fields
        flops = 8 * 2.5 * N * math.log2(N)
        return {"bytes": float(N * (19 + 4 + 3 + 3) * es), "flops": flops}
    if kind == "prerelax":
        # an iteration reads and writes the populations and the density and
        # reads the velocity
        return {"bytes": float((case["steps"] + 2) * N * (2 * 19 + 2 + 3) * es + 19 * 8 * N),
                "flops": 300.0 * N * (case["steps"] + 2)}
    ends = {"coupled": 2}.get(kind, 1)
    return {"bytes": float(case["steps"] * 2 * 19 * es * N + ends * 19 * 8 * N),
            "flops": 300.0 * N * case["steps"]}


# ---- the same in plain 64-bit torch ----------------------------------------------

_CX = [0, 1, -1, 0, 0, 0, 0, 1, -1, 1, -1, 1, -1, 1, -1, 0, 0, 0, 0]
_CY = [0, 0, 0, 1, -1, 0, 0, 1, 1, -1, -1, 0, 0, 0, 0, 1, -1, 1, -1]
_CZ = [0, 0, 0, 0, 0, 1, -1, 0, 0, 0, 0, 1, 1, -1, -1, 1, 1, -1, -1]
_W = [1 / 3] + [1 / 18] * 6 + [1 / 36] * 12
_OPP = [0, 2, 1, 4, 3, 6, 5, 10, 9, 8, 7, 14, 13, 12, 11, 18, 17, 16, 15]


class _Fluid:
    """D3Q19 MRT collision with Guo forcing and streaming, FP64 tensors
    (19, nz, ny, nx) of deviations from w_i."""

    def __init__(self, c):
        def t(v):
            return torch.tensor(v, dtype=torch.float64, device="cuda")

        self.c = torch.stack([t(_CX), t(_CY), t(_CZ)])
        self.w = t(_W)
        x, y, z = self.c
        s = x * x + y * y + z * z                     # |c|^2: 0, 1, 2
        face = s == 1
        rows = [torch.ones_like(x), torch.where(s == 0, -30.0, torch.where(face, -11.0, 8.0)),
                torch.where(s == 0, 12.0, torch.where(face, -4.0, 1.0)), x, y, z]
        rows += [torch.where(face, -4.0 * a, a) for a in (x, y, z)]
        rows += [3 * x * x - s]
        rows += [torch.where(face, -2.0, 1.0) * (3 * x * x - s), y * y - z * z]
        rows += [torch.where(face, -2.0, 1.0) * (y * y - z * z), x * y, y * z, x * z]
        rows += [x * (y * y - z * z), y * (z * z - x * x), z * (x * x - y * y)]
        self.M = torch.stack(rows).to(torch.float64)
        self.Minv = self.M.T / (self.M * self.M).sum(1)
        s9 = 1.0 / (3.0 * 0.0036 + 0.5)
        self.rates = t([1.19, 1.4, 1.2, 1.2, 1.2, s9, 1.4, s9, 1.4, s9, s9, s9, 1.98, 1.98, 1.98])
        self.walls = c["walls"]
        self.F = torch.zeros(3, dtype=torch.float64, device="cuda")
        if c["forcing"] == "constant":
            ustar = 2.0 * 180.0 * 0.0036 / c["nx"]
            self.F[1] = 2.0 * ustar * ustar / c["nx"]

    def feq(self, u):
        cu = torch.einsum("aq,azyx->qzyx", self.c, u)
        return self.w.view(-1, 1, 1, 1) * (3.0 * cu + 4.5 * cu * cu - 1.5 * (u * u).sum(0))

    def macro(self, f):
        return f.sum(0), torch.einsum("aq,qzyx->azyx", self.c, f) + 0.5 * self.F.view(3, 1, 1, 1)

    def collide(self, f, rho, u):
        cu = torch.einsum("aq,azyx->qzyx", self.c, u)
        cF = (self.c * self.F.view(3, 1)).sum(0).view(-1, 1, 1, 1)
        uF = torch.einsum("azyx,a->zyx", u, self.F)
        half = 0.5 * self.w.view(-1, 1, 1, 1) * (3.0 * cF + 9.0 * cF * cu - 3.0 * uF)
        m = torch.einsum("kq,qzyx->kzyx", self.M, f + half)
        ux, uy, uz = u
        sx, sy, sz = ux * ux, uy * uy, uz * uz
        t1 = sx + sy + sz
        zero = torch.zeros_like(rho)
        eq = torch.stack([-11.0 * rho + 19.0 * t1, -475.0 / 63.0 * t1, -2 / 3 * ux, -2 / 3 * uy,
                          -2 / 3 * uz, 2 * sx - sy - sz, zero, sy - sz, zero, ux * uy, uy * uz,
                          ux * uz, zero, zero, zero])
        # rows: rho, e, eps, j (3), q (3), then the ten stress and third-order moments
        idx = [1, 2, 6, 7, 8, 9, 10, 11, 12, 13, 14, 15, 16, 17, 18]
        m[0], m[3], m[4], m[5] = rho, ux, uy, uz
        m[idx] -= self.rates.view(-1, 1, 1, 1) * (m[idx] - eq)
        return torch.einsum("qk,kzyx->qzyx", self.Minv, m) + half

    def stream(self, f):
        out = torch.empty_like(f)
        for q in range(19):
            out[q] = torch.roll(f[q], (_CZ[q], _CY[q], _CX[q]), (0, 1, 2))
        if self.walls:
            for q in range(19):
                if _CX[q]:
                    edge = 0 if _CX[q] == -1 else -1
                    out[_OPP[q]][:, :, edge] = f[q][:, :, edge]
        return out


def _no_particles():
    return {k: torch.zeros((0, 3), dtype=torch.float64)
            for k in ("ypglb", "wp", "omgp", "fHIp", "flubp", "torqp")}


def _exact_steps(c, u):
    fl = _Fluid(c)
    f = fl.feq(u)
    for _ in range(c["steps"]):
        rho, v = fl.macro(f)
        f = fl.stream(fl.collide(f, rho, v))
    return {"f": f.permute(1, 2, 3, 0).contiguous().cpu(), "particles": _no_particles()}


def _exact_prerelax(c, u):
    fl = _Fluid(dict(c, forcing="none"))
    f, rho, n = fl.feq(u), torch.zeros_like(u[0]), 0
    while True:
        f = fl.stream(fl.collide(f, rho, u))
        old, rho = rho, f.sum(0)
        err = float((rho - old).abs().max())
        if n > c["steps"]:
            break
        n += 1
    return {"iterations": n, "err": err, "f": f.permute(1, 2, 3, 0).contiguous().cpu()}


def _exact_statistics(c, u):
    nx, ny, nz = c["nx"], c["ny"], c["nz"]
    N = nx * ny * nz
    v = torch.fft.rfftn(u, dim=(1, 2, 3)) / N
    ints = []
    for n in (nz, ny):
        k = torch.arange(n, device="cuda", dtype=torch.float64)
        ints.append(torch.where(k <= n // 2, k, k - n))
    ints.append(torch.arange(nx // 2 + 1, device="cuda", dtype=torch.float64))
    kz, ky, kx = torch.meshgrid(*ints, indexing="ij")
    e = (v.real ** 2 + v.imag ** 2).sum(0)
    e = torch.where(kx == 0, 0.5 * e, e)
    d = 2.0 * 0.0036 * (2 * math.pi) ** 2 * ((kx / nx) ** 2 + (ky / ny) ** 2 + (kz / nz) ** 2) * e
    shell = (torch.sqrt(kx * kx + ky * ky + kz * kz) + 0.5).to(torch.int64)
    nek = int(nx / 2 - 1.5)
    ek, dk = (torch.bincount(shell.reshape(-1), a.reshape(-1), minlength=nek + 1)[1:nek + 1]
              for a in (e, d))

    def wave(k, n):
        return torch.where(2 * k == n, torch.zeros_like(k), k) * 1j

    ix, iy, iz = wave(kx, nx), wave(ky.abs(), ny) * ky.sign(), wave(kz.abs(), nz) * kz.sign()

    def back(a):
        return torch.fft.irfftn(a * N, s=(nz, ny, nx), dim=(0, 1, 2))

    wx, wy = back(ix * v[0]), back(iy * v[1])
    m2, m3, m4 = (float(((2 * wx ** p + wy ** p) / 3.0).mean()) for p in (2, 3, 4))
    qq = float(ek.sum())
    stats = {"ek": ek.cpu(), "dk": dk.cpu(), "energy": qq, "dissipation": float(dk.sum()),
             "skewness": m3 / m2 ** 1.5, "flatness": m4 / m2 ** 2, "uprime": math.sqrt(2 * qq / 3)}
    om = [back(iy * v[2] - iz * v[1]), back(iz * v[0] - ix * v[2]), back(ix * v[1] - iy * v[0])]
    um = [float(a.mean()) for a in u]
    ur = [math.sqrt(float(((a - m) ** 2).mean())) for a, m in zip(u, um)]
    omn = [float(a.mean()) for a in om]
    omr = [math.sqrt(float(((a - m) ** 2).mean())) for a, m in zip(om, omn)]

    def norm(a):
        return math.sqrt(sum(x * x for x in a))

    row = [float(N), N / float(nx) ** 3, *um, *ur, norm(ur), norm(um)] + [0.0] * 8
    row += [*omn, *omr, norm(omr) / 2, norm(omn)] + [0.0] * 8 + [norm(omr) ** 2, norm(ur) ** 2]
    diag = {"vmax": math.sqrt(float((u * u).sum(0).max())), "idwp": 0, "wpmax": 0.0, "idomgp": 0,
            "omgpmax": 0.0}
    return _output_interval(stats, dict(zip(LBMBox.RMS_COLUMNS, row)), diag)


def exact(case, seed):
    kind = case["kind"]
    if kind in ("ensemble", "serving", "routines"):
        return None  # moving spheres and the stochastic forcing: no few lines of torch
    if kind in ("steps", "coupled") and (case["npart"] or case["forcing"] == "stochastic"):
        return None
    u = _velocity(case["nx"], case["ny"], case["nz"], case["k0"], case["u_rms"], seed)
    return {"steps": _exact_steps, "coupled": _exact_steps, "prerelax": _exact_prerelax,
            "statistics": _exact_statistics}[kind](case, u)
