"""Performance cases: the work that a user of this framework has it do, through its public entry
points, from one soil column to the 56.6M-cell combined workload.

Kinds ("kind" of a case):
  column    a 1-D infiltration column (b2-gw), the reference scheme with its default CG + SOR,
            adaptive time step: the smallest calls, latency and launches
  section   a 2-D layered section under partial recharge (b3-kirkland), same solver
  ponded    homogeneous loam under a ponded top face (40x40x100 configuration)
  grf       heterogeneous loam with a hydrostatic start, rain and a fixed bottom head
            (256x256x128 configuration)
  layers    sand / loam / clay layers, dry start, rain (768x768x96 combined workload)
  seam      the linear-solver seam: a 7-point system assembled from host triplets and solved
  net       one application of the learned preconditioner's U-Net
  train     loss and parameter gradients of the U-Net on one training pair

A pass of the step kinds is a short scenario, as a calibration or an ensemble runs it again and
again on one handle: the initial head is set, the run starts, `steps` steps, and the head and the
water content are copied into device buffers.
"""
from __future__ import annotations

import ctypes as C
import math
import os

import numpy as np
import torch

from frehg_gb300 import workloads as W
from frehg_gb300.abi import SolverConfig, check, load_library
from frehg_gb300.learned import DEFAULT_WEIGHTS, UNet
from frehg_gb300.linear import makeLinearSolver
from frehg_gb300.re_solver import Grid, ReSolver, SoilMap

DEV = "cuda"


# ---------------------------------------------------------------------------------------------
# the cases

def step_case(name, kind, scheme, solver, nx, ny, nz, steps):
    return dict(name=name, kind=kind, scheme=scheme, solver=solver, nx=nx, ny=ny, nz=nz,
                steps=steps)


def listed():
    return [
        # one vertical column, as in the b2-gw benchmark: thousands of tiny adaptive steps
        step_case("column-sor", "column", "pca", "sor", 1, 1, 100, 20),
        # the b3-kirkland section: 1,500 cells, two soils, partial recharge
        step_case("section-sor", "section", "pca", "sor", 50, 1, 30, 20),
        # the 40x40x100 configuration with the reference scheme and Jacobi-PCG
        step_case("ponded-pca-jacobi", "ponded", "pca", "jacobi", 40, 40, 100, 4),
        # a reference user's setup at field-plot size: default CG + SOR, ragged grid
        step_case("ponded-pca-sor", "ponded", "pca", "sor", 90, 75, 60, 1),
        # the 40x40x100 configuration with the Picard scheme and the mixed line solver
        step_case("ponded-picard-line", "ponded", "picard", "line", 40, 40, 100, 3),
        # heterogeneous soil in plain FP64 (the path results are checked against), ragged grid
        step_case("grf-picard-jacobi", "grf", "picard", "jacobi", 101, 77, 53, 2),
        # the 256x256x128 configuration with the recommended solver
        step_case("grf-picard-line", "grf", "picard", "line", 256, 256, 128, 2),
        # a catchment-sized ragged grid of the combined workload
        step_case("layers-picard-line-ragged", "layers", "picard", "line", 203, 149, 96, 3),
        # the combined workload at full size
        step_case("layers-picard-line", "layers", "picard", "line", 768, 768, 96, 3),
        # a host code's own assembly through the linear seam
        dict(name="seam-jacobi", kind="seam", solver="jacobi", nx=32, ny=32, nz=32),
        # network application at the size the preconditioner is used on
        dict(name="net-forward", kind="net", nx=256, ny=256, nz=128),
        # a training pair of the published recipe's shape
        dict(name="train-gradient", kind="train", nx=128, ny=128, nz=64),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["column", "section", "ponded", "ponded", "grf", "layers", "seam", "net",
                       "train"])
    if kind == "column":
        return dict(kind=kind, scheme="pca", solver=rng.choice(["sor", "jacobi"]), nx=1, ny=1,
                    nz=rng.randint(40, 200), steps=rng.randint(8, 20))
    if kind == "section":
        return dict(kind=kind, scheme="pca", solver=rng.choice(["sor", "jacobi"]),
                    nx=rng.randint(30, 120), ny=1, nz=rng.randint(24, 60),
                    steps=rng.randint(5, 20))
    if kind == "ponded":
        scheme = rng.choice(["pca", "picard"])
        solver = rng.choice(["sor", "jacobi"] if scheme == "pca" else ["line", "jacobi"])
        return dict(kind=kind, scheme=scheme, solver=solver, nx=_log(rng, 8, 120),
                    ny=_log(rng, 8, 120), nz=rng.randint(30, 100), steps=rng.randint(1, 3))
    if kind == "grf":
        solver = rng.choice(["line", "jacobi"])
        top = 256 if solver == "line" else 110
        return dict(kind=kind, scheme="picard", solver=solver, nx=_log(rng, 40, top),
                    ny=_log(rng, 40, top), nz=rng.randint(40, 128), steps=rng.randint(1, 2))
    if kind == "layers":
        return dict(kind=kind, scheme="picard", solver="line", nx=_log(rng, 48, 600),
                    ny=_log(rng, 48, 600), nz=96, steps=rng.randint(1, 3))
    if kind == "seam":
        return dict(kind=kind, solver=rng.choice(["jacobi", "sor"]), nx=_log(rng, 4, 40),
                    ny=_log(rng, 4, 40), nz=_log(rng, 4, 40))
    if kind == "net":
        return dict(kind=kind, nx=4 * _log(rng, 8, 64), ny=4 * _log(rng, 8, 64),
                    nz=4 * _log(rng, 6, 32))
    return dict(kind=kind, nx=4 * _log(rng, 4, 32), ny=4 * _log(rng, 4, 32),
                nz=4 * _log(rng, 4, 24))


# ---------------------------------------------------------------------------------------------
# inputs

def _gen(seed, salt=0):
    return torch.Generator(device=DEV).manual_seed(int(seed) * 1000003 + salt)


def _grf(shape, corr, seed, salt):
    """standard-normal field with exponential covariance (circulant embedding, as grf.py)"""
    lag = []
    for n, l in zip(shape, corr):
        k = torch.arange(n, device=DEV, dtype=torch.float64)
        lag.append(torch.minimum(k, n - k) / l)
    r2 = lag[0][:, None, None] ** 2 + lag[1][None, :, None] ** 2 + lag[2][None, None, :] ** 2
    amp = torch.fft.rfftn(torch.exp(-torch.sqrt(r2))).real.clamp_min(0.0).sqrt()
    noise = torch.randn(shape, device=DEV, dtype=torch.float64, generator=_gen(seed, salt))
    f = torch.fft.irfftn(torch.fft.rfftn(noise) * amp, s=shape)
    f -= f.mean()
    return f / f.std()


SECTION = dict(alpha=2.8, n=2.239, theta_s=0.3658, theta_r=0.029, Ks=6.26e-5)
SECTION_LENS = dict(alpha=1.04, n=1.395, theta_s=0.4686, theta_r=0.106, Ks=1.52e-6)


def _setup(case, seed):
    """What defines a run: ReParams, soil (classes and ids, Ks, alpha), initial head, top flux;
    device tensors of shape (nz, ny, nx)."""
    kind, nx, ny, nz = case["kind"], case["nx"], case["ny"], case["nz"]
    shape = (nz, ny, nx)
    rng = np.random.Generator(np.random.PCG64(seed))
    d = dict(classes=None, ids=None, Ks=None, alpha=None, qtop=None)
    if kind == "column":
        p = W.b2gw_column().params
        p.botz = -p.dz * nz
        p.dt = float(rng.uniform(0.5, 2.0))
        # h(theta) of a water content near the benchmark's 0.033
        s = p.soil
        th = 0.033 * rng.uniform(1.0, 1.5)
        m = 1.0 - 1.0 / s.n
        h0 = -((((s.theta_s - s.theta_r) / (th - s.theta_r)) ** (1.0 / m) - 1.0)
               ** (1.0 / s.n)) / s.alpha
        d["h"] = torch.full(shape, h0, device=DEV, dtype=torch.float64)
    elif kind == "section":
        p = W.b2gw_column().params
        p.soil = W.soil(SECTION)
        p.soil.air_entry = 0.0
        p.dx = p.dy = p.dz = 0.1
        p.botz = -0.1 * nz
        p.dt, p.dt_min, p.dt_max = 5.0, 0.01, 10.0
        p.use_full3d = 1
        p.bc_type = (C.c_int32 * 6)(0, 0, 0, 0, 0, 2)
        lens = W.soil(SECTION_LENS)
        lens.air_entry = 0.0
        ids = torch.ones(shape, device=DEV, dtype=torch.int32)
        ids[:nz // 3, :, nx // 5:nx - nx // 5] = 0
        ids[2 * nz // 3:] = 0
        d["classes"], d["ids"] = [p.soil.copy(), lens], ids
        q = np.zeros((ny, nx))
        q[:, nx // 5:nx - nx // 5] = -5.7e-6 * rng.uniform(0.8, 1.2)
        d["qtop"] = q
        d["h"] = -500.0 * (1.0 + 0.02 * torch.rand(shape, device=DEV, dtype=torch.float64,
                                                   generator=_gen(seed, 1)))
    elif kind == "ponded":
        p = W.config0(case["scheme"], nx=4, ny=4, nz=nz).params
        d["h"] = -2.0 + 0.05 * _grf(shape, (4.0, 8.0, 8.0), seed, 1)
    elif kind == "grf":
        w = W.config1(case["scheme"], nx=4, ny=4, nz=nz)
        p = w.params
        p.picard_dt_adapt = 1  # a step that fails is retried at half dt; dt stays 60 s
        xk = _grf(shape, (4.0, 8.0, 8.0), seed, 1)
        xa = _grf(shape, (4.0, 8.0, 8.0), seed, 2)
        d["Ks"] = W.LOAM["Ks"] * torch.exp(xk)
        d["alpha"] = W.LOAM["alpha"] * torch.exp(0.3 * (0.7 * xk + math.sqrt(0.51) * xa))
        # the water table at 0.625 of the depth (4 m at 6.4 m)
        zc = (torch.arange(nz, device=DEV, dtype=torch.float64) + 0.5) * p.dz
        d["h"] = (zc - 0.625 * nz * p.dz)[:, None, None].expand(shape).contiguous()
        p.hbot = 0.375 * nz * p.dz
    else:
        p = W.config4(nx=4, ny=4, nz=nz).params
        k1 = int(rng.integers(nz // 6, nz // 3))
        k2 = int(rng.integers(nz // 2, (5 * nz) // 6))
        ids = torch.zeros(shape, device=DEV, dtype=torch.int32)
        ids[k1:k2] = 1
        ids[k2:] = 2
        base = torch.tensor([W.SAND["Ks"], W.LOAM["Ks"], W.CLAY["Ks"]], device=DEV,
                            dtype=torch.float64)
        d["classes"], d["ids"] = [W.soil(W.SAND), W.soil(W.LOAM), W.soil(W.CLAY)], ids
        d["Ks"] = base[ids.long()] * torch.exp(1.5 * _grf(shape, (4.0, 8.0, 8.0), seed, 1))
        d["h"] = torch.full(shape, -5.0, device=DEV, dtype=torch.float64)
    d["p"] = p
    return d


def _solver(case):
    if case["solver"] == "line":
        return SolverConfig("cg", "line", rtol=1e-12, max_it=20000, precision=1, ir_rtol=1e-12)
    rtol = 1e-10 if case["kind"] in ("column", "section") else 1e-12
    return SolverConfig("cg", case["solver"], rtol=rtol, max_it=20000)


def _prepare_step(case, seed):
    d = _setup(case, seed)
    p, nx, ny, nz = d["p"], case["nx"], case["ny"], case["nz"]
    g = ReSolver(Grid(nx, ny, nz, p.dx, p.dy, p.dz), p)
    if d["classes"] is not None:
        m = SoilMap()
        m.setClasses(d["classes"])
        m.setClassIndex3D(nx, ny, nz, d["ids"].cpu().numpy())
        g.set_soil_map(m)
    if d["Ks"] is not None:
        g.set_cell_fields(d["Ks"].cpu().numpy(),
                          None if d["alpha"] is None else d["alpha"].cpu().numpy())
    g.initialize_geometry()
    g.attach_solver(_solver(case))
    if d["qtop"] is not None:
        g.set_top_flux_field(d["qtop"])
    h0 = torch.empty((nz, ny, nx), dtype=torch.float64, pin_memory=True)
    h0.copy_(d["h"])
    g.set_initial_head(h0.numpy())
    g.finalize_initial_state()
    out = {k: torch.empty((nz, ny, nx), dtype=torch.float64, device=DEV) for k in ("h", "wc")}
    return dict(kind="step", g=g, h0=h0, dt=p.dt, steps=case["steps"], out=out)


def _seam_system(case, seed):
    """random symmetric diagonally dominant 7-point system: diagonal and the couplings of each
    cell with its next neighbour along k, i, j (arrays (ny, nx, nz), k fastest), and b"""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    rng = np.random.default_rng(seed)
    up = [-rng.uniform(0.1, 2.0, (ny, nx, nz)) for _ in range(3)]
    up[0][:, :, -1] = 0.0
    up[1][:, -1, :] = 0.0
    up[2][-1, :, :] = 0.0
    diag = rng.uniform(1e-3, 0.5, (ny, nx, nz))
    for a, ax in zip(up, (2, 1, 0)):
        diag -= a + np.roll(a, 1, axis=ax)  # the wrapped-around entries are zero
    return diag, up, rng.standard_normal(nx * ny * nz)


def _prepare_seam(case, seed):
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    diag, up, b = _seam_system(case, seed)
    n = nx * ny * nz
    r = np.arange(n, dtype=np.int32)
    rows, cols, vals = [r], [r], [diag.ravel()]
    for a, off in zip(up, (1, nz, nz * nx)):
        q = np.flatnonzero(a.ravel() != 0.0).astype(np.int32)
        v = a.ravel()[q]
        rows += [q, q + off]
        cols += [q + off, q]
        vals += [v, v]
    s = makeLinearSolver("gb300", SolverConfig("cg", case["solver"], rtol=1e-12, max_it=20000))
    return dict(kind="seam", s=s, A=s.createSystem(nx, ny, nz),
                rows=np.concatenate(rows).astype(np.int32),
                cols=np.concatenate(cols).astype(np.int32), vals=np.concatenate(vals), b=b,
                x=np.empty(n))


def _net_inputs(case, seed):
    shape = (case["nz"], case["ny"], case["nx"])
    g = _gen(seed, 7)
    r = torch.randn(shape, device=DEV, generator=g)
    lnk = _grf(shape, (4.0, 8.0, 8.0), seed, 8).mul(1.5).sub(12.0).float()
    cap = torch.rand(shape, device=DEV, generator=g).mul(0.2)
    tgt = torch.randn(shape, device=DEV, generator=g).mul(0.5).add(0.5 * r)
    return r, lnk, cap, tgt


def prepare(case, seed):
    if case["kind"] == "seam":
        return _prepare_seam(case, seed)
    if case["kind"] in ("net", "train"):
        net = UNet(0)
        assert os.path.exists(DEFAULT_WEIGHTS)
        net.load(DEFAULT_WEIGHTS)
        r, lnk, cap, tgt = _net_inputs(case, seed)
        return dict(kind=case["kind"], net=net, dims=(case["nx"], case["ny"], case["nz"]), r=r,
                    lnk=lnk, cap=cap, tgt=tgt, y=torch.empty_like(r),
                    grad=np.empty(net.nparam, dtype=np.float32))
    return _prepare_step(case, seed)


def run(s):
    if s["kind"] == "step":
        g = s["g"]
        g.set_initial_head(s["h0"].numpy())
        g.prime_adaptive_dt(s["dt"])
        g.finalize_initial_state()
        g.advance_steps(s["steps"])
        for k, t in s["out"].items():
            g.interior_to_device(k, t.data_ptr())
        return s["out"]
    if s["kind"] == "seam":
        A = s["A"]
        A.zeroEntries()
        A.addCOO(s["rows"], s["cols"], s["vals"])
        A.endAssembly()
        return {"x": s["s"].solve(A, s["b"], s["x"])}
    lib, net = load_library(), s["net"]
    st = torch.cuda.current_stream().cuda_stream
    ptr = [s[k].data_ptr() for k in ("r", "lnk", "cap")]
    if s["kind"] == "net":
        check(lib.frehg_unet_forward(net.handle, *s["dims"], *ptr, s["y"].data_ptr(), st),
              "forward")
        return {"y": s["y"]}
    loss = C.c_double()
    check(lib.frehg_unet_loss_grad(net.handle, *s["dims"], *ptr, s["tgt"].data_ptr(),
                                   C.byref(loss), s["grad"].ctypes.data_as(C.POINTER(C.c_float)),
                                   st), "loss_grad")
    return {"loss": loss.value, "grad": s["grad"]}


def work(case):
    """Compulsory traffic and operations of one pass.  Steps: per step the head and the water
    content read and written and the per-cell soil read once, and one evaluation of the
    constitutive relations and of the six face fluxes per cell (the numbers of Picard and Krylov
    iterations are the method's own).  Network: its input and output fields and its
    multiply-adds (the gradients: three times the forward's)."""
    n = float(case["nx"]) * case["ny"] * case["nz"]
    kind = case["kind"]
    if kind in ("net", "train"):
        f = UNet.flops(case["nx"], case["ny"], case["nz"])
        return {"bytes": 16.0 * n, "flops": f} if kind == "net" else \
            {"bytes": 16.0 * n + 4.0 * 354145, "flops": 3.0 * f}
    if kind == "seam":
        return {"bytes": n * (7 * 16 + 16), "flops": 14.0 * n}
    soil = {"grf": 16.0, "layers": 9.0, "section": 1.0}.get(kind, 0.0)
    return {"bytes": case["steps"] * n * (32.0 + soil), "flops": case["steps"] * n * 150.0}


# ---------------------------------------------------------------------------------------------
# the same results in 64 bits, in plain torch

def _up(a, ax):
    """a of the next cell along ax, 0 beyond the last"""
    return torch.cat([a.narrow(ax, 1, a.shape[ax] - 1), torch.zeros_like(a.narrow(ax, 0, 1))], ax)


def _dn(a, ax):
    return torch.cat([torch.zeros_like(a.narrow(ax, 0, 1)), a.narrow(ax, 0, a.shape[ax] - 1)], ax)


def _cg(d, off, b, rtol=1e-14, max_it=20000):
    """Jacobi-PCG for diag d and couplings off[ax] with the next cell along ax"""
    x, r = torch.zeros_like(b), b.clone()
    z = r / d
    p = z.clone()
    rz = (r * z).sum()
    stop = rtol * float(z.norm())
    lo = [_dn(o, ax) for ax, o in enumerate(off)]
    for it in range(max_it):
        if float(z.norm()) <= stop:
            break
        w = d * p
        for ax in range(3):
            w += off[ax] * _up(p, ax) + lo[ax] * _dn(p, ax)
        a = rz / (p * w).sum()
        x += a * p
        r -= a * w
        z = r / d
        rz, old = (r * z).sum(), rz
        p = z + (rz / old) * p
    return x


class _Soil:
    """per-cell van Genuchten parameters and relations"""

    def __init__(self, d, shape):
        p = d["p"]
        cl = d["classes"] or [p.soil]
        ids = d["ids"].long() if d["ids"] is not None else torch.zeros(shape, device=DEV).long()

        def field(f):
            return torch.tensor([float(getattr(c, f)) for c in cl], device=DEV,
                                dtype=torch.float64)[ids]

        self.alpha = d["alpha"] if d["alpha"] is not None else field("alpha")
        self.n, self.ths, self.thr = field("n"), field("theta_s"), field("theta_r")
        self.Ss, self.aev = field("Ss"), field("air_entry")
        self.K = [d["Ks"]] * 3 if d["Ks"] is not None else \
            [field("Ks_z"), field("Ks_y"), field("Ks_x")]
        self.m = 1.0 - 1.0 / self.n

    def se(self, h):
        t = (self.alpha * h).abs() ** self.n
        return t, (1.0 + t) ** -self.m

    def theta(self, h, aev):
        _, se = self.se(h)
        return torch.where(h > aev, self.ths, self.thr + (self.ths - self.thr) * se)

    def kr(self, h):
        t, se = self.se(h)
        q = torch.expm1(-self.m * torch.log1p(1.0 / t))
        return torch.where(h > 0, torch.ones_like(h), torch.sqrt(se) * q * q).clamp_max(1.0)

    def cap(self, h):
        t, se = self.se(h)
        ah = (self.alpha * h).abs()
        c = self.alpha * self.n * self.m * (self.ths - self.thr) * t * se / (ah * (1.0 + t))
        return torch.where((h > 0) | (ah == 0), torch.zeros_like(h), c)

    def head(self, wc):
        th = torch.maximum(wc, self.thr + 1e-7)
        x = torch.expm1(torch.log((self.ths - self.thr) / (th - self.thr)) / self.m)
        return torch.where(th < self.ths, -(x ** (1.0 / self.n)) / self.alpha,
                           torch.zeros_like(wc))

    def dkdwc(self, wc):
        near = (wc > 0.9999 * self.ths) & (wc < self.ths)
        th = torch.where(near, 0.9999 * self.ths, wc)
        se = (th - self.thr) / (self.ths - self.thr)
        a = 1.0 - se ** (1.0 / self.m)
        t0 = a ** self.m
        t1 = 0.5 * self.K[0] * se ** -0.5 * (1.0 - t0) ** 2
        t2 = 2.0 * self.K[0] * se ** ((2.0 - self.m) / (2.0 * self.m)) * (1.0 - t0) * \
            a ** (self.m - 1.0)
        return (t1 + t2) / (self.ths - self.thr)


def _faces(K):
    """arithmetic face means along each axis (z, y, x), 0 beyond the last cell"""
    out = []
    for ax in range(3):
        f = 0.5 * (K[ax] + _up(K[ax], ax))
        f.narrow(ax, K[ax].shape[ax] - 1, 1).zero_()
        out.append(f)
    return out


def _exact_picard(d, shape, steps):
    p, s = d["p"], _Soil(d, shape)
    dx, dy, dz = p.dx, p.dy, p.dz
    V, Az = dx * dy * dz, dx * dy
    g = [Az / dz, dx * dz / dy, dy * dz / dx]
    h = d["h"].clone()
    wc = s.theta(h, s.aev)
    dt, time = p.dt, 0.0

    def flux(h, K, with_t):
        kf = _faces(K)
        q, ts = torch.zeros_like(h), torch.zeros_like(h)
        for ax in range(3):
            t = kf[ax] * g[ax]
            f = t * (_up(h, ax) - h)
            if ax == 0:
                f = f - Az * kf[0]
            f.narrow(ax, h.shape[ax] - 1, 1).zero_()
            q += f - _dn(f, ax)
            ts += t + _dn(t, ax)
        Kt, ht = s.K[0][0], h[0]
        if p.bc_type[5] == 1:
            t = Kt * 2 * g[0]
            q[0] += t * (p.htop - ht) + Az * Kt
            ts[0] += t
        elif p.bc_type[5] == 2:
            rain = p.rain_rate != 0.0
            qv = (p.rain_rate if time < p.rain_until else 0.0) if rain else p.qtop
            qin = torch.full_like(ht, -qv * Az)
            tD = Kt * 2 * g[0]
            fD = -tD * ht + Az * Kt
            lim = (qin > 0) & (fD < qin) if rain else torch.zeros_like(ht, dtype=torch.bool)
            q[0] += torch.where(lim, fD, qin)
            ts[0] += torch.where(lim, tD, torch.zeros_like(tD))
        Kb, hb = K[0][-1], h[-1]
        if p.bc_type[4] == 1:
            kb = s.K[0] * s.kr(torch.full_like(h, p.hbot))
            k2 = 0.5 * (Kb + kb[-1])
            t = k2 * 2 * g[0]
            q[-1] += t * (p.hbot - hb) - Az * k2
            ts[-1] += t
        elif p.bc_type[4] == 3:
            q[-1] -= Kb * Az
        return q, ts, [k * c for k, c in zip(kf, g)]

    for _ in range(steps):
        hn, wn = h, wc
        st = s.Ss * wn / s.ths
        while True:
            h, done = hn.clone(), False
            for it in range(p.picard_max_it):
                kr = s.kr(h)
                K = [k * kr for k in s.K]
                q, ts, tf = flux(h, K, True)
                rhs = -(V * (s.theta(h, torch.zeros_like(h)) - wn) + V * st * (h - hn) - dt * q)
                dl = _cg(V * (s.cap(h) + st) + dt * ts, [-dt * t for t in tf], rhs)
                if p.picard_dh_max > 0:
                    dl = dl.clamp(-p.picard_dh_max, p.picard_dh_max)
                h = h + dl
                if float(dl.abs().max()) < p.picard_tol:
                    done = True
                    break
            if done or not p.picard_dt_adapt or dt <= p.dt_min / 16:
                break
            dt = max(0.5 * dt, p.dt_min / 16)
        q, _, _ = flux(h, K, False)
        wc = wn + (dt * q - V * st * (h - hn)) / V
        time += dt
        its = it + 1
        if p.picard_dt_adapt:
            if its <= 3:
                dt = min(dt * 1.25, p.dt_max)
            elif its >= 8:
                dt = max(dt * 0.7, min(dt, p.dt_min))
    return {"h": h, "wc": wc}


def _exact_pca(d, shape, steps):
    p, s = d["p"], _Soil(d, shape)
    nz = shape[0]
    dx, dy, dz = p.dx, p.dy, p.dz
    A = [dx * dy, dx * dz, dy * dz]
    L = [dz, dy, dx]
    V = dx * dy * dz
    h = d["h"].clone()
    wc = s.theta(h, s.aev)
    dt = dtn = p.dt
    qtop = torch.as_tensor(d["qtop"], device=DEV) if d["qtop"] is not None else None
    top_sat = p.bc_type[5] == 1 and p.htop >= 0.0
    false = torch.zeros(shape, device=DEV, dtype=torch.bool)
    for step in range(steps):
        hn, wn = h, wc
        K = [k * s.kr(hn) for k in s.K]
        kf = _faces(K)
        store = s.cap(hn) + s.Ss * wn / s.ths
        off = [-dt * kf[ax] * A[ax] / L[ax] for ax in range(3)]
        diag = store * V
        for ax in range(3):
            diag = diag - off[ax] - _dn(off[ax], ax)
        rhs = store * hn * V - dt * A[0] * (kf[0] - _dn(kf[0], 0))
        if p.bc_type[5] == 1:
            t = s.K[0][0] * dt * 2 * A[0] / dz
            diag[0] += t
            rhs[0] += dt * A[0] * s.K[0][0] + t * p.htop
        else:
            rhs[0] -= dt * A[0] * qtop
        h = _cg(diag, off, rhs)
        kr = s.kr(h)
        K = [k * kr for k in s.K]
        kf = _faces(K)
        wch = s.theta(h, s.aev)
        qp, qm = [], []
        for ax in range(3):
            grad = (_up(h, ax) - h) / L[ax] - (1.0 if ax == 0 else 0.0)
            f = A[ax] * kf[ax] * grad
            f.narrow(ax, f.shape[ax] - 1, 1).zero_()
            qp.append(f)
            qm.append(_dn(f, ax))
        qm[0][0] = qtop * A[0] if p.bc_type[5] == 2 else \
            A[0] * s.K[0][0] * ((h[0] - p.htop) * (2.0 / dz) - 1.0)
        wc = (wn * V + dt * sum(a - b for a, b in zip(qp, qm))) / \
            (V * (1.0 + s.Ss * (h - hn) / s.ths))
        old, wsat = wc >= s.ths, wch >= s.ths
        oy, ox = kf[1] != 0, kf[2] != 0
        succ = _up(old, 0) | (oy & _up(old, 1)) | (ox & _up(old, 2))
        if step > 0:
            succ[-1] |= wn[-1] >= s.ths[-1]
        sat = old.clone()
        while True:
            pred = _dn(sat, 0) | _dn(sat & oy, 1) | _dn(sat & ox, 2)
            if top_sat:
                pred[0] = True
            new = old | (wsat & (pred | succ))
            if bool((new == sat).all()):
                break
            sat = new
        adj = (pred | succ) & ~old
        refit = ~old & ~adj & (wc < 0.9999 * s.ths)
        h = torch.where(refit, s.head(wc), h)
        wc = torch.where(old, s.ths, torch.where(adj, wch, wc))
        wc = torch.minimum(torch.maximum(wc, s.thr), s.ths)
        if p.adaptive_dt:
            dq = sum((a - b) / f for a, b, f in zip(qp, qm, A)).abs() * dtn / dz
            m = float(dq[1:].max()) if nz > 1 else 0.0
            co = torch.where(wc < s.ths, p.co_max * dz / s.dkdwc(wc), torch.inf)[1:]
            co = co[~co.isnan()]
            dt = dtn * (0.75 if m > 0.02 else 1.25 if m < 0.01 else 1.0)
            dt = min(dt, min(float(co.min()) if co.numel() else math.inf, 1.0e8), p.dt_max)
            dt = dtn = max(dt, p.dt_min)
    return {"h": h, "wc": wc}


CONVS = [(16, 16), (16, 16), (16, 32), (32, 32), (32, 64), (64, 64), (96, 32), (32, 32),
         (48, 16), (16, 16)]


def _exact_net(case, seed):
    """forward (and, for "train", gradients by autograd) of the network in 64 bits"""
    d = np.load(DEFAULT_WEIGHTS)
    kmean, kscale, cscale = (float(v) for v in d["scaling"])
    par = torch.tensor(d["params"], device=DEV, dtype=torch.float64,
                       requires_grad=case["kind"] == "train")
    r, lnk, cap, tgt = (t.double() for t in _net_inputs(case, seed))
    rms = r.square().mean().sqrt()
    off = 0
    layers = []
    for ci, co in CONVS:
        layers.append((par[off:off + 27 * ci * co].view(27, co, ci),
                       par[off + 27 * ci * co:off + 27 * ci * co + co]))
        off += 27 * ci * co + co
    wo, bo = par[off:off + 16], par[off + 16]

    def conv(l, x):
        w, b = layers[l]
        z, y, n = x.shape[:3]
        xp = torch.nn.functional.pad(x, (0, 0, 1, 1, 1, 1, 1, 1))
        o = b.expand(z, y, n, b.numel())
        for t in range(27):
            dz, dy, dx = t // 9, (t // 3) % 3, t % 3
            o = o + xp[dz:dz + z, dy:dy + y, dx:dx + n] @ w[t].T
        return torch.relu(o)

    def pool(x):
        z, y, n, c = x.shape
        return x.reshape(z // 2, 2, y // 2, 2, n // 2, 2, c).mean(dim=(1, 3, 5))

    def up(x):
        return x.repeat_interleave(2, 0).repeat_interleave(2, 1).repeat_interleave(2, 2)

    x0 = torch.zeros(r.shape + (16,), device=DEV, dtype=torch.float64)
    x0[..., 0], x0[..., 1], x0[..., 2] = r / rms, (lnk - kmean) * kscale, cap * cscale
    e1 = conv(1, conv(0, x0))
    e2 = conv(3, conv(2, pool(e1)))
    e3 = conv(5, conv(4, pool(e2)))
    d2 = conv(7, conv(6, torch.cat([up(e3), e2], 3)))
    d1 = conv(9, conv(8, torch.cat([up(d2), e1], 3)))
    y = d1 @ wo + bo
    if case["kind"] == "net":
        return {"y": (y * rms)}
    loss = (y - tgt / rms).square().mean()
    loss.backward()
    return {"loss": float(loss.detach()), "grad": par.grad.cpu().numpy()}


def exact(case, seed):
    if case["kind"] == "seam":
        diag, up, b = _seam_system(case, seed)
        t = [torch.as_tensor(a, device=DEV) for a in (diag, up[2], up[1], up[0])]
        x = _cg(t[0], t[1:], torch.as_tensor(b, device=DEV).view_as(t[0]))
        return {"x": x.ravel().cpu().numpy()}
    n = case["nx"] * case["ny"] * case["nz"]
    if case["kind"] in ("net", "train"):
        # 64-bit activations of every layer (and their gradients) in the card's memory
        return _exact_net(case, seed) if n <= (9 << 20 if case["kind"] == "net" else 3 << 19) \
            else None
    if n > 3 << 20:
        return None  # the 64-bit Picard solves take over 20 seconds
    d = _setup(case, seed)
    shape = (case["nz"], case["ny"], case["nx"])
    f = _exact_pca if case["scheme"] == "pca" else _exact_picard
    return f(d, shape, case["steps"])
