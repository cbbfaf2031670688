"""Performance cases of the LES library, through its public entry points.

A pass of a "steps" case is what a run does between two looks at the flow: some
time steps of the device-resident state, then the velocity brought home as
arrays.  The other kinds are the calls a program makes with its own data: the
horizontal gradients of a field it holds on the device, time steps of velocity
arrays it keeps in host memory, and the gradient of the learned closure's loss.

Every case starts from a developed-looking flow: the log-law profile plus
fluctuations of the size of the friction velocity with a k^(-5/3) spectrum.
"""
from __future__ import annotations

import math
import tempfile

import numpy as np
import torch

from new_repo_b200 import LES, RunParams, load

KAPPA = 0.4
#: Static scratch of the allocation-free gradients (LES_NOALLOC_SCRATCH_BYTES).
GRAD_SCRATCH = 32 << 20
#: Hidden width and input count of the learned closure.
HIDDEN, FEATURES = 64, 8


def _steps(name, nx, ny, nz, precision, sgs, steps, dealias="padd", wall="wall_filter", scalar="none", stats=False):
    return {"name": name, "kind": "steps", "nx": nx, "ny": ny, "nz": nz, "precision": precision, "sgs": sgs,
            "steps": steps, "dealias": dealias, "wall": wall, "scalar": scalar, "stats": stats}


def listed():
    return [
        # an in-situ hook's gradients of a tiny field: launches and latency only
        {"name": "grad_16x16x6", "kind": "grad", "nx": 16, "ny": 16, "levels": 6},
        # the same on a ragged grid: a row length with a factor of three, an odd level count
        {"name": "grad_96x64x51", "kind": "grad", "nx": 96, "ny": 64, "levels": 51},
        # the largest field of 128-point rows the static scratch holds
        {"name": "grad_128x128x83", "kind": "grad", "nx": 128, "ny": 128, "levels": 83},
        # a parity-sized double-precision run, where launches count
        _steps("steps_32x32x16_fp64", 32, 32, 16, "fp64", "dyn_LagScaleDep", 20),
        # a small production run with the constant coefficient
        _steps("steps_64x64x64_mixed", 64, 64, 64, "mixed", "cst_Smag", 20),
        # an odd grid with the other options: plane-averaged dynamic model, 2/3-rule dealiasing,
        # unfiltered wall law, running statistics and the energy budget after every step
        _steps("stats_128x64x41_fp64", 128, 64, 41, "fp64", "dyn_Smag", 10, "trunc", "wall_inst", stats=True),
        # passive scalar with the dynamic Prandtl model in double precision
        _steps("scalar_128x128x128_fp64", 128, 128, 128, "fp64", "dyn_LagScaleDep", 20, scalar="passive"),
        # the benchmark's workload: mixed precision and the learned closure
        _steps("closure_256x256x256_mixed", 256, 256, 256, "mixed", "mlp", 20),
        # the same grid in double precision with the Lagrangian dynamic model
        _steps("lasd_256x256x256_fp64", 256, 256, 256, "fp64", "dyn_LagScaleDep", 10),
        # convective boundary layer on the widest rows: heat flux, inversion, buoyancy, sponge
        _steps("cbl_512x512x96_mixed", 512, 512, 96, "mixed", "dyn_LagScaleDep", 10, scalar="buoyant"),
        # a driver whose own host arrays stay authoritative: in and out at every step
        {"name": "host_128x128x128_fp64", "kind": "host", "nx": 128, "ny": 128, "nz": 128, "steps": 10},
        # loss gradient of the learned closure over one large host batch (forward and backward)
        {"name": "closure_grad_100003", "kind": "closure", "rows": 100003},
    ]


def _size(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["grad", "steps", "steps", "steps", "steps", "host", "closure"])
    if kind == "grad":
        while True:
            nx = rng.choice([16, 24, 32, 48, 64, 96, 128, 192, 256])
            ny = rng.choice([16, 32, 64, 128, 256])
            most = int(0.95 * GRAD_SCRATCH / (3 * 16 * ny * (nx // 2 + 1)))
            if most >= 4:
                return {"kind": kind, "nx": nx, "ny": ny, "levels": _size(rng, 3, most)}
    if kind == "closure":
        return {"kind": kind, "rows": _size(rng, 2000, 200000)}
    if kind == "host":
        return {"kind": kind, "nx": rng.choice([32, 64, 128]), "ny": rng.choice([32, 64, 128]),
                "nz": _size(rng, 16, 128), "steps": rng.choice([5, 10])}
    while True:
        nx, ny = rng.choice([32, 64, 128, 256, 512]), rng.choice([32, 64, 128, 256, 512])
        nz = _size(rng, 12, 260)
        if nx * ny * nz <= 256 * 256 * 160 and max(nx, ny) <= 8 * min(nx, ny):
            break
    precision = rng.choice(["fp64", "mixed"])
    sgs = rng.choice(["cst_Smag", "dyn_LagScaleDep", "dyn_Smag", "dyn_LagScaleDep"] + ["mlp"] * (precision == "mixed"))
    return {k: v for k, v in _steps("", nx, ny, nz, precision, sgs, 10, rng.choice(["padd", "padd", "trunc"]),
                                    rng.choice(["wall_filter", "wall_filter", "wall_inst"]),
                                    rng.choice(["none", "none", "passive", "buoyant"]),
                                    rng.random() < 0.2).items() if k != "name"}


# ------------------------------------------------------------------ inputs
def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _fluctuation(shape, gen):
    """Unit-variance noise (nz, ny, nx) with the k^(-5/3) energy spectrum of a box 2 pi x 2 pi x 1."""
    nz, ny, nx = shape
    h = torch.fft.rfftn(torch.randn(shape, generator=gen, device="cuda", dtype=torch.float64))
    kz = 2 * math.pi * nz * torch.fft.fftfreq(nz, device="cuda", dtype=torch.float64)
    ky = ny * torch.fft.fftfreq(ny, device="cuda", dtype=torch.float64)
    kx = torch.arange(nx // 2 + 1, device="cuda", dtype=torch.float64)
    k2 = kz[:, None, None] ** 2 + ky[:, None] ** 2 + kx**2 + 4.0
    f = torch.fft.irfftn(h * k2 ** (-11.0 / 12.0), s=shape)
    f -= f.mean()
    return f / f.std()


def _params(case):
    stats = bool(case.get("stats"))
    return RunParams(nx=case["nx"], ny=case["ny"], nz=case["nz"], dt=1e-4, lbc_dz0=1e-4, pfx=1.0,
                     sgs_model="dyn_LagScaleDep" if case.get("sgs", "mlp") == "mlp" else case["sgs"], cs_count=5,
                     dyn_init=5, lbc_special="wall_law", wall_model=case.get("wall", "wall_filter"),
                     dealias=case.get("dealias", "padd"), stat_flag=stats, tke_flag=stats,
                     running_period=10**9, tke_period=10**9,
                     out_path=tempfile.mkdtemp() + "/" if stats else "./")


def _velocity(p, seed):
    """u, v, w (nz, ny, nx) on the device: log law plus fluctuations of 1.5, 1.2 and 0.9 friction velocities."""
    gen = _generator(seed)
    shape = (p.nz, p.ny, p.nx)
    z = ((torch.arange(p.nz, device="cuda", dtype=torch.float64) + 0.5) * p.dz)[:, None, None]
    zw = (torch.arange(p.nz, device="cuda", dtype=torch.float64) * p.dz)[:, None, None]
    u = torch.log(z / p.z0) / KAPPA + 1.5 * _fluctuation(shape, gen)
    v = 1.2 * _fluctuation(shape, gen)
    w = 0.9 * torch.sin(math.pi * zw) * _fluctuation(shape, gen)
    return u, v, w


def _closure_parameters(seed):
    """A closure as a trained one looks: Glorot-sized weights, feature statistics of a developed flow, a change of
    log Cs^2 of some percent per update, and a range that covers the flow."""
    r = np.random.RandomState(seed)
    n = HIDDEN
    blocks = [r.randn(FEATURES * n) * math.sqrt(2.0 / (FEATURES + n)), np.zeros(n),
              r.randn(n * n) * math.sqrt(1.0 / n), np.zeros(n), r.randn(n) * math.sqrt(2.0 / (n + 1)), np.zeros(1)]
    mean = [3.0, 5.0, 5.0, 0.0, 3.0, -4.5, 0.0, 5.5]
    std = [1.5, 2.5, 2.5, 5.0, 1.2, 1.0, 4.0, 1.0]
    low, high = [-1e30] * FEATURES, [1e30] * FEATURES
    low[5], high[5] = -1.5, 1.2  # log Cs^2 between -6 and -3.3
    return np.concatenate(blocks + [mean, std, low, high, [0.0, 0.05, -3.0, 3.0]]).astype(np.float32)


def _les(case, seed, precision):
    p = _params(case)
    les = LES(p, precision=precision)
    les.set_initial_conditions(*(f.cpu().numpy() for f in _velocity(p, seed)))
    if max(p.nx, p.ny) >= 512:
        les.set_cs2_max(0.25)  # the dynamic coefficient's clip that 512-point rows need
    if case.get("scalar", "none") != "none":
        buoyant = case["scalar"] == "buoyant"
        z = ((torch.arange(p.nz, device="cuda", dtype=torch.float64) + 0.5) * p.dz)[:, None, None]
        noise = 0.1 * _fluctuation((p.nz, p.ny, p.nx), _generator(seed + 7001))
        if buoyant:
            les.scalar_init(surface_flux=0.24, top_gradient=10.0, buoyancy=9.81 * 1000.0 / 300.0, sgs="dynamic")
            theta = torch.where(z > 0.5, 10.0 * (z - 0.5), torch.zeros_like(z)) + torch.where(z < 0.4, noise, 0.1 * noise)
            les.sponge_init(0.8)
        else:
            les.scalar_init(surface_flux=0.0, top_gradient=1.0, buoyancy=0.0, sgs="dynamic")
            theta = z + noise
        les.scalar_set_initial(theta.cpu().numpy())
    if case.get("sgs") == "mlp":
        les.mlp_init(0)
        les.mlp_set_params(_closure_parameters(11))
        les.set_sgs_model("mlp")
        les.mlp_set_wall_levels(8)
    return les


def _closure_rows(case, seed):
    gen = _generator(seed)
    x = torch.randn((case["rows"], FEATURES), generator=gen, device="cuda", dtype=torch.float32)
    t = torch.tanh(x[:, 0] - 0.5 * x[:, 3]) + 0.1 * torch.randn(case["rows"], generator=gen, device="cuda")
    return x, t


def prepare(case, seed):
    kind = case["kind"]
    if kind == "grad":
        shape = (case["levels"], case["ny"], case["nx"])
        f = 2.0 * _fluctuation(shape, _generator(seed)) + 18.0
        return {"case": case, "call": load().les_grad_xy_noalloc, "f": f, "dx": torch.empty_like(f),
                "dy": torch.empty_like(f), "lx": 2 * math.pi, "ly": 2 * math.pi}
    if kind == "closure":
        # the closure lives in a state; a small one does where only its network is used
        les = LES(RunParams(nx=16, ny=16, nz=4), precision="mixed")
        les.mlp_init(0)
        les.mlp_set_params(_closure_parameters(11))
        x, t = _closure_rows(case, seed)
        return {"case": case, "les": les, "x": x.cpu().numpy(), "t": t.cpu().numpy()}
    precision = case.get("precision", "fp64")
    les = _les(case, seed, precision)
    levels = case["nz"] + (2 if kind == "host" else 0)
    names = ("u", "v", "w") + (("theta",) if case.get("scalar", "none") != "none" else ())
    host = {n: torch.empty((levels, case["ny"], case["nx"]), dtype=torch.float64, pin_memory=True) for n in names}
    if kind == "host":
        for n in names:
            les.download_async(n, host[n].data_ptr())
        les.sync()
    return {"case": case, "les": les, "host": host, "diag": torch.zeros(4, dtype=torch.float64, pin_memory=True)}


# -------------------------------------------------------------------- runs
def _run_grad(s):
    c, f, dx, dy = s["case"], s["f"], s["dx"], s["dy"]
    status = s["call"](f.data_ptr(), dx.data_ptr(), dy.data_ptr(), c["nx"], c["ny"], c["levels"], s["lx"], s["ly"],
                       torch.cuda.current_stream().cuda_stream)
    if status:
        raise RuntimeError("les_grad_xy_noalloc: status %d" % status)
    return {"f": f, "dfdx": dx, "dfdy": dy}


def _run_steps(s):
    les, case, host = s["les"], s["case"], s["host"]
    les.step(case["steps"])
    out = {}
    if case["precision"] == "fp64":
        for n, h in host.items():
            les.download_async(n, h.data_ptr(), 1, case["nz"])
        les.sync()
        out.update(host)
    else:
        # FP32 fields: onto the device as FP32 tensors for what follows the run there; one field
        # travels back in while the next one comes out
        for n, h in host.items():
            les.download_async(n, h.data_ptr(), 1, case["nz"])
            les.sync()
            out[n] = h.to("cuda", non_blocking=True).float()
        torch.cuda.current_stream().synchronize()
    if case["stats"]:
        out["budget"] = les.tke_profiles()[0]
    return out


def _run_host(s):
    host = s["host"]
    s["les"].step_host(host["u"].data_ptr(), host["v"].data_ptr(), host["w"].data_ptr(), s["diag"].data_ptr(),
                       n=s["case"]["steps"])
    s["les"].sync()
    return {"u": host["u"], "v": host["v"], "w": host["w"], "diagnostics": s["diag"]}


def _run_closure(s):
    grad, loss = s["les"].mlp_grad(s["x"], s["t"])
    return {"grad": grad, "loss": loss}


def run(state):
    return {"grad": _run_grad, "steps": _run_steps, "host": _run_host, "closure": _run_closure}[state["case"]["kind"]](state)


# -------------------------------------------------------------------- work
def work(case):
    """Bytes: for time steps, the operators' inputs read once and outputs written once in the state's precision (105
    field passes a step, 28 more per update of a dynamic coefficient, 17 for a scalar) plus the arrays brought home.
    Flops: 2.5 n log2 n per real 2-D transform."""
    kind = case["kind"]
    if kind == "grad":
        n = case["nx"] * case["ny"] * case["levels"]
        return {"bytes": 4 * 8.0 * n, "flops": 4 * 2.5 * n * math.log2(case["nx"] * case["ny"])}
    if kind == "closure":
        macs = FEATURES * HIDDEN + HIDDEN * HIDDEN + HIDDEN
        return {"bytes": 4.0 * (FEATURES + 1) * case["rows"], "flops": 6.0 * macs * case["rows"]}
    n = case["nx"] * case["ny"] * case["nz"]
    size = 4.0 if case.get("precision") == "mixed" else 8.0
    scalar = case.get("scalar", "none") != "none"
    passes = 105.0 + (0.0 if case.get("sgs") == "cst_Smag" else 28.0 / 5) + (17.0 if scalar else 0.0)
    # transforms: 12 gradients, 18 convection (half of them on 2.25 times the points), 9 stress divergence, 6 pressure
    transforms = 45.0 + (11.25 if case.get("dealias", "padd") == "padd" else 0.0) + (14.0 if scalar else 0.0)
    moved = (3 + scalar) * 8.0 * n * (2 * case["steps"] if kind == "host" else 1)
    return {"bytes": case["steps"] * passes * size * n + moved,
            "flops": case["steps"] * transforms * 2.5 * n * math.log2(case["nx"] * case["ny"])}


# ------------------------------------------------------------------- exact
class _Grid:
    def __init__(self, p):
        self.p, self.norm = p, 1.0 / (p.nx * p.ny)
        kx = torch.arange(p.nx // 2 + 1, device="cuda", dtype=torch.float64) * (2 * math.pi / p.lx)
        ky = torch.fft.fftfreq(p.ny, 1.0 / p.ny, device="cuda", dtype=torch.float64) * (2 * math.pi / p.ly)
        keep = torch.ones(p.ny, p.nx // 2 + 1, device="cuda", dtype=torch.float64)
        keep[:, -1] = 0
        keep[p.ny // 2] = 0
        self.kx, self.ky, self.keep = kx * keep, ky[:, None] * keep, keep

    def to(self, f):
        return torch.fft.rfft2(f) * (self.norm * self.keep)

    def back(self, h):
        return torch.fft.irfft2(h, s=(self.p.ny, self.p.nx), norm="forward")


def _exact_grad(case, seed):
    shape = (case["levels"], case["ny"], case["nx"])
    f = 2.0 * _fluctuation(shape, _generator(seed)) + 18.0
    g = _Grid(RunParams(nx=case["nx"], ny=case["ny"], nz=8))
    h = g.to(f)
    return {"f": g.back(h), "dfdx": g.back(1j * g.kx * h), "dfdy": g.back(1j * g.ky * h)}


def _pad(h, p, fy, fx):
    """Spectrum (.., ny, nx/2+1) without its Nyquist modes on the 3/2 grid, as physical values there."""
    big = torch.zeros(h.shape[:-2] + (fy, fx // 2 + 1), dtype=h.dtype, device=h.device)
    ny, n = p.ny // 2, p.nx // 2
    big[..., :ny, :n] = h[..., :ny, :n]
    big[..., fy - ny + 1:, :n] = h[..., ny + 1:, :n]
    return torch.fft.irfft2(big, s=(fy, fx), norm="forward")


def _unpad(f, p, fy, fx):
    big = torch.fft.rfft2(f) / (fy * fx)
    h = torch.zeros(f.shape[:-2] + (p.ny, p.nx // 2 + 1), dtype=big.dtype, device=f.device)
    ny, n = p.ny // 2, p.nx // 2
    h[..., :ny, :n] = big[..., :ny, :n]
    h[..., ny + 1:, :n] = big[..., fy - ny + 1:, :n]
    return torch.fft.irfft2(h, s=(p.ny, p.nx), norm="forward")


def _mid(f):
    """Mean of each level and the one below it (levels 2..)."""
    return 0.5 * (f[2:] + f[1:-1])


def _exact_steps(case, seed):
    """The time steps with the constant coefficient, log-law wall and padded products, in 64 bits."""
    p = _params(case)
    g, nz, dz, dt = _Grid(p), p.nz, p.dz, p.dt_nd
    fx, fy = 3 * p.nx // 2, 3 * p.ny // 2
    zero = lambda: torch.zeros((nz + 2, p.ny, p.nx), device="cuda", dtype=torch.float64)  # noqa: E731
    vel = [zero(), zero(), zero()]
    for f, x in zip(vel, _velocity(p, seed)):
        f[1:-1] = x
    u, v, w = vel
    u[0], v[0], u[-1], v[-1] = -u[1], -v[1], u[-2], v[-2]
    w[0], w[1], w[-1] = 0.0, 0.0, 0.0
    length = (p.dx * p.dy * dz) ** (1.0 / 3.0)
    z = torch.arange(-1, nz + 1, device="cuda", dtype=torch.float64) * dz
    z[1] = 0.5 * dz
    z[0] = dz
    l2 = (1.0 / (p.cs0**2 / (KAPPA * z) ** 2 + length**-2))[:, None, None]
    # the cutoff lies on a wavenumber: which side that falls to is told in single precision
    cut = (g.kx**2 + g.ky**2).float().double() < (math.pi / (2.0 * math.sqrt(p.dx * p.dy))) ** 2
    rhs = [zero(), zero(), zero()]
    interior = slice(1, nz + 1)
    for step in range(case["steps"]):
        # wall law on the filtered (or plain) first level
        u1, v1 = u[1], v[1]
        if p.wall_model == "wall_filter":
            u1, v1 = g.back(g.to(u1) * cut), g.back(g.to(v1) * cut)
        speed = torch.sqrt(u1**2 + v1**2)
        star = KAPPA * speed / math.log(0.5 * dz / p.z0)
        bu, bv = (star / (0.5 * dz * KAPPA) * x / speed for x in (u1, v1))
        wall_tx, wall_ty = star**2 * u1 / speed, star**2 * v1 / speed
        # gradients (the velocity loses its Nyquist modes)
        dx, dy = [], []
        for f in vel:
            h = g.to(f)
            dx.append(g.back(1j * g.kx * h))
            dy.append(g.back(1j * g.ky * h))
            f.copy_(g.back(h))

        def ghosts():
            u[0], v[0], w[1] = u[1] - bu * dz, v[1] - bv * dz, 0.0
            u[-1], v[-1], w[-1] = u[-2], v[-2], 0.0

        ghosts()
        uz, vz, wz = zero(), zero(), zero()
        uz[1:], vz[1:] = (u[1:] - u[:-1]) / dz, (v[1:] - v[:-1]) / dz
        wz[1:-1] = (w[2:] - w[1:-1]) / dz
        (ux, vx, wx), (uy, vy, wy) = dx, dy
        # strain on uvp nodes at the wall, on w nodes above, and the stresses
        s11, s12, s13, s22, s23, s33 = (zero() for _ in range(6))
        s11[1], s22[1], s33[1], s12[1] = ux[1], vy[1], wz[1], 0.5 * (uy[1] + vx[1])
        s13[1] = 0.5 * (uz[1] + 0.5 * (wx[1] + wx[2]))
        s23[1] = 0.5 * (vz[1] + 0.5 * (wy[1] + wy[2]))
        s11[2:], s22[2:], s33[2:] = _mid(ux), _mid(vy), _mid(wz)
        s12[2:] = 0.5 * (_mid(uy) + _mid(vx))
        s13[2:], s23[2:] = 0.5 * (uz[2:] + wx[2:]), 0.5 * (vz[2:] + wy[2:])
        norm = torch.sqrt(2.0 * (s11**2 + s22**2 + s33**2 + 2.0 * (s12**2 + s13**2 + s23**2)))
        nu = norm * p.cs0**2 * l2
        at = nu.clone()
        at[2:-1] = 0.5 * (nu[2:-1] + nu[3:])
        at[-1] = 0.0
        txx, tyy, tzz, txy = 2 * at * ux, 2 * at * vy, 2 * at * wz, at * (uy + vx)
        txz, tyz = 2 * nu * s13, 2 * nu * s23
        txz[1], tyz[1], tzz[0] = wall_tx, wall_ty, tzz[1]
        # rotational convective term on the 3/2 grid
        o1, o2, o3 = wy - vz, uz - wx, vx - uy
        o1[1] = 0.5 * (wy[1] + wy[2]) - vz[1]
        o2[1] = uz[1] - 0.5 * (wx[1] + wx[2])
        ub, vb, wb, o1, o2, o3 = (_pad(g.to(f), p, fy, fx) for f in (u, v, w, o1, o2, o3))
        cx, cy, cz = (torch.zeros_like(ub) for _ in range(3))
        cx[1:-1] = vb[1:-1] * o3[1:-1] - 0.5 * wb[2:] * o2[2:]
        cy[1:-1] = -ub[1:-1] * o3[1:-1] + 0.5 * wb[2:] * o1[2:]
        cx[2:-1] -= 0.5 * wb[2:-1] * o2[2:-1]
        cy[2:-1] += 0.5 * wb[2:-1] * o1[2:-1]
        cz[2:-1] = 0.5 * ((ub[2:-1] + ub[1:-2]) * o2[2:-1] - (vb[2:-1] + vb[1:-2]) * o1[2:-1])
        old, rhs = rhs, [_unpad(c, p, fy, fx) for c in (cx, cy, cz)]
        del ub, vb, wb, o1, o2, o3, cx, cy, cz
        flux = [g.back(1j * (g.kx * g.to(a) + g.ky * g.to(b))) for a, b in ((txx, txy), (txy, tyy), (txz, tyz))]
        for q, t in ((0, txz), (1, tyz)):
            rhs[q][interior] += flux[q][interior] + (t[2:] - t[1:-1]) / dz
        wflux = flux[2][interior] + (tzz[1:-1] - tzz[:-2]) / dz
        rhs[2][interior] += wflux
        rhs[0][interior] += p.pfx
        rhs[1][interior] += p.pfy
        bottom, top = wflux[0], flux[2][-1]
        # advance, pressure, projection
        a1, a2 = (1.0, 0.0) if step == 0 else (1.5, -0.5)
        for f, r, o in zip(vel, rhs, old):
            f[interior] += dt * (a1 * r[interior] + a2 * o[interior])
        w[0], w[-1] = 0.0, 0.0
        hx, hy, hz = (g.to(f) / (a1 * dt) for f in vel)
        r = torch.zeros_like(hx)
        r[0], r[-1] = g.to(bottom) * dz, g.to(top) * dz
        r[interior] = 1j * (g.kx * hx + g.ky * hy)[interior] + (hz[2:] - hz[1:-1]) / dz
        r[0, 0, 0] = 0.0
        lower = 1.0 / dz**2
        diag = -(g.kx**2 + g.ky**2 + 2.0 / dz**2)
        beta = torch.full_like(diag, -1.0)
        upper = torch.ones_like(diag)
        beta[0, 0], upper[0, 0] = 1.0, 0.0
        gam, x = torch.zeros((nz + 2,) + diag.shape, device="cuda", dtype=torch.float64), torch.zeros_like(r)
        x[0] = r[0] / beta
        for k in range(1, nz + 2):
            below, here = (lower, diag) if k <= nz else (-1.0, torch.ones_like(diag))
            gam[k] = upper / beta
            beta = here - below * gam[k]
            x[k] = (r[k] - below * x[k - 1]) / torch.where(g.keep > 0, beta, torch.ones_like(beta))
            upper = torch.full_like(diag, lower)
        for k in range(nz, -1, -1):
            x[k] -= gam[k + 1] * x[k + 1]
        x = torch.where(g.keep > 0, x, torch.zeros_like(x))
        px, py, pr = g.back(1j * g.kx * x), g.back(1j * g.ky * x), g.back(x)
        pz = torch.zeros_like(pr)
        pz[interior] = (pr[interior] - pr[:nz]) / dz
        for f, q, d in zip(vel, rhs, (px, py, pz)):
            f[interior] -= dt * a1 * d[interior]
            q[interior] -= d[interior]
        w[1], w[-1] = 0.0, 0.0
        ghosts()
    return {n: f[interior].clone() for n, f in zip("uvw", vel)}


def _exact_closure(case, seed):
    """The gradient of the mean squared error of the 8 -> 64 -> 64 -> 1 network (tanh-form GELU), in 64 bits."""
    x, t = (a.double() for a in _closure_rows(case, seed))
    n = HIDDEN
    theta = torch.from_numpy(_closure_parameters(11)).double().cuda()[: FEATURES * n + n * n + 3 * n + 1].requires_grad_()
    w1, b1, w2, b2, w3, b3 = torch.split(theta, [FEATURES * n, n, n * n, n, n, 1])
    gelu = torch.nn.functional.gelu
    h = gelu(x @ w1.view(FEATURES, n) + b1, approximate="tanh")
    h = gelu(h @ w2.view(n, n) + b2, approximate="tanh")
    loss = ((h @ w3 + b3 - t) ** 2).mean()
    loss.backward()
    return {"grad": theta.grad, "loss": loss.detach()}


def exact(case, seed):
    """Values in 64 bits.  The dynamic coefficients have none: their clips round to single precision, so that a point
    on a rounding edge may fall to either side."""
    if case["kind"] == "grad":
        return _exact_grad(case, seed)
    if case["kind"] == "closure":
        return _exact_closure(case, seed)
    if (case["kind"] == "steps" and case["sgs"] == "cst_Smag" and case["dealias"] == "padd"
            and case["scalar"] == "none" and not case["stats"]):
        return _exact_steps(case, seed)
    return None
