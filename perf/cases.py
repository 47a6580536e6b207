"""The work that programs have this solver do, as timed cases.

A case is one call pattern of a driver of the channel: a run of RK3 steps
between two outputs and the read-back of the fields it ends with, a step with
the fields kept in the driver's own arrays, a step with an immersed body, the
diagnostics of an output interval, one pass of the learned preconditioner's
training.  Sizes and options are those of this repository's workloads and
tests; the marker counts follow the grids.

Kinds
  run   nsteps RK3 steps resident on the GPU, then U, V, W read back into the
        driver's page-locked arrays (what a driver does every nsave/nstats
        steps).  poisson "fp64" or "mixed"; cfl > 0: dt from the fields before
        every step, cfl < 0: dt = -cfl.
  host  nsteps RK3 steps with U, V, W living in the driver's arrays.
  ib    nsteps RK3 steps with an immersed body, U, V, W and the surface
        unknowns read back.
  diag  statistics profiles and the monitor line of the current fields.
  net   forward, loss and parameter gradient of the preconditioner's network
        on a batch of marker rows.
"""
import math

import numpy as np
import torch

import channel3d_parallel_b200 as c3d
from channel3d_parallel_b200 import lib as L

NU = 1.0 / 5600.0
SMOOTH = (16, 18, 24, 32, 36, 48, 54, 64, 72, 96, 108, 128, 144, 162, 192, 216, 256, 288, 324, 384)


def _channel(kind, Nx, Ny, Nz, Lx, Lz, nsteps, **kw):
    """A channel of Nx x Ny x Nz cells; alpha 0 gives a uniform y grid."""
    c = dict(kind=kind, Nx=Nx, Ny=Ny, Nz=Nz, Lx=Lx, Lz=Lz, nsteps=nsteps, nu=NU, cfl=-1e-3, alpha=2.0,
             mass=1, poisson="fp64", amplitude=0.1)
    c.update(kw)
    return c


def _wave(Nx, Ny, Nz, Lx, Lz, nsteps, precond, tol=1e-12):
    """An immersed standing-wave plane, one marker per x and z cell."""
    return _channel("ib", Nx, Ny, Nz, Lx, Lz, nsteps, body="wall_standing_wave", nxb=Nx, nzb=Nz, p1=0.02,
                    p2=2 * math.pi / 5, p3=1.0, p4=0.2, buffer=0.45, precond=precond, tol=tol, amplitude=0.05)


def listed():
    pi = math.pi
    return [
        # one step of the minimal channel by a driver that looks at the fields
        # after every step: launch and synchronisation latency
        dict(_channel("run", 32, 64, 32, pi, pi / 2, 1), name="step_minimal"),
        # the minimal channel's own run of 100 steps
        dict(_channel("run", 32, 64, 32, pi, pi / 2, 100), name="run_minimal"),
        # the Re_tau = 180 channel between two outputs: the benchmark's workload
        dict(_channel("run", 192, 128, 192, 4 * pi, 4 * pi / 3, 50), name="run_180"),
        # the same with the time step from the fields (compute_dt before every step)
        dict(_channel("run", 192, 128, 192, 4 * pi, 4 * pi / 3, 20, cfl=0.12), name="cfl_180"),
        # the same with the mixed-precision Poisson solve
        dict(_channel("run", 192, 128, 192, 4 * pi, 4 * pi / 3, 20, poisson="mixed"), name="mixed_180"),
        # the same with the fields in the driver's own arrays, as the
        # reference's time loop keeps them
        dict(_channel("host", 192, 128, 192, 4 * pi, 4 * pi / 3, 4), name="host_180"),
        # a channel whose extents fit no tile and no power of two, driven by a
        # fixed pressure gradient
        dict(_channel("run", 162, 113, 108, 10.0, 4.0, 30, mass=0), name="run_ragged"),
        # the Re_tau = 550 channel between two outputs
        dict(_channel("run", 384, 256, 384, 2 * pi, pi, 10, nu=1.0 / 20000.0), name="run_550"),
        # the benchmark's immersed wave (36,864 markers) with the band preconditioner
        dict(_wave(192, 128, 192, 4 * pi, 4 * pi / 3, 1, "band"), name="ib_wave"),
        # the benchmark's two rotating cylinders (51,200 markers), band preconditioner
        dict(_channel("ib", 256, 128, 128, 4.5, 2.0, 1, alpha=0.0, body="two_cylinders_z", nxb=200, nzb=128,
                      p1=0.15, p2=0.5, p3=1.5, p4=0.3, buffer=0.0, precond="band", tol=1e-12), name="ib_cylinders"),
        # the statistics and monitor calls of an output interval
        dict(_channel("diag", 192, 128, 192, 4 * pi, 4 * pi / 3, 0), name="diagnostics_180"),
        # one training pass of the preconditioner's network (forward and backward)
        dict(kind="net", rows=36864, name="network"),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choices(("run", "cfl", "mixed", "host", "ib", "diag", "net"), (46, 12, 14, 8, 10, 5, 5))[0]
    if kind == "net":
        return dict(kind="net", rows=int(_log(rng, 200, 40000)))
    if kind == "ib":
        Nx, Nz = rng.choice(SMOOTH[3:15]), rng.choice(SMOOTH[:15])
        Ny = rng.randint(48, 128)
        return _wave(Nx, Ny, Nz, Nx * 0.0654, Nz * 0.0327, 1, rng.choice(("none", "band")))
    while True:
        Nx, Nz = rng.choice(SMOOTH), rng.choice(SMOOTH)
        Ny = int(_log(rng, 16, 256))
        cells = Nx * Ny * Nz
        if cells <= 30e6 and cells * 3 >= _log(rng, 2e4, 3e7):
            break
    n = max(1, min(int(_log(rng, 1, 60)), int(3e8 / cells)))
    c = _channel("run" if kind in ("cfl", "mixed") else kind, Nx, Ny, Nz, Nx * 0.0654, Nz * 0.0327, n,
                 alpha=rng.choice((0.0, 2.0, 2.0)), mass=rng.choice((0, 1, 1)))
    if kind == "cfl":
        # a CFL number that gives time steps of about 3e-3 on this y grid
        y = _faces(c)
        dy = float((y[1:] - y[:-1]).min())
        c["cfl"] = min(0.2, 3e-3 * c["nu"] / dy ** 2)
    if kind == "mixed":
        c["poisson"] = "mixed"
    if kind == "host":
        c["nsteps"] = min(n, 4)
    if kind == "diag":
        c["nsteps"] = 0
    return c


# --------------------------------------------------------------------------
# seeded inputs
# --------------------------------------------------------------------------
def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _faces(c):
    """y faces: uniform, or tanh-stretched on [0, 2]."""
    y = torch.arange(c["Ny"] + 1, dtype=torch.float64) * (2.0 / c["Ny"])
    if c["alpha"] > 0:
        y = torch.tanh(c["alpha"] * (y - 1.0)) / math.tanh(c["alpha"])
        y = y - y.min()
        y = y * (2.0 / y.max())
    return y


def _unique(c, seed):
    """Laminar profile plus uniform perturbations on the distinct points:
    u (Nz, Ny, Nx), v (Nz, Ny-1, Nx) between the walls, w (Nz, Ny, Nx)."""
    dev = _device()
    g = torch.Generator(device=dev).manual_seed(1 + int(seed))
    y = _faces(c).to(dev)
    ym = 0.5 * (y[1:] + y[:-1])
    a = c["amplitude"]

    def noise(n):
        return 2.0 * a * (torch.rand((c["Nz"], n, c["Nx"]), generator=g, device=dev, dtype=torch.float64) - 0.5)

    u = noise(c["Ny"]) + (1.5 * ym * (2.0 - ym))[None, :, None]
    return u, noise(c["Ny"] - 1), noise(c["Ny"])


def _full(u, v, w):
    """The reference's arrays with their ghost cells (Fortran order = these
    tensors' memory): periodic copies in x and z, walls in y."""
    Nz, Ny, Nx = u.shape
    dev = u.device

    def ix(n, m):
        return (torch.arange(n, device=dev) - 1) % m

    odd = lambda f: torch.cat([-f[:, :1], f, -f[:, -1:]], 1)      # noqa: E731
    zero = torch.zeros_like(v[:, :1])
    U = odd(u)[ix(Nz + 3, Nz)][:, :, ix(Nx + 2, Nx)]
    V = torch.cat([zero, v, zero], 1)[ix(Nz + 3, Nz)][:, :, ix(Nx + 3, Nx)]
    W = odd(w)[ix(Nz + 2, Nz)][:, :, ix(Nx + 3, Nx)]
    return U, V, W


def _pinned(t):
    out = torch.empty(t.shape, dtype=t.dtype, pin_memory=torch.cuda.is_available())
    out.copy_(t)
    return out


# --------------------------------------------------------------------------
# the driver's side
# --------------------------------------------------------------------------
class State:
    pass


def _read_back(s):
    """U, V, W into the driver's arrays."""
    lib = L.load()
    for name, buf in s.host.items():
        lb, ub = s.box[name]
        L.check(lib.c3d_download(s.ch.handle, L.FIELD[name], L.C.cast(buf.data_ptr(), L._D), lb, ub), s.ch.handle)
    return s.host


def prepare(case, seed):
    s = State()
    s.case = case
    if case["kind"] == "net":
        m = case["rows"]
        s.params, s.feats, s.moments, s.sig = _net_inputs(m, seed)
        s.ch = c3d.Channel(nx_global=18, ny_global=17, nz_global=18, Lxp=1.0, Lzp=1.0, nu=NU, CFL=-1e-3)
        s.ch.precond_set_params(s.params, s.sig)
        return s
    kw = dict(nx_global=case["Nx"] + 2, ny_global=case["Ny"] + 1, nz_global=case["Nz"] + 2, Lxp=case["Lx"],
              Lzp=case["Lz"], nu=case["nu"], CFL=case["cfl"], x_mass_cte=case["mass"], dPdx=3.0 * case["nu"])
    if case["kind"] == "ib":
        kw.update(grid_type=2 if case["buffer"] else 0, alpha_stretch=2.0 if case["buffer"] else 0.0,
                  min_buffer_width=case["buffer"], body_type=case["body"], nxb=case["nxb"], nzb=case["nzb"],
                  body_param_1=case["p1"], body_param_2=case["p2"], body_param_3=case["p3"],
                  body_param_4=case["p4"], cg_tol=case["tol"], cg_max_iter=600)
    else:
        kw.update(grid_type=1 if case["alpha"] > 0 else 0, alpha_stretch=case["alpha"])
    ch = s.ch = c3d.Channel(**kw)
    if case["kind"] == "ib":
        ch.compute_heaviside()
    fields = dict(zip("UVW", (_pinned(f) for f in _full(*_unique(case, seed)))))
    s.box = {n: L.box(*ch.bounds(n)) for n in fields}
    s.host = fields
    for n, f in fields.items():
        ch.upload(n, f.numpy().T)
    ch.set_scalars(dPdx=3.0 * case["nu"])
    ch.compute_dt()
    ch.compute_non_IB_projection(rk_step=0)
    ch.apply_boundary_conditions("UVW")
    ch.set_scalars(dPdx=3.0 * case["nu"], Qflow_x_0=ch.compute_mean_mass_flow_U())
    if case["kind"] == "ib":
        ch.set_mode(precond={"none": L.PRECOND_NONE, "band": L.PRECOND_BAND}[case["precond"]])
    elif case["poisson"] == "mixed":
        ch.set_mode(poisson=L.POISSON_MIXED)
    if case["kind"] == "host":
        _read_back(s)
        s.views = [s.host[n].numpy().T for n in "UVW"]
    return s


def run(s):
    c, ch = s.case, s.ch
    if c["kind"] == "net":
        out, grad, loss = ch.precond_eval(s.feats, s.moments, s.sig)
        return {"out": out, "grad": grad, "loss": loss}
    if c["kind"] == "diag":
        st = ch.compute_statistics()
        mon = ch.output_monitor()
        # zero but for round-off on a divergence-free field between walls
        for k in ("Vmean", "Qflow_y"):
            st.pop(k)
        for k in ("meanV", "max_divergence"):
            mon.pop(k)
        return {"stats": st, "monitor": mon}
    if c["kind"] == "host":
        ch.compute_time_step_RK3_host(*s.views, nsteps=c["nsteps"])
        return s.host
    ch.compute_time_step_RK3(c["nsteps"])
    out = dict(_read_back(s))
    if c["kind"] == "ib":
        out["FB"] = ch.download("FB")
    else:
        out["dPdx"] = ch.stats()["dPdx"]
    return out


def work(case):
    """Bytes and operations of one pass.  A stage of a step reads u, v, w, the
    accumulators and the potential and writes u, v, w (80 B a cell); its
    Poisson solve reads u, v, w, moves the spectrum through memory twice each
    way (the two transposes) and writes the potential (64 B).  Operations: the
    right-hand sides (about 100 a cell), the transforms and the tridiagonal
    solves."""
    if case["kind"] == "net":
        m = case["rows"]
        mac = 32 * 128 + 128 * 128 + 128 * 16
        return {"bytes": m * (32 * 4 + 36 * 4 + 16 * 4) + 2 * 22800 * 4, "flops": 6.0 * m * mac}
    n = case["Nx"] * case["Ny"] * case["Nz"]
    if case["kind"] == "diag":
        return {"bytes": 24.0 * n, "flops": 30.0 * n}
    fft = 5.0 * (math.log2(case["Nx"]) + math.log2(case["Nz"]))
    step = {"bytes": 432.0 * n, "flops": 3 * n * (100.0 + fft + 20.0)}
    got = {k: v * case["nsteps"] for k, v in step.items()}
    if case["poisson"] == "mixed":
        # the refinement's residual and second solve: u, v, w and the
        # potential again, the FP32 spectrum, the potential updated
        got["bytes"] += case["nsteps"] * 3 * (32.0 + 16.0 + 16.0 - 16.0) * n
    if case["kind"] == "host":
        got["bytes"] += 48.0 * n * case["nsteps"]
    else:
        got["bytes"] += 24.0 * n
    if case["kind"] == "ib":
        # three Schur solves a step; an iteration applies S and the
        # preconditioner twice.  Ten iterations, on the rows the stencils reach
        rows = 12 if case["body"] == "wall_standing_wave" else 44
        got["bytes"] += case["nsteps"] * 3 * 20 * 120.0 * rows * case["Nx"] * case["Nz"]
    return got


# --------------------------------------------------------------------------
# what run() returns, in 64 bits
# --------------------------------------------------------------------------
def exact(case, seed):
    """None for the immersed bodies: their step solves a dense Schur system of
    four unknowns a marker (147,456 and 204,800) to a tolerance; factored
    directly it takes far longer than a few seconds."""
    if case["kind"] == "ib":
        return None
    if case["kind"] == "net":
        return _net_exact(case, seed)
    u, v, w = _unique(case, seed)
    ch = _Exact(case, u.device)
    u, v, w = ch.project(u, v, w)
    if case["kind"] == "diag":
        return _diag_exact(ch, u, v, w)
    dPdx, q0 = 3.0 * case["nu"], ch.flux(u)
    for _ in range(case["nsteps"]):
        dt = ch.dt(u, v, w)
        gu = gv = gw = None
        for stage, (cs, cg) in enumerate(((8.0 / 15.0, 0.25), (5.0 / 12.0, 0.0), (0.75, 0.0))):
            fu, fv, fw = ch.rhs(u, v, w, dPdx)
            if stage == 0:
                gu, gv, gw = u + dt * cg * fu, v + dt * cg * fv, w + dt * cg * fw
                u, v, w = u + dt * cs * fu, v + dt * cs * fv, w + dt * cs * fw
            else:
                u, v, w = gu + dt * cs * fu, gv + dt * cs * fv, gw + dt * cs * fw
            u, v, w = ch.project(u, v, w)
        if case["mass"]:
            shift = q0 - ch.flux(u)
            u = u + shift
            dPdx = 0.5 * (dPdx + shift / dt)
    out = dict(zip("UVW", _full(u, v, w)))
    if case["kind"] == "run":
        out["dPdx"] = dPdx
    return out


def _up(f, d):
    return torch.roll(f, -1, d)


def _dn(f, d):
    return torch.roll(f, 1, d)


class _Exact:
    """The channel's step on the distinct points (z, y, x), plain torch."""

    def __init__(self, c, dev):
        self.c = c
        self.Nx, self.Ny, self.Nz = c["Nx"], c["Ny"], c["Nz"]
        self.dx, self.dz = c["Lx"] / c["Nx"], c["Lz"] / c["Nz"]
        self.y = y = _faces(c).to(dev)
        ym = 0.5 * (y[1:] + y[:-1])
        self.yg = yg = torch.cat([2 * y[:1] - ym[:1], ym, 2 * y[-1:] - ym[-1:]])
        self.rdy = (1.0 / (y[1:] - y[:-1]))[None, :, None]          # cells
        self.rdyg = (1.0 / (yg[1:] - yg[:-1]))[None, :, None]       # faces, walls included
        kx = torch.arange(self.Nx // 2 + 1, device=dev, dtype=torch.float64)
        kz = torch.arange(self.Nz, device=dev, dtype=torch.float64)
        lx = 2.0 * (torch.cos(2 * math.pi * kx / self.Nx) - 1.0) / self.dx ** 2
        lz = 2.0 * (torch.cos(2 * math.pi * kz / self.Nz) - 1.0) / self.dz ** 2
        self.lam = lx[None, :] + lz[:, None]                        # (Nz, nkx)
        r, rg = self.rdy.flatten(), self.rdyg.flatten()
        self.up = r[:-1] * rg[1:-1]
        self.lo = r[1:] * rg[1:-1]
        self.dd = torch.zeros_like(r)
        self.dd[:-1] -= self.up
        self.dd[1:] -= self.lo

    def dt(self, u, v, w):
        c = self.c
        if c["cfl"] < 0:
            return -c["cfl"]
        # the reference takes the largest spacing/|velocity|; v is zero on the
        # upper wall, so it sets no limit
        conv = min(self.dx / u.abs().min().item(), self.dz / w.abs().min().item())
        dymin = float((self.yg[1:] - self.yg[:-1]).min())
        visc = min(self.dx ** 2, dymin ** 2, self.dz ** 2) / c["nu"]
        return min(c["cfl"] * conv, c["cfl"] * visc, 0.1)

    def rhs(self, u, v, w, dPdx):
        nu, dx, dz = self.c["nu"], self.dx, self.dz
        rdy, rdyg = self.rdy, self.rdyg
        zero = torch.zeros_like(v[:, :1])
        ue = torch.cat([-u[:, :1], u, -u[:, -1:]], 1)               # centres with ghosts
        we = torch.cat([-w[:, :1], w, -w[:, -1:]], 1)
        vf = torch.cat([zero, v, zero], 1)                          # faces, walls included
        z, x = 0, 2
        # momentum fluxes on the cell edges and centres
        exy = 0.25 * (ue[:, 1:] + ue[:, :-1]) * (vf + _up(vf, x))   # (z, face, x+1/2)
        exz = 0.25 * (u + _up(u, z)) * (w + _up(w, x))
        eyz = 0.25 * (vf + _up(vf, z)) * (we[:, 1:] + we[:, :-1])
        cx = 0.25 * (_dn(u, x) + u) ** 2                            # cell centres
        cy = 0.25 * (vf[:, 1:] + vf[:, :-1]) ** 2
        cz = 0.25 * (_dn(w, z) + w) ** 2
        fu = -(_up(cx, x) - cx) / dx - (exy[:, 1:] - exy[:, :-1]) * rdy - (exz - _dn(exz, z)) / dz
        fw = -(_up(cz, z) - cz) / dz - (exz - _dn(exz, x)) / dx - (eyz[:, 1:] - eyz[:, :-1]) * rdy
        fv = -(cy[:, 1:] - cy[:, :-1]) * rdyg[:, 1:-1] - ((exy - _dn(exy, x)) / dx + (eyz - _dn(eyz, z)) / dz)[:, 1:-1]

        def lap(f):
            return (_up(f, x) - 2 * f + _dn(f, x)) / dx ** 2 + (_up(f, z) - 2 * f + _dn(f, z)) / dz ** 2

        def dyc(fe):                                                # centres with ghosts
            g = (fe[:, 1:] - fe[:, :-1]) * rdyg
            return (g[:, 1:] - g[:, :-1]) * rdy

        g = (vf[:, 1:] - vf[:, :-1]) * rdy
        fu = fu + nu * (lap(u) + dyc(ue)) + dPdx
        fw = fw + nu * (lap(w) + dyc(we))
        fv = fv + nu * (lap(v) + (g[:, 1:] - g[:, :-1]) * rdyg[:, 1:-1])
        return fu, fv, fw

    def project(self, u, v, w):
        zero = torch.zeros_like(v[:, :1])
        vf = torch.cat([zero, v, zero], 1)
        div = (u - _dn(u, 2)) / self.dx + (vf[:, 1:] - vf[:, :-1]) * self.rdy + (w - _dn(w, 0)) / self.dz
        h = torch.fft.fft(torch.fft.rfft(div, dim=2), dim=0)        # (kz, y, kx)
        b = list(h.unbind(1))
        n = self.Ny
        d = [self.dd[j] + self.lam for j in range(n)]
        d[0] = d[0].clone()
        d[0][0, 0] *= 1.5
        for j in range(1, n):
            m = self.lo[j - 1] / d[j - 1]
            d[j] = d[j] - m * self.up[j - 1]
            b[j] = b[j] - m * b[j - 1]
        b[n - 1] = b[n - 1] / d[n - 1]
        for j in range(n - 2, -1, -1):
            b[j] = (b[j] - self.up[j] * b[j + 1]) / d[j]
        p = torch.fft.irfft(torch.fft.ifft(torch.stack(b, 1), dim=0), n=self.Nx, dim=2)
        u = u - (_up(p, 2) - p) / self.dx
        v = v - (p[:, 1:] - p[:, :-1]) * self.rdyg[:, 1:-1]
        w = w - (_up(p, 0) - p) / self.dz
        return u, v, w

    def flux(self, u):
        """Trapezoid between the first and last centre; plane 2 counts twice
        (the reference sums its periodic copy)."""
        s = u.sum(2)
        s = s.sum(0) + s[0]
        wy = 0.5 * (self.yg[2:-1] - self.yg[1:-2])
        q = ((s[1:] + s[:-1]) * wy).sum()
        return (q / (2.0 * wy.sum() * self.Nx * (self.Nz + 1))).item()


def _diag_exact(ch, u, v, w):
    c = ch.c
    U, V, W = _full(u, v, w)
    nxg, nzg, nz = c["Nx"] + 3, c["Nz"] + 3, c["Nz"] + 2
    t1 = 0.5 * (U[1:nzg - 2, :, 0:nxg - 3] + U[1:nzg - 2, :, 1:nxg - 2])
    Vk = V[1:nzg - 2, :, 1:nxg - 2]
    t2 = 0.5 * (Vk[:, 1:] + Vk[:, :-1])
    t2 = torch.cat([-t2[:, :1], t2, -t2[:, -1:]], 1)
    Wk = W[1:nzg - 2, :, 1:nxg - 2]
    nuv, nw = (nxg - 3) * (nzg - 3), (nxg - 3) * (nz - 2)
    st = {"Umean": t1, "Wmean": Wk, "U2mean": t1 * t1, "V2mean": t2 * t2, "W2mean": Wk * Wk,
          "UVmean": t1 * t2}
    st = {k: f.sum((0, 2)) / (nw if k[0] == "W" else nuv) for k, f in st.items()}
    y, yg, nu = ch.y, ch.yg, c["nu"]
    ly = float(y[-1] - y[0])

    def tau(m):
        t = nu * ((m[1] - m[0]) / (yg[1] - yg[0]) - (m[-1] - m[-2]) / (yg[-1] - yg[-2])) / ly
        return math.sqrt(t) if t >= 0 else math.nan

    st["utau"], st["wtau"] = tau(st["Umean"]), None
    st["Retau_u"], st["Retau_w"] = st["utau"] * ly / 2.0 / nu, None
    st["Qflow_x"], st["Qflow_z"] = ch.flux(u), None
    st["nonfinite"] = False
    vol = float((c["Nx"] + 1) * c["Ny"] * (c["Nz"] + 1))
    # interior boxes of the reference's loops
    boxes = {"U": U[1:-1, 1:-1, 1:-1], "V": V[1:-1, 1:-1, 1:-1], "W": W[1:-1, 1:-1, 1:-1]}
    mon = {"mean" + k: (boxes[k].sum() / vol).item() for k in "UW"}
    mon.update({"max" + k: f.max().item() for k, f in boxes.items()}, max_slip=0.0)
    return {"stats": st, "monitor": mon}


def _net_inputs(m, seed):
    """Parameters (W1 b1 W2 b2 W3 b3 of 32-128-128-16), features, moments
    (Crr 16, Cer 16, Cee 4 a row) and their scales, of the sizes training meets."""
    rng = np.random.default_rng(int(seed))
    n = rng.standard_normal
    p = [n(128 * 32) * math.sqrt(2.0 / 32), n(128) * 0.1, n(128 * 128) * math.sqrt(2.0 / 128), n(128) * 0.1,
         n(16 * 128) * 0.05, np.eye(4).ravel() + n(16) * 0.1]
    x = rng.uniform(-1.0, 1.0, (m, 32))
    r = n((m, 4, 6))
    crr = (r @ r.transpose(0, 2, 1) / 6).reshape(m, 16)
    cer = (n((m, 4, 4)) * 0.5 + np.eye(4)).reshape(m, 16)
    mom = np.concatenate([crr, cer, rng.uniform(0.5, 2.0, (m, 4))], axis=1)
    sig = rng.uniform(0.5, 2.0, 8)
    return tuple(a.astype(np.float32) for a in (np.concatenate(p), x, mom, sig))


def _net_exact(case, seed):
    params, x, mom, sig = (torch.from_numpy(a).double().to(_device()) for a in _net_inputs(case["rows"], seed))
    sizes = (128 * 32, 128, 128 * 128, 128, 16 * 128, 16)
    w1, b1, w2, b2, w3, b3 = params.split(sizes)
    w1, w2, w3 = w1.view(128, 32), w2.view(128, 128), w3.view(16, 128)
    h1 = torch.relu(x @ w1.T + b1)
    h2 = torch.relu(h1 @ w2.T + b2)
    out = h2 @ w3.T + b3
    a = out.view(-1, 4, 4)
    sr, se = sig[:4], sig[4:]
    crr = mom[:, :16].view(-1, 4, 4) / torch.outer(sr, sr)
    cer = mom[:, 16:32].view(-1, 4, 4) / torch.outer(se, sr)
    cee = (mom[:, 32:] / se ** 2).sum(1)
    ac = a @ crr
    loss = ((ac * a).sum((1, 2)) - 2 * (a * cer).sum((1, 2)) + cee).sum().item()
    go = (2.0 * (ac - cer)).view(-1, 16)
    g2 = (go @ w3) * (h2 > 0)
    g1 = (g2 @ w2) * (h1 > 0)
    grad = torch.cat([(g1.T @ x).flatten(), g1.sum(0), (g2.T @ h1).flatten(), g2.sum(0), (go.T @ h2).flatten(),
                      go.sum(0)])
    return {"out": out, "grad": grad, "loss": loss}
