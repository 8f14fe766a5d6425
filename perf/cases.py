"""The work that users of the solver have it do, as cases that can be timed and compared.

Every case goes through the package's public entry points.  Kinds of case:

  channel   a program steps a channel on the GPU and reads the fields, TIME and DELTA_T
            back as device arrays after a few RK3 steps ("flow" kh: a sheared layer
            between free-slip walls with scalars and buoyancy, fixed DELTA_T; "flow" wall:
            a pressure-driven channel between no-slip walls, DELTA_T from the CFL number)
  periodic  the same for the triply periodic solver
  host      the drop-in boundary: the state lives in the caller's pinned host arrays in the
            reference's layout, goes in, is stepped, comes back, and the statistics
            profiles of that state are taken
  ensemble  the server: requests of small sheared layers of mixed sizes are queued together,
            stepped and returned

exact() repeats a pass in 64 bits with plain torch, from the equations: explicit RK3 for the
nonlinear terms with 2/3-rule spectral derivatives in x and z and second-order differences
in y, Crank-Nicolson for the wall-normal viscous terms, and a pressure projection per substep.
"""
import math

import numpy as np
import torch

from diablo_b200 import configs, serve
from diablo_b200.grid import create_grid, grid_metrics
from diablo_b200.solver import Channel, Periodic

C128 = torch.complex128

# lengths that the mixed-precision transforms take
MIXED_LENGTHS = (16, 32, 48, 64, 96, 128, 192, 256, 384, 512)


# ------------------------------------------------------------------ the cases
def listed():
    return [
        # the smallest request of an ensemble study, one step at a time: launches and latency
        dict(name="kh_64x33x16_1step", kind="channel", flow="kh", nx=64, ny=33, nz=16, n_th=1,
             mixed=False, les=False, steps=1),
        # the Kelvin-Helmholtz run of the benchmark, fields read every 10 steps
        dict(name="kh_128x65x32", kind="channel", flow="kh", nx=128, ny=65, nz=32, n_th=1,
             mixed=False, les=False, steps=10),
        # the largest layer of the ensemble's range in mixed precision
        dict(name="kh_256x129x64_mixed", kind="channel", flow="kh", nx=256, ny=129, nz=64, n_th=1,
             mixed=True, les=False, steps=5),
        # odd sizes: lengths with a factor 5, an even number of rows, two scalars
        dict(name="kh_160x98x60_2th", kind="channel", flow="kh", nx=160, ny=98, nz=60, n_th=2,
             mixed=False, les=False, steps=2),
        # the headline: Re_tau = 180 channel, DELTA_T from COURANT on every step
        dict(name="wall_128x129x128", kind="channel", flow="wall", nx=128, ny=129, nz=128, n_th=0,
             mixed=False, les=False, steps=5),
        # the largest configuration: Re_tau ~ 550 with a passive scalar
        dict(name="wall_512x257x384_1th", kind="channel", flow="wall", nx=512, ny=257, nz=384,
             n_th=1, mixed=False, les=False, steps=1),
        # a mid-size wall-bounded run in mixed precision
        dict(name="wall_192x193x192_mixed", kind="channel", flow="wall", nx=192, ny=193, nz=192,
             n_th=0, mixed=True, les=False, steps=2),
        # the subgrid model at the headline size
        dict(name="les_wall_128x129x128", kind="channel", flow="wall", nx=128, ny=129, nz=128,
             n_th=0, mixed=False, les=True, steps=2),
        # decaying turbulence in a periodic box, the benchmark's size
        dict(name="periodic_256", kind="periodic", nx=256, ny=256, nz=256, n_th=0, mixed=False,
             steps=2),
        # a smaller box with a scalar in mixed precision
        dict(name="periodic_96x64x96_mixed", kind="periodic", nx=96, ny=64, nz=96, n_th=1,
             mixed=True, steps=5),
        # the host program owns the state: copies in and out on every step, statistics
        dict(name="host_128x129x128", kind="host", flow="wall", nx=128, ny=129, nz=128, n_th=0,
             mixed=False, les=False, steps=1),
        # six requests of an ensemble study, served together
        dict(name="ensemble_6", kind="ensemble", requests=6, sizes=11, steps=20),
    ]


def _smooth(lo, hi, step=2):
    """Lengths that the transforms take: even, with factors 2, 3 and 5."""
    out = []
    for n in range(lo, hi + 1, step):
        m = n
        for f in (2, 3, 5):
            while m % f == 0:
                m //= f
        if m == 1:
            out.append(n)
    return out


def _log_pick(rng, values):
    """One of the values, evenly over their logarithm."""
    x = math.exp(rng.uniform(math.log(values[0]), math.log(values[-1])))
    return min(values, key=lambda v: abs(math.log(v / x)))


def _steps(rng, points):
    return max(1, min(rng.choice((1, 2, 5, 10)), int(8e6 / points)))


def draw(rng):
    kind = rng.choice(("kh", "kh", "wall", "wall", "mixed", "mixed", "les", "les", "periodic",
                       "periodic", "host", "ensemble"))
    if kind == "ensemble":
        return dict(kind="ensemble", requests=rng.randint(2, 8), sizes=rng.randrange(1000),
                    steps=rng.randint(5, 30))
    if kind == "periodic":
        mixed = rng.random() < 0.5
        lengths = [n for n in MIXED_LENGTHS if n <= 256] if mixed else _smooth(16, 256)
        nx, ny, nz = (_log_pick(rng, lengths) for _ in range(3))
        return dict(kind="periodic", nx=nx, ny=ny, nz=nz, n_th=rng.choice((0, 0, 1)), mixed=mixed,
                    steps=_steps(rng, nx * ny * nz))
    mixed = kind == "mixed" or (kind == "les" and rng.random() < 0.25)
    big = 256 if kind in ("kh", "host") else 128 if kind == "les" else 512
    while True:
        some = list(MIXED_LENGTHS) if mixed else _smooth(16, 512)
        nx = _log_pick(rng, [n for n in some if 32 <= n <= big])
        nz = _log_pick(rng, [n for n in some if 16 <= n <= min(big, 384)])
        ny = round(math.exp(rng.uniform(math.log(17), math.log(257))))
        if nx * ny * nz <= 16e6:
            break
    flow = kind if kind in ("kh", "wall") else "wall" if kind == "host" else rng.choice(("kh", "wall"))
    return dict(kind="host" if kind == "host" else "channel", flow=flow, nx=nx, ny=ny, nz=nz,
                n_th=rng.choice((0, 1, 1, 2)), mixed=mixed, les=kind == "les",
                steps=1 if kind == "host" else _steps(rng, nx * ny * nz * (3 if kind == "les" else 1)))


def _params(case):
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    if case["kind"] == "periodic":
        p, gy = configs.periodic_256()
        p = p.replace(nx=nx, ny=ny, nz=nz, n_th=case["n_th"])
    elif case["flow"] == "kh":
        p, gy = configs.kh_shear_layer(nx, ny, nz)
        p = p.replace(n_th=case["n_th"])
        gy = create_grid(2, ny, 20.0, 1.5)
        p.ri[0], p.pr[1] = 0.1, 0.7
    else:
        p, gy = configs.channel_re180(nx, ny, nz)
        p = p.replace(n_th=case["n_th"])
        p.pr[0] = 0.71
    for n in range(case["n_th"]):
        p.th_bc_ymin_c1[n], p.th_bc_ymax_c1[n] = -1.0, 1.0
    return p.replace(precision=int(case["mixed"]), les=int(case.get("les", False))), gy


# ------------------------------------------------------------------ inputs
def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _draw_modes(gen, *shape):
    return torch.complex(torch.randn(*shape, generator=gen, dtype=torch.float64),
                         torch.randn(*shape, generator=gen, dtype=torch.float64))


def _waves(n, length, dev):
    """2 pi k / length for the packed retained modes 0..n/3, -n/3..-1."""
    k = n // 3
    return torch.tensor(list(range(k + 1)) + list(range(-k, 0)), dtype=torch.float64,
                        device=dev) * (2 * math.pi / length)


def _real_field(c, axes):
    """Modes of a real field: on kx = 0, the value at -k is the conjugate of the one at k."""
    z = c[..., 0]
    c[..., 0] = 0.5 * (z + torch.roll(torch.flip(z, axes), [1] * len(axes), axes).conj())
    return c


def _channel_modes(p, gy, seed, flow):
    """A developed flow before its projection: mean profile, and eddies that are smooth in y,
    vanish at the walls and fall off with the wavenumber."""
    dev = _device()
    gen = torch.Generator().manual_seed(int(seed))
    _, gyf, _, _ = grid_metrics(gy)
    y = torch.tensor(gyf, device=dev)
    lo, hi = float(gyf[1]), float(gyf[p.ny])
    eta = ((y - lo) / (hi - lo)).clamp(0, 1)
    shapes = torch.stack([torch.sin(math.pi * (m + 1) * eta) / (m + 1) for m in range(8)])
    kx, kz = _waves(p.nx, p.nx, dev)[: p.nkx + 1], _waves(p.nz, p.nz, dev)
    k = torch.sqrt((kx[None, :] * p.nx / 6.3) ** 2 + (kz[:, None] * p.nz / 6.3) ** 2)
    fall = torch.where(k > 0, (1 + k) ** -2.0, torch.zeros_like(k))
    if flow == "kh":
        mean, th_mean, amp, width = torch.tanh(y), torch.tanh(y), 0.05, torch.exp(-(y / 4) ** 2)
    else:
        mean, th_mean = 1.5 * p.ubulk0 * (1 - y.clamp(-1, 1) ** 2), y.clamp(-1, 1)
        amp, width = 0.1 * p.ubulk0, torch.ones_like(y)
    out = {}
    for name in ["CU1", "CU2", "CU3"] + ["CTH%d" % n for n in range(p.n_th)]:
        c = _real_field(_draw_modes(gen, 8, p.tnkz + 1, p.nkx + 1), [1]).to(dev) * fall
        f = torch.einsum("mzx,mj->jzx", c, (shapes * width).to(C128)).contiguous()
        f *= (amp if name[1] == "U" else 0.05) / 2
        if name == "CU1":
            f[:, 0, 0] += mean
        elif name[1] == "T":
            f[:, 0, 0] += th_mean
        out[name] = f
    return out


def _periodic_modes(p, seed):
    """Random phases with E(k) ~ k^4 exp(-2 (k/4)^2), r.m.s. of order one; a scalar alike."""
    dev = _device()
    gen = torch.Generator().manual_seed(int(seed))
    ky, kz = _waves(p.ny, p.ly, dev)[:, None, None], _waves(p.nz, p.lz, dev)[None, :, None]
    kx = _waves(p.nx, p.lx, dev)[None, None, : p.nkx + 1]
    k = torch.sqrt(kx ** 2 + ky ** 2 + kz ** 2)
    fall = 0.02 * k * torch.exp(-((k / 4) ** 2))
    return {n: _real_field(_draw_modes(gen, p.tnky + 1, p.tnkz + 1, p.nkx + 1).to(dev) * fall,
                           [0, 1]).contiguous()
            for n in ["CU1", "CU2", "CU3"] + ["CTH%d" % i for i in range(p.n_th)]}


def _requests(case):
    """Parameters of the ensemble's requests: sizes and physics of the served study."""
    rng = np.random.Generator(np.random.PCG64(case["sizes"]))
    out = []
    for _ in range(case["requests"]):
        p, _gy = _params(dict(kind="channel", flow="kh", nx=int(rng.choice([64, 128, 256])),
                              ny=int(rng.choice([33, 65, 129])), nz=int(rng.choice([16, 32, 64])),
                              n_th=1, mixed=False))
        p = p.replace(nu=1.0 / float(rng.uniform(500, 5000)))
        p.ri[0] = float(rng.uniform(0.05, 0.25))
        out.append((p, _gy))
    return out


def _names(p, pressure=True):
    return ["CU1", "CU2", "CU3"] + (["CP"] if pressure else []) + ["CTH%d" % n for n in range(p.n_th)]


# ------------------------------------------------------------------ state and pass
class _State:
    """What a program keeps between passes: the solver on the program's stream and its arrays."""

    solver = server = None

    def __del__(self):
        if self.solver is not None:
            self.solver.close()
        if self.server is not None:
            self.server.close()


def prepare(case, seed):
    s = _State()
    s.case, s.ts = case, 1
    if case["kind"] == "ensemble":
        s.todo = []
        for i, (p, gy) in enumerate(_requests(case)):
            modes = _channel_modes(p, gy, seed * 1000 + i, "kh")
            modes["CP"] = torch.zeros_like(modes["CU1"])
            s.todo.append((p, gy, {k: v.cpu().numpy() for k, v in modes.items()}))
        s.server = serve.Server(max_active=8, group_cases=4, autotune=False)
        return s
    p, gy = _params(case)
    s.p, s.stream = p, torch.cuda.Stream()
    periodic = case["kind"] == "periodic"
    modes = _periodic_modes(p, seed) if periodic else _channel_modes(p, gy, seed, case["flow"])
    torch.cuda.current_stream().synchronize()
    handle = s.stream.cuda_stream
    s.solver = ch = Periodic(p, stream=handle) if periodic else Channel(p, gy, stream=handle)
    for name, v in modes.items():
        ch.set_field_device(name, v.data_ptr())
    if periodic:
        ch.rem_div_per()
        ch.poisson_p_per()
    else:
        ch.apply_bc_vel()
        ch.rem_div_chan()
        ch.apply_bc_vel()
    ch.set_time(0.0, p.delta_t)
    ch.synchronize()
    s.out = {n: torch.empty_like(modes["CU1"]) for n in _names(p)}
    if case["kind"] == "host":
        shape = (p.ny + 2, p.nz + 2, p.nx // 2 + 1)
        s.host = {n: torch.zeros(shape, dtype=C128, pin_memory=True).numpy() for n in _names(p)}
        ch.get_fields(s.host, layout="reference_retained")
    return s


def run(s):
    case = s.case
    if case["kind"] == "ensemble":
        ids = [s.server.submit(p, gy, st, case["steps"]) for p, gy, st in s.todo]
        return [s.server.wait(i)[0] for i in ids]
    ch = s.solver
    if case["kind"] == "host":
        ch.set_fields(s.host, layout="reference_retained")
        ch.steps(s.ts, 1)
        s.ts += 1
        ch.get_fields(s.host, layout="reference_retained")
        prof = ch.save_stats()
        return {"state": s.host, "time": list(ch.get_time()),
                "profiles": {k: prof[k] for k in ("ume", "wme", "urms", "vrms", "wrms", "uv")}}
    ch.steps(s.ts, case["steps"])
    s.ts += case["steps"]
    for name, v in s.out.items():
        ch.get_field_device(name, v.data_ptr())
    out = s.out
    if case["mixed"]:
        # a mixed-precision run keeps its snapshots in single precision
        with torch.cuda.stream(s.stream):
            out = {n: v.to(torch.complex64) for n, v in out.items()}
    return {"state": out, "time": list(ch.get_time())}


# ------------------------------------------------------------------ what a pass cannot do without
def _step_work(p):
    """One RK3 step.  Each substep reads the fields, the pressure and (twice of three times) the
    old nonlinear terms and writes them; its transforms and solves are counted as operations."""
    nf = 3 + p.n_th
    rows = p.tnky + 1 if p.num_per_dir == 3 else p.ny + 2
    modes = rows * (p.tnkz + 1) * (p.nkx + 1)
    nbytes = 3 * 16 * modes * (2 * (nf + 1) + nf * 4 / 3)
    points = p.nx * p.ny * p.nz
    length = math.log2(p.nx * p.nz * (p.ny if p.num_per_dir == 3 else 1))
    forward = 6 + 3 * p.n_th if p.num_per_dir == 3 else 2 * nf
    flops = 3 * (2.5 * points * length * (nf + forward) + 100 * modes * nf)
    if p.les:  # strain rates and stresses: 9 + nf more to points, 7 + nf back; columns of points
        flops += 3 * (2.5 * points * length * (16 + 4 * nf) + 60 * points * (2 + nf))
    return nbytes, flops, 16 * modes * (nf + 1)


def work(case):
    if case["kind"] == "ensemble":
        each = [_step_work(p) for p, _ in _requests(case)]
        return {"bytes": sum(case["steps"] * b + 2 * s for b, _, s in each),
                "flops": sum(case["steps"] * f for _, f, _ in each)}
    b, f, state = _step_work(_params(case)[0])
    return {"bytes": case["steps"] * b + 2 * state, "flops": case["steps"] * f}


# ------------------------------------------------------------------ the same pass in plain torch
H_BAR, BETA_BAR, ZETA_BAR = (8 / 15, 2 / 15, 5 / 15), (1.0, 25 / 8, 9 / 4), (0.0, -17 / 8, -5 / 4)


def _solve(low, diag, up, rhs, j0, j1):
    """Tridiagonal solves along the first axis, rows j0..j1; the other axes broadcast."""
    d, g = [None] * (j1 + 1), [None] * (j1 + 1)
    d[j0], g[j0] = diag[j0], rhs[j0]
    for j in range(j0 + 1, j1 + 1):
        w = low[j] / d[j - 1]
        d[j] = diag[j] - w * up[j - 1]
        g[j] = rhs[j] - w * g[j - 1]
    x = rhs.clone()
    x[j1] = g[j1] / d[j1]
    for j in range(j1 - 1, j0 - 1, -1):
        x[j] = (g[j] - up[j] * x[j + 1]) / d[j]
    return x


class _PlainChannel:
    """Rows 0..NY+1 first: U1, U3, scalars and pressure at cell centres, U2 on faces."""

    def __init__(self, p, gy, modes):
        dev = modes["CU1"].device
        self.p, self.time, self.dt = p, 0.0, p.delta_t
        _, gyf, dy, dyf = grid_metrics(gy)
        col = lambda a: torch.tensor(a, device=dev)[:, None, None]  # noqa: E731
        self.dy, self.dyf, self.host_dy = col(dy), col(dyf), dy
        self.ikx = 1j * _waves(p.nx, p.lx, dev)[None, None, : p.nkx + 1]
        self.ikz = 1j * _waves(p.nz, p.lz, dev)[None, :, None]
        self.k2 = -(self.ikx ** 2 + self.ikz ** 2).real
        self.u = [modes[n].clone() for n in ("CU1", "CU2", "CU3")]
        self.th = [modes["CTH%d" % n].clone() for n in range(p.n_th)]
        self.cp = torch.zeros_like(self.u[0])
        self.f = [torch.zeros_like(self.cp) for _ in range(3 + p.n_th)]
        self.walls()
        self.project()
        self.walls()

    def to_points(self, c):
        nkz, p = self.p.nkz, self.p
        z = torch.zeros(c.shape[0], p.nz, p.nkx + 1, dtype=C128, device=c.device)
        z[:, : nkz + 1] = c[:, : nkz + 1]
        z[:, p.nz - nkz:] = c[:, nkz + 1:]
        return torch.fft.irfft(torch.fft.ifft(z, dim=1, norm="forward"), n=p.nx, dim=2, norm="forward")

    def to_modes(self, v):
        p, nkz = self.p, self.p.nkz
        z = torch.fft.fft(torch.fft.rfft(v, dim=2, norm="forward")[:, :, : p.nkx + 1], dim=1, norm="forward")
        return torch.cat([z[:, : nkz + 1], z[:, p.nz - nkz:]], dim=1)

    def walls(self):
        """Ghost and wall rows: no slip or no gradient for U1 and U3, no flow through for U2."""
        n = self.p.ny
        for u, kind in ((self.u[0], self.p.u_bc_ymin), (self.u[2], self.p.w_bc_ymin)):
            if kind == 0:
                u[:2] = 0
                u[n:] = 0
            else:
                u[1] = u[2]
                u[0] = u[1]
                u[n] = u[n - 1]
                u[n + 1] = u[n]
        v = self.u[1]
        v[1] = -v[2]
        v[0] = v[1]
        v[n + 1, 0, 0] = -v[n, 0, 0]

    def project(self):
        """Removes the divergence; returns phi (rows 1..NY)."""
        n, dy, dyf, u = self.p.ny, self.dy, self.dyf, self.u
        j = slice(1, n + 1)
        phi = torch.zeros_like(self.cp)
        div = self.ikx * u[0][j] + (u[1][2:n + 2] - u[1][j]) / dyf[j] + self.ikz * u[2][j]
        low, up = torch.zeros_like(self.k2.expand(n + 2, -1, -1)), torch.zeros_like(self.k2.expand(n + 2, -1, -1))
        diag = torch.ones_like(low)
        low[j] = (1 / (dy[j] * dyf[j])).expand_as(low[j])
        up[j] = (1 / (dy[2:n + 2] * dyf[j])).expand_as(up[j])
        diag[j] = -self.k2 - low[j] - up[j]
        phi[j] = div
        phi[1], phi[n] = 0, 0
        diag[1], up[1] = 1, -1
        up[1, 0, 0] = 0
        low[n], diag[n] = 1, -1
        phi = _solve(low, diag, up, phi, 1, n)
        u[0][j] -= self.ikx * phi[j]
        u[2][j] -= self.ikz * phi[j]
        i = slice(2, n + 1)
        u[1][i] -= (phi[i] - phi[1:n]) / dy[i]
        return phi

    def implicit(self, field, rhs, nu, nut, h, face, j0, low_wall, high_wall):
        """(1 - h/2 d/dy (nu + nut) d/dy) x = rhs on rows j0..NY of points; the wall rows hold a
        value (kind 0) or a zero gradient (kind 1)."""
        n, dy, dyf = self.p.ny, self.dy, self.dyf
        low = torch.zeros(n + 2, 1, 1, dtype=torch.float64, device=rhs.device)
        if nut is not None:
            low = low.expand_as(rhs).clone()
        up, diag, g = low.clone(), torch.ones_like(low), torch.zeros_like(rhs)
        j, jm, jp = slice(j0, n + 1), slice(j0 - 1, n), slice(j0 + 1, n + 2)
        if face:
            am, ap = 1 / (dyf[jm] * dy[j]), 1 / (dyf[j] * dy[j])
            vm, vp = (nu, nu) if nut is None else (nu + 0.5 * (nut[j] + nut[jm]), nu + 0.5 * (nut[j] + nut[jp]))
        else:
            am, ap = 1 / (dy[j] * dyf[j]), 1 / (dy[jp] * dyf[j])
            vm, vp = (nu, nu) if nut is None else (nu + nut[j], nu + nut[jp])
        low[j], up[j] = -0.5 * h * vm * am, -0.5 * h * vp * ap
        diag[j] = 1 + 0.5 * h * vm * am + 0.5 * h * vp * ap
        g[j] = rhs[j]

        def row(i, lo, di, hi, value):
            low[i], diag[i], up[i], g[i] = lo, di, hi, value

        row(0, 0, 1, 0, 0)
        if face:
            row(1, 0, 1, 0, 0)
            row(2, 0, 1, 0, 0)
            row(n, 0, 1, 0, 0)
            row(n + 1, 0, 1, 0, 0)
        else:
            row(1, *((0, 1, 0, low_wall[1]) if low_wall[0] == 0 else (0, -1, 1, 0)))
            row(n, *((0, 1, 0, high_wall[1]) if high_wall[0] == 0 else (-1, 1, 0, 0)))
            row(n + 1, 0, 1, 0, 0)
        x = _solve(low, diag, up, g, 0, n + 1)
        first = 1 if face else j0 - 1
        field[first:] = x[first:]

    def limit(self, u):
        """DELTA_T from the CFL number and the viscous and buoyancy limits."""
        p, n = self.p, self.p.ny
        dx, dz = p.lx / p.nx, p.lz / p.nz
        dt = min(999.0, 0.5 * min(dx, float(self.host_dy[1])) ** 2 / p.nu)
        for i in range(p.n_th):
            dt = min(dt, dt * p.pr[i])
            if p.ri[i] != 0:
                dt = min(dt, float(np.float32(0.1)) * 2 * math.pi / math.sqrt(abs(p.ri[i] * p.th_bc_ymin_c1[i])))
        j = slice(1, n + 1)
        for v, d in ((u[0], dx), (u[1], self.dy[j]), (u[2], dz)):
            dt = min(dt, float((p.cfl * d / v[j].abs()).min()))
        return dt

    def smagorinsky(self):
        """Constant Smagorinsky model: adds the explicit stress divergence to self.f, returns
        the eddy viscosity at faces and the velocity at points."""
        p, n, dy, dyf, ikx, ikz = self.p, self.p.ny, self.dy, self.dyf, self.ikx, self.ikz
        self.walls()
        u1, u2, u3 = self.u
        c = [torch.zeros_like(u1) for _ in range(6)]
        a, b = slice(1, n + 1), slice(2, n + 2)
        g, gm = slice(1, n + 2), slice(0, n + 1)
        c[0][a], c[2][a] = ikx * u1[a], ikz * u3[a]
        c[1][a] = (u2[b] - u2[a]) / dyf[a]
        c[4][a] = 0.5 * (ikz * u1[a] + ikx * u3[a])
        c[3][g] = 0.5 * ((u1[g] - u1[gm]) / dy[g] + ikx * u2[g])
        c[5][g] = 0.5 * (ikz * u2[g] + (u3[g] - u3[gm]) / dy[g])
        s = [self.to_points(x) for x in c]
        v = [self.to_points(x) for x in self.u]
        shear = []
        for q in (u1, u3):
            m = q[:, 0, 0].real.clone()[:, None, None]
            t = torch.zeros_like(m)
            t[g] = 0.5 * (m[g] - m[gm]) / dy[g]
            shear.append(t)
        j, jp, jm = slice(2, n + 1), slice(3, n + 2), slice(1, n)
        mid4 = 0.5 * ((s[3][jp] - shear[0][jp]) + (s[3][j] - shear[0][j]))
        mid6 = 0.5 * ((s[5][jp] - shear[1][jp]) + (s[5][j] - shear[1][j]))
        at_centre = torch.zeros_like(v[0])
        at_centre[j] = torch.sqrt(2 * (s[0][j] ** 2 + s[1][j] ** 2 + s[2][j] ** 2)
                                  + 4 * (mid4 ** 2 + s[4][j] ** 2 + mid6 ** 2))
        k, km = slice(2, n + 2), slice(1, n + 1)
        face = lambda x: (x[k] * dyf[km] + x[km] * dyf[k]) / (2 * dy[k])  # noqa: E731
        at_face = torch.zeros_like(v[0])
        at_face[k] = torch.sqrt(2 * (face(s[0]) ** 2 + face(s[1]) ** 2 + face(s[2]) ** 2)
                                + 4 * ((s[3][k] - shear[0][k]) ** 2 + face(s[4]) ** 2
                                       + (s[5][k] - shear[1][k]) ** 2))
        for i in (0, 2, 4):
            s[i][j] *= at_centre[j]
        for i, q in ((3, v[0]), (5, v[2])):
            s[i][k] = at_face[k] * (s[i][k] - 0.5 * (q[k] - q[km]) / dy[k])
        width = lambda d: -2 * 0.13 ** 2 * (p.lx / p.nx * d * 2 * p.lz / p.nz) ** (2 / 3)  # noqa: E731
        nut = torch.zeros_like(v[0])
        nut[3:n] = -0.5 * width(dy[3:n]) * at_face[3:n]
        t = [None if i == 1 else self.to_modes(x) for i, x in enumerate(s)]
        for i in (0, 2, 4):
            t[i][1:] *= width(dyf[1:])
        for i in (3, 5):
            t[i][2:] *= width(dy[2:])
        q, qp = slice(2, n), slice(3, n + 1)
        self.f[0][q] -= ikx * t[0][q] + (t[3][qp] - t[3][q]) / dyf[q] + ikz * t[4][q]
        self.f[2][q] -= ikx * t[4][q] + (t[5][qp] - t[5][q]) / dyf[q] + ikz * t[2][q]
        self.f[1][j] -= ikx * t[3][j] + ikz * t[5][j]
        for d, q in ((ikx, v[0]), (ikz, v[2])):
            x = torch.zeros_like(nut)
            x[j] = nut[j] * (q[j] - q[jm]) / dy[j]
            self.f[1][j] += d * self.to_modes(x)[j]
        # the ghost rows of the velocity at points
        for q, kind in ((v[0], p.u_bc_ymin), (v[2], p.w_bc_ymin)):
            if kind == 0:
                q[:2], q[n:] = 0, 0
            else:
                q[1] = q[2]
                q[0] = q[1]
                q[n] = q[n - 1]
                q[n + 1] = q[n]
        v[1][1] = -v[1][2]
        v[1][0] = v[1][1]
        v[1][n + 1] = -v[1][n]
        for i, th in enumerate(self.th):
            js = slice(self.first_row(i), n + 1)
            for d in (ikx, ikz):
                x = d * th
                x[0] = 0
                self.f[3 + i][js] += (d * self.to_modes(nut * self.to_points(x)))[js]
        return nut, v

    def first_row(self, i):
        return 1 if self.p.th_bc_ymin[i] == 1 else 2

    def substep(self, rk):
        p, n, dy, dyf, ikx, ikz = self.p, self.p.ny, self.dy, self.dyf, self.ikx, self.ikz
        h = self.dt * H_BAR[rk]
        j, jp, jm = slice(2, n + 1), slice(3, n + 2), slice(1, n)
        rhs = [x.clone() for x in self.u + self.th]
        if rk > 0:
            rhs = [r + ZETA_BAR[rk] * h * f for r, f in zip(rhs, self.f)]
        rhs[0] -= h * ikx * self.cp
        rhs[2] -= h * ikz * self.cp
        rhs[1][j] -= h * (self.cp[j] - self.cp[jm]) / dy[j]
        if p.f_type == 1:
            rhs[0][j, 0, 0] -= h * p.px0
        nus = [p.nu] * 3 + [p.nu / p.pr[i] for i in range(p.n_th)]
        self.f = [-nu * self.k2 * x for nu, x in zip(nus, self.u + self.th)]
        for i, th in enumerate(self.th):
            t = p.ri[i] * p.grav_y * (th[j] * dyf[jm] + th[jm] * dyf[j]) / (2 * dy[j])
            t[:, 0, 0] = 0
            self.f[1][j] += t
        nut = None
        if p.les:
            nut, v = self.smagorinsky()
        else:
            v = [self.to_points(x) for x in self.u]
        q = [self.to_points(x) for x in self.th]
        u1, u2, u3 = v
        c = torch.zeros_like(u1)

        def term(x, rows=j):
            y = c.clone()
            y[rows] = x
            return self.to_modes(y)

        def rise(a, rows):
            up, down = slice(rows.start + 1, rows.stop + 1), slice(rows.start - 1, rows.stop - 1)
            return term(((a[up] + a[rows]) * u2[up] - (a[rows] + a[down]) * u2[rows]) / (2 * dyf[rows]), rows)

        mix = lambda a: ((dyf[j] * a[j] + dyf[jm] * a[jm]) / (2 * dy[j])) * u2[j]  # noqa: E731
        t13 = term(u1[j] * u3[j])
        self.f[0] -= ikx * term(u1[j] ** 2) + ikz * t13 + rise(u1, j)
        self.f[2] -= ikx * t13 + ikz * term(u3[j] ** 2) + rise(u3, j)
        self.f[1] -= ikx * term(mix(u1)) + ikz * term(mix(u3)) + term(
            0.25 * ((u2[j] + u2[jp]) ** 2 - (u2[j] + u2[jm]) ** 2) / dy[j])
        for i, th in enumerate(q):
            js = slice(self.first_row(i), n + 1)
            self.f[3 + i] -= ikx * term(th[js] * u1[js], js) + ikz * term(th[js] * u3[js], js) + rise(th, js)
        walls = {0: (p.u_bc_ymin, p.u_bc_ymax), 2: (p.w_bc_ymin, p.w_bc_ymax)}
        for i in [1, 0, 2] + list(range(3, 3 + p.n_th)):
            x, nu, face = (v + q)[i], nus[i], i == 1
            j0 = 2 if i < 3 else self.first_row(i - 3)
            js, ju, jd = slice(j0, n + 1), slice(j0 + 1, n + 2), slice(j0 - 1, n)
            r = self.to_points(rhs[i] + BETA_BAR[rk] * h * self.f[i])
            if face:
                vm, vp = (nu, nu) if nut is None else (nu + 0.5 * (nut[js] + nut[jd]), nu + 0.5 * (nut[js] + nut[ju]))
                r[js] += 0.5 * h * (vp * (x[ju] - x[js]) / dyf[js] - vm * (x[js] - x[jd]) / dyf[jd]) / dy[js]
            else:
                vm, vp = (nu, nu) if nut is None else (nu + nut[js], nu + nut[ju])
                r[js] += 0.5 * h * (vp * (x[ju] - x[js]) / dy[ju] - vm * (x[js] - x[jd]) / dy[js]) / dyf[js]
            if i < 3:
                lo, hi = (((walls[i][0], 0.0), (walls[i][1], 0.0)) if i in walls else (None, None))
            else:
                lo = (p.th_bc_ymin[i - 3], p.th_bc_ymin_c1[i - 3])
                hi = (p.th_bc_ymax[i - 3], p.th_bc_ymax_c1[i - 3])
            self.implicit(x, r, nu, nut, h, face, j0, lo, hi)
        dt = self.limit(v) if p.variable_dt and rk == 2 else self.dt
        self.u = [self.to_modes(x) for x in v]
        self.th = [self.to_modes(x) for x in q]
        phi = self.project()
        self.cp[j] += phi[j] / h
        self.dt = dt

    def steps(self, count):
        for _ in range(count):
            for rk in range(3):
                self.substep(rk)
            self.time += self.dt

    def state(self, names):
        have = dict(zip(("CU1", "CU2", "CU3", "CP"), self.u + [self.cp]))
        have.update({"CTH%d" % i: t for i, t in enumerate(self.th)})
        return {k: have[k] for k in names}


class _PlainPeriodic:
    def __init__(self, p, modes):
        dev = modes["CU1"].device
        self.p, self.time, self.dt = p, 0.0, p.delta_t
        self.ik = [1j * _waves(p.nx, p.lx, dev)[None, None, : p.nkx + 1],
                   1j * _waves(p.ny, p.ly, dev)[:, None, None], 1j * _waves(p.nz, p.lz, dev)[None, :, None]]
        self.k2 = -sum(k ** 2 for k in self.ik).real
        self.small = float(np.float32(1e-9))
        self.u = [modes[n].clone() for n in ("CU1", "CU2", "CU3")]
        self.th = [modes["CTH%d" % n].clone() for n in range(p.n_th)]
        self.f = [0.0] * (3 + p.n_th)
        self.project()
        g = [[self.to_points(k * u) for k in self.ik] for u in self.u]
        t = g[0][0] ** 2 + g[0][0] * g[2][2] + g[2][2] ** 2
        t = t + g[0][1] * g[1][0] + g[0][2] * g[2][0] + g[1][2] * g[2][1]
        self.cp = self.to_modes(2 * t) / (self.k2 + self.small)
        self.cp[0, 0, 0] = 0

    def to_points(self, c):
        p = self.p
        full = torch.zeros(p.ny, p.nz, p.nkx + 1, dtype=C128, device=c.device)
        iy = list(range(p.nky + 1)) + list(range(p.ny - p.nky, p.ny))
        iz = list(range(p.nkz + 1)) + list(range(p.nz - p.nkz, p.nz))
        full[torch.tensor(iy)[:, None], torch.tensor(iz)[None, :]] = c
        return torch.fft.irfft(torch.fft.ifft2(full, dim=(0, 1), norm="forward"), n=p.nx, dim=2, norm="forward")

    def to_modes(self, v):
        p = self.p
        c = torch.fft.fft2(torch.fft.rfft(v, dim=2, norm="forward")[:, :, : p.nkx + 1], dim=(0, 1), norm="forward")
        c = torch.cat([c[: p.nky + 1], c[p.ny - p.nky:]], dim=0)
        return torch.cat([c[:, : p.nkz + 1], c[:, p.nz - p.nkz:]], dim=1)

    def project(self):
        phi = -sum(k * u for k, u in zip(self.ik, self.u)) / (self.k2 + self.small)
        self.u = [u - k * phi for k, u in zip(self.ik, self.u)]
        return phi

    def steps(self, count):
        p = self.p
        for _ in range(count):
            for rk in range(3):
                h = self.dt * H_BAR[rk]
                nus = [p.nu] * 3 + [p.nu / p.pr[i] for i in range(p.n_th)]
                rhs = [(1 - 0.5 * h * nu * self.k2) * x + ZETA_BAR[rk] * h * f
                       for nu, x, f in zip(nus, self.u + self.th, self.f)]
                v = [self.to_points(x) for x in self.u + self.th]
                self.f = [-sum(k * self.to_modes(v[i] * x) for k, x in zip(self.ik, v[:3])) for i in range(len(v))]
                for i in range(p.n_th):
                    self.f[1] = self.f[1] + p.ri[i] * self.th[i]
                rhs = [r - h * k * self.cp if i < 3 else r
                       for i, (r, k) in enumerate(zip(rhs, self.ik + [0.0] * p.n_th))]
                new = [(r + BETA_BAR[rk] * h * f) / (1 + 0.5 * h * nu * self.k2)
                       for r, f, nu in zip(rhs, self.f, nus)]
                self.u, self.th = new[:3], new[3:]
                self.cp = self.cp + self.project() / h
            self.time += self.dt

    state = _PlainChannel.state


def exact(case, seed):
    if case["kind"] == "ensemble":
        out = []
        for i, (p, gy) in enumerate(_requests(case)):
            q = _PlainChannel(p, gy, _channel_modes(p, gy, seed * 1000 + i, "kh"))
            q.steps(case["steps"])
            out.append({k: v.cpu().numpy() for k, v in q.state(serve.state_names(p)).items()})
        return out
    p, gy = _params(case)
    if case["kind"] == "periodic":
        q = _PlainPeriodic(p, _periodic_modes(p, seed))
    else:
        q = _PlainChannel(p, gy, _channel_modes(p, gy, seed, case["flow"]))
    q.steps(case["steps"])
    state = q.state(_names(p))
    if case["kind"] != "host":
        return {"state": state, "time": [q.time, q.dt]}
    shape = (p.ny + 2, p.nz + 2, p.nx // 2 + 1)
    host = {}
    for k, v in state.items():
        host[k] = np.zeros(shape, dtype=np.complex128)
        host[k][:, : p.tnkz + 1, : p.nkx + 1] = v.cpu().numpy()
    # the statistics' wall rows follow their own conventions: no values for the profiles here
    return {"state": host, "time": [q.time, q.dt],
            "profiles": {k: None for k in ("ume", "wme", "urms", "vrms", "wrms", "uv")}}
