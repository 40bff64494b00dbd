"""Performance cases of the annulus time step: what users of this library run.

Kinds of case
  nonlin     the nonlinear pass (falcon_nonlin_dev, or the allocation-free
             falcon_nonlin_noalloc_dev) on fields already on the device, as a
             host that owns its own time loop calls it
  cheb       Chebyshev derivative transforms of device columns
             (falcon_cheb_fwd_dev, then falcon_cheb_d1d2_dev)
  run        a batch of instances: initial temperatures uploaded, `steps` time
             steps, every instance's fields and diagnostics read back
  monitor    the same with the diagnostics read after every step
  serve      requests through the serving loop until all are done

Fields have the library's layouts: X[r][m][b] on the device, Fortran
(Nm + 1, Nr) per instance on the host.
"""
import ctypes
import math
import os
import random
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "falcon-dns_gb300"))
import falcon_gpu as fg  # noqa: E402

ETA = 0.35


def listed():
    return [
        # one run's radial lines through the caller's own time loop: the smallest call
        dict(name="nonlin_one_run", kind="nonlin", nr=33, nm=42, nb=1, alloc=False),
        # half of the benchmark's uniform batch: many lines of Np = 510
        dict(name="nonlin_batch", kind="nonlin", nr=65, nm=170, nb=128, alloc=True),
        # the longest azimuthal grid (Ntheta = 1536), power-of-two factors
        dict(name="nonlin_long", kind="nonlin", nr=129, nm=512, nb=8, alloc=True),
        # an odd grid and batch (Np = 345 = 3 x 5 x 23)
        dict(name="nonlin_ragged", kind="nonlin", nr=49, nm=115, nb=37, alloc=True),
        # radial derivatives of one field of a batch of 64
        dict(name="cheb_derivatives", kind="cheb", nr=65, ncol=171 * 64),
        # the plain reference run: one small instance, latency of a step
        dict(name="run_plain", kind="run", nr=33, nm=42, scheme="CNAB2", n=1, steps=200, ra=1e5, dt=1e-5),
        # one larger instance with an IMEX Runge-Kutta scheme (Np = 1023)
        dict(name="run_single_large", kind="run", nr=97, nm=341, scheme="ARS443", n=1, steps=20, ra=1e8, dt=2e-7),
        # the uniform batch: a Rayleigh-number sweep on one grid
        dict(name="run_sweep", kind="run", nr=65, nm=170, scheme="SBDF3", n=256, steps=60, ra=1e7, dt=1e-6),
        # a small sweep of a fine radial grid
        dict(name="run_sweep_fine", kind="run", nr=129, nm=85, scheme="BPR353", n=16, steps=10, ra=1e6, dt=1e-7),
        # an uneven batch: four grids and three schemes, mixed Pr
        dict(name="run_mixed", kind="run", nr=0, nm=0, scheme="mixed", n=48, steps=10, ra=1e6, dt=0.0),
        # a small batch watched at every step
        dict(name="monitor_batch", kind="monitor", nr=33, nm=85, scheme="SBDF2", n=12, steps=50, ra=1e5, dt=2e-6),
        # a burst of requests through the serving loop
        dict(name="serve_burst", kind="serve", nr=33, nm=42, scheme="CNAB2", n=16, steps=40, ra=1e5, dt=5e-6),
    ]


def _loguniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 0.49)))))


def _largest_prime(n):
    p, big = 2, 1
    while n > 1:
        while n % p == 0:
            big, n = p, n // p
        p += 1
    return big


def _mode_count(rng, lo, hi):
    while True:  # azimuthal lengths 3 Nm with prime factors up to 61
        nm = _loguniform(rng, lo, hi)
        if _largest_prime(nm) <= 61:
            return nm


def draw(rng: random.Random):
    kind = rng.choice(("nonlin", "nonlin", "cheb", "run", "run", "run", "monitor", "serve"))
    if kind == "nonlin":
        nr, nm = _loguniform(rng, 9, 129), _mode_count(rng, 8, 512)
        most = max(1, min(256, 65 * 170 * 128 // (nr * nm)))
        return dict(kind=kind, nr=nr, nm=nm, nb=_loguniform(rng, 1, most), alloc=rng.random() < 0.75)
    if kind == "cheb":
        return dict(kind=kind, nr=_loguniform(rng, 9, 129), ncol=_loguniform(rng, 16, 24000))
    nr, nm = _loguniform(rng, 17, 113), _mode_count(rng, 12, 342)
    scheme = rng.choice(("CNAB2", "SBDF2", "SBDF3", "ARS443", "BPR353"))
    most = 12 if kind != "run" else max(1, min(128, 65 * 170 * 64 // (nr * nm)))
    n = _loguniform(rng, 1, most)
    steps = rng.randint(5, 30) if kind == "run" else rng.randint(10, 30)
    return dict(kind=kind, nr=nr, nm=nm, scheme=scheme, n=n, steps=steps, ra=10.0 ** rng.uniform(5.0, 7.0),
                dt=0.2 * _cfl(nr, nm))


def _radius(nr):
    i = np.arange(nr)
    return ETA / (1.0 - ETA) + 0.5 * (1.0 + np.cos((nr - 1 - i) * np.pi / (nr - 1)))


def _cfl(nr, nm):
    """The diffusive time scales of the grid (radial and azimuthal spacing squared)."""
    r = _radius(nr)
    dr = np.diff(r)
    return min(float(np.min(dr * dr)), float(np.min((2.0 / 3.0 * r * np.pi / nm) ** 2)))


def _instances(case):
    """(nr, nm, scheme, ra, pr, dt) of each instance of a run, monitor or serve case."""
    out = []
    for k in range(case["n"]):
        ra = case["ra"] * 10.0 ** (2.0 * ((k * 0.618034) % 1.0) - 1.0)
        if case["scheme"] == "mixed":
            nr, nm = ((33, 42), (65, 85), (65, 170), (97, 85))[k % 4]
            scheme = ("CNAB2", "SBDF3", "BPR353")[(k // 4) % 3]
            out.append((nr, nm, scheme, ra, (0.1, 1.0, 10.0)[(k // 12) % 3], 0.2 * _cfl(nr, nm)))
        else:
            out.append((case["nr"], case["nm"], case["scheme"], ra, 1.0, case["dt"]))
    return out


def _initial_temperature(case, seed):
    """Conductive profile plus complex noise on modes 1..Nm at interior radii
    (the library's own seeded initial state), every instance back to back."""
    rng = np.random.default_rng(seed)
    fields = []
    for nr, nm, *_ in _instances(case):
        t = np.zeros((nr, nm + 1), np.complex128)
        r = _radius(nr)
        t[:, 0] = np.log(r * (1.0 - ETA)) / math.log(ETA)
        noise = rng.standard_normal((nr - 2, nm, 2))
        t[1:-1, 1:] = 1e-3 * (noise[..., 0] + 1j * noise[..., 1])
        fields.append(t)
    return fields


def _flow_fields(case, seed):
    """T, omega, u_phi, u_r with the decaying azimuthal spectra of a developed
    flow and their usual magnitudes (T of order one, velocities 1e2, vorticity
    1e3), on the device as X[r][m][b]; mode 0 is real."""
    g = torch.Generator().manual_seed(int(seed))
    shape = (case["nr"], case["nm"] + 1, case["nb"])
    decay = torch.exp(-8.0 * torch.arange(shape[1], dtype=torch.float64) / case["nm"])[None, :, None]
    out = []
    for scale in (1.0, 1e3, 1e2, 1e2):
        x = torch.complex(torch.randn(shape, generator=g, dtype=torch.float64),
                          torch.randn(shape, generator=g, dtype=torch.float64)) * (scale * decay)
        x[:, 0].imag.zero_()
        out.append(x.to(_device()))
    return out


def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _params(case):
    return [fg.make_params(nr, nm, scheme, ra=ra, dt=dt, pr=pr) for nr, nm, scheme, ra, pr, dt in _instances(case)]


def prepare(case, seed):
    kind = case["kind"]
    if kind == "nonlin":
        fields = _flow_fields(case, seed)
        return dict(case=case, ins=fields, outs=[torch.empty_like(f) for f in fields])
    if kind == "cheb":
        g = torch.Generator().manual_seed(int(seed))
        x = torch.complex(torch.randn((case["ncol"], case["nr"]), generator=g, dtype=torch.float64),
                          torch.randn((case["ncol"], case["nr"]), generator=g, dtype=torch.float64))
        x = x.to(_device())
        return dict(case=case, x=x, spec=torch.empty_like(x), d1=torch.empty_like(x), d2=torch.empty_like(x))
    fields = _initial_temperature(case, seed)
    if kind == "serve":
        return dict(case=case, params=_params(case), fields=fields, server=fg.Server(16 << 30))
    total = sum(f.size for f in fields)
    pinned = lambda: torch.zeros(total, dtype=torch.complex128, pin_memory=True).numpy()  # noqa: E731
    start = pinned()
    start[:] = np.concatenate([f.ravel() for f in fields])
    b = fg.Batch(_params(case))
    return dict(case=case, batch=b, start=start, sizes=[f.size for f in fields],
                fields={k: pinned() for k in ("T", "omg", "up", "ur", "psi")})


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "nonlin":
        lib = fg.lib()
        f = lib.falcon_nonlin_dev if case["alloc"] else lib.falcon_nonlin_noalloc_dev
        stream = torch.cuda.current_stream().cuda_stream
        fg.check(f(case["nr"], case["nm"], case["nb"], *[x.data_ptr() for x in state["ins"] + state["outs"]], stream))
        return state["outs"]
    if kind == "cheb":
        lib = fg.lib()
        stream = torch.cuda.current_stream().cuda_stream
        x, spec, d1, d2 = (state[k].data_ptr() for k in ("x", "spec", "d1", "d2"))
        fg.check(lib.falcon_cheb_fwd_dev(case["nr"], case["ncol"], x, spec, stream))
        fg.check(lib.falcon_cheb_d1d2_dev(case["nr"], case["ncol"], spec, d1, d2, stream))
        return [state["spec"], state["d1"], state["d2"]]
    if kind == "serve":
        srv = state["server"]
        ids = [srv.submit_state(p, t, horizon=1 + case["steps"] * (k + 1) // case["n"])
               for k, (p, t) in enumerate(zip(state["params"], state["fields"]))]
        active, queued = srv.iterate()
        while active or queued:
            active, queued = srv.iterate()
        done = [srv.result(i) for i in ids]
        return {k: np.concatenate([d[3][k].ravel() for d in done]) for k in ("T", "omg", "up", "ur")}
    b = state["batch"]
    b.set_states(state["start"])
    if kind == "monitor":
        diags = []
        for _ in range(case["steps"]):
            b.step(1)
            diags.append(b.diagnostics_array())
        diag = np.concatenate(diags)
    else:
        b.step(case["steps"])
        diag = b.diagnostics_array()
    lib, at = fg.lib(), 0
    ptr = ctypes.POINTER(ctypes.c_double)
    for i, size in enumerate(state["sizes"]):
        into = [state["fields"][k][at:].ctypes.data_as(ptr) for k in ("T", "omg", "up", "ur", "psi")]
        fg.check(lib.falcon_batch_get_state(b.h, i, *into))
        at += size
    # time, dt are sums over the handle's whole life; the flow's values are this run's
    return dict(state["fields"], diag=np.stack([diag[k] for k in diag.dtype.names if k not in ("time", "dt")]))


STAGES = {"ARS443": 4, "BPR353": 4}


def work(case):
    kind = case["kind"]
    if kind == "nonlin":
        lines, p = case["nr"] * case["nb"], 3 * case["nm"]
        return dict(bytes=8 * lines * (case["nm"] + 1) * 16,
                    flops=lines * (4 * 5 * p * math.log2(p) + 4 * p))
    if kind == "cheb":  # a fast transform of each column and two back
        n, length = case["ncol"], 2 * case["nr"] - 2
        return dict(bytes=4 * n * case["nr"] * 16, flops=3 * n * 2.5 * length * math.log2(length))
    size, flops = 0, 0.0
    for k, (nr, nm, scheme, *_) in enumerate(_instances(case)):
        steps = 1 + case["steps"] * (k + 1) // case["n"] if kind == "serve" else case["steps"]
        p = 3 * nm
        nonlin = nr * (4 * 5 * p * math.log2(p) + 4 * p)
        # radial derivatives of two products, the temperature and the coupled omega-psi solves (one right-hand side)
        radial = 2 * 2 * nr * nr * 2 * (nm + 1)
        solves = 4 * 2 * nr * nr * 2 * (nm + 1)
        flops += steps * STAGES.get(scheme, 1) * (nonlin + radial + solves)
        size += nr * (nm + 1) * 16
    return dict(bytes=size * (5 if kind == "serve" else 6), flops=flops)


# ---------------------------------------------------------------------------
# The same results by plain torch in 64 bits
# ---------------------------------------------------------------------------
def _grid_products(t, w, up, ur, nm):
    """u_phi T, u_r T, u_phi omega, u_r omega over azimuthal grids of 3 Nm points (modes along axis 1)."""
    p = 3 * nm
    t, w, up, ur = (torch.fft.irfft(x, n=p, dim=1, norm="forward") for x in (t, w, up, ur))
    return [torch.fft.rfft(x, dim=1, norm="forward")[:, :nm + 1] for x in (up * t, ur * t, up * w, ur * w)]


def _chebyshev(nr):
    """Polynomials T_j, their first and second r-derivatives at the radii
    (interval length 1), with the halved end columns of the interpolant, and
    the values-to-coefficients matrix."""
    n = nr - 1
    x = np.cos((n - np.arange(nr)) * np.pi / n)
    t, d, d2 = np.zeros((3, nr, nr))
    t[:, 0], t[:, 1], d[:, 1] = 1.0, x, 1.0
    for j in range(2, nr):
        t[:, j] = 2.0 * x * t[:, j - 1] - t[:, j - 2]
        d[:, j] = 2.0 * t[:, j - 1] + 2.0 * x * d[:, j - 1] - d[:, j - 2]
        d2[:, j] = 4.0 * d[:, j - 1] + 2.0 * x * d2[:, j - 1] - d2[:, j - 2]
    h = np.ones(nr)
    h[[0, -1]] = 0.5
    to_coef = (t * (2.0 * h)[:, None]).T / n
    dev = _device()
    return [torch.as_tensor(a, device=dev) for a in (t * h, 2.0 * d * h, 4.0 * d2 * h, to_coef)]


ARS443_A = ([0] * 5, [1 / 2, 0, 0, 0, 0], [11 / 18, 1 / 18, 0, 0, 0], [5 / 6, -5 / 6, 1 / 2, 0, 0],
            [1 / 4, 7 / 4, 3 / 4, -7 / 4, 0])
ARS443_D = ([0] * 5, [0, 1 / 2, 0, 0, 0], [0, 1 / 6, 1 / 2, 0, 0], [0, -1 / 2, 1 / 2, 1 / 2, 0],
            [0, 3 / 2, -3 / 2, 1 / 2, 1 / 2])
BPR353_A = ([0] * 5, [1, 0, 0, 0, 0], [4 / 9, 2 / 9, 0, 0, 0], [1 / 4, 0, 3 / 4, 0, 0], [1 / 4, 0, 3 / 4, 0, 0])
BPR353_D = ([0] * 5, [1 / 2, 1 / 2, 0, 0, 0], [5 / 18, -1 / 9, 1 / 2, 0, 0], [1 / 2, 0, 0, 1 / 2, 0],
            [1 / 4, 0, 3 / 4, -1 / 2, 1 / 2])
TABLEAUS = {"ARS443": (ARS443_A, ARS443_D), "BPR353": (BPR353_A, BPR353_D)}
# implicit weight of the new level, weights of the old levels, explicit weights (constant time step)
MULTISTEP = {"CNAB2": (0.5, (0.5, 0.0), (1.5, -0.5)),
             "SBDF2": (2 / 3, (4 / 3, -1 / 3), (4 / 3, -2 / 3)),
             "SBDF3": (6 / 11, (18 / 11, -9 / 11, 2 / 11), (18 / 11, -18 / 11, 6 / 11))}


class _Annulus:
    """Instances of one (nr, nm, scheme, pr, dt), fields [instance, mode, radius]
    stepped in 64 bits with dense collocation operators."""

    def __init__(self, nr, nm, scheme, ra, pr, dt, t0):
        self.nm, self.scheme, self.pr, self.dt = nm, scheme, pr, dt
        dev = t0.device
        t, d, d2, to_coef = _chebyshev(nr)
        r = torch.as_tensor(_radius(nr), device=dev)
        m = torch.arange(nm + 1, device=dev, dtype=torch.float64)
        self.ra_pr = torch.as_tensor(ra, device=dev)[:, None, None] / pr
        wt = MULTISTEP[scheme][0] if scheme in MULTISTEP else 0.5
        lap = (d2 + d / r[:, None])[None] - (m[:, None] / r)[:, :, None].square() * t
        at = t - wt * dt / pr * lap
        at[:, [0, -1]] = t[[0, -1]]
        eye = torch.eye(nr, device=dev, dtype=torch.float64)
        self.solve_t = t @ torch.linalg.solve(at, eye.expand_as(at))
        au = t - wt * dt * (lap[0] - t / r[:, None].square())
        au[[0, -1]] = t[[0, -1]]
        self.solve_u = t @ torch.linalg.solve(au, eye)
        # unknowns psi, omega: lap psi + omega = 0 and omega - wt dt lap omega = rhs, psi = dpsi/dr = 0 at the walls
        af = torch.zeros(nm, 2 * nr, 2 * nr, device=dev, dtype=torch.float64)
        af[:, :nr, :nr], af[:, :nr, nr:] = lap[1:], t
        af[:, nr:, nr:] = t - wt * dt * lap[1:]
        af[:, [0, nr - 1, nr, 2 * nr - 1]] = 0.0
        af[:, [0, nr - 1], :nr], af[:, [nr, 2 * nr - 1], :nr] = t[[0, -1]], d[[0, -1]]
        rhs = torch.zeros(2 * nr, nr, device=dev, dtype=torch.float64)
        rhs[nr:] = eye
        x = torch.linalg.solve(af, rhs.expand(nm, -1, -1))
        self.solve_psi, self.solve_w, self.solve_up = t @ x[:, :nr], t @ x[:, nr:], -(d @ x[:, :nr])
        self.d1, self.d2 = d @ to_coef, d2 @ to_coef
        self.ir, self.imr = 1.0 / r, 1j * m[:, None] / r
        self.t = t0
        self.w, self.up, self.ur, self.psi = (torch.zeros_like(t0) for _ in range(4))
        self.products = [torch.zeros_like(t0) for _ in range(4)]
        self.n_step = 0

    @staticmethod
    def _apply(op, x):
        """A radial operator (or one per mode) on [instance, mode, radius]."""
        op = op.to(x.dtype)
        if op.dim() == 2:
            return x @ op.T
        return torch.einsum("mij,bmj->bmi", op, x)

    def _radial(self, x, square):
        """d2 x/dr2 + (1/r) dx/dr - square x"""
        return self._apply(self.d2, x) + self.ir * self._apply(self.d1, x) - square * x

    def _advection(self, up_x, ur_x):
        return self.imr * up_x + self._apply(self.d1, ur_x) + self.ir * ur_x

    def _nonlinear(self):
        fields = [x.transpose(1, 2).reshape(-1, self.nm + 1) for x in (self.t, self.w, self.up, self.ur)]
        shape = (self.t.shape[0], self.t.shape[2], self.nm + 1)
        self.products = [x.reshape(shape).transpose(1, 2) for x in _grid_products(*fields, self.nm)]

    def _set_temperature(self, rhs):
        rhs[:, :, [0, -1]] = 0.0
        rhs[:, 0, 0] = 1.0
        self.t = self._apply(self.solve_t, rhs)

    def _set_flow(self, rhs_u, rhs):
        rhs_u[:, [0, -1]] = 0.0
        u = rhs_u @ self.solve_u.T
        rhs = rhs[:, 1:].clone()
        rhs[:, :, [0, -1]] = 0.0
        for name, op in (("w", self.solve_w), ("up", self.solve_up), ("psi", self.solve_psi)):
            x = torch.zeros_like(self.t)
            x[:, 1:] = self._apply(op, rhs)
            setattr(self, name, x)
        self.ur = self.imr * self.psi
        self.up[:, 0] = u
        self.w[:, 0] = u * self.ir + u @ self.d1.T

    def step(self):
        if self.n_step:
            self._nonlinear()
        if self.scheme in MULTISTEP:
            self._multistep()
        else:
            self._runge_kutta()
        self.n_step += 1

    def _multistep(self):
        wt, w_old, w_exp = MULTISTEP[self.scheme]
        dt, crank = self.dt, self.scheme == "CNAB2"
        if not self.n_step:
            zero = lambda x, n: [torch.zeros_like(x) for _ in range(n)]  # noqa: E731
            self.old = [zero(self.t, 4), zero(self.t, 4), zero(self.up[:, 0].real, 4)]
            self.exp = [zero(self.t, 4), zero(self.t, 4), zero(self.up[:, 0].real, 4)]
        up_t, ur_t, up_w, ur_w = self.products
        u = self.up[:, 0].real
        m2 = self.imr.imag.square()
        rhs = []
        for k, (x, e, square, kappa) in enumerate(((self.t, self._advection(up_t, ur_t), m2, 1.0 / self.pr),
                                                   (self.w, self._advection(up_w, ur_w), m2, 1.0),
                                                   (u, ur_w[:, 0].real, self.ir.square(), 1.0))):
            self.old[k] = [x] + self.old[k][:-1]
            self.exp[k] = [e] + self.exp[k][:-1]
            if crank:
                y = x + 0.5 * dt * kappa * self._radial(x, square)
            else:
                y = sum(a * o for a, o in zip(w_old, self.old[k]))
            rhs.append(y - dt * sum(a * o for a, o in zip(w_exp, self.exp[k])))
        before = self.t
        self._set_temperature(rhs[0])
        buoyancy = -self.ra_pr * self.imr * (0.5 * (self.t + before) if crank else wt * self.t)
        self._set_flow(rhs[2], rhs[1] + dt * buoyancy)

    def _runge_kutta(self):
        a, d = TABLEAUS[self.scheme]
        dt, m2 = self.dt, self.imr.imag.square()
        t0, w0, u0 = self.t, self.w, self.up[:, 0].real
        exp, imp, buo = [], [], []
        for s in range(5):
            if s:
                part = [sum(a[s][i] * exp[i][k] + d[s][i] * imp[i][k] for i in range(s)) for k in range(3)]
                self._set_temperature(t0 + dt * part[0])
                buo.append(-self.ra_pr * self.imr * self.t)
                part[1] = part[1] + sum(d[s][i] * buo[i] for i in range(s + 1))
                self._set_flow(u0 + dt * part[2], w0 + dt * part[1])
                if sum(row[s] for row in a) + a[4][s] != 0.0:
                    self._nonlinear()
            else:
                buo.append(-self.ra_pr * self.imr * self.t)
            up_t, ur_t, up_w, ur_w = self.products
            u = self.up[:, 0].real
            exp.append((-self._advection(up_t, ur_t), -self._advection(up_w, ur_w), -ur_w[:, 0].real))
            imp.append((self._radial(self.t, m2) / self.pr, self._radial(self.w, m2),
                        self._radial(u, self.ir.square())))


def exact(case, seed):
    kind = case["kind"]
    if kind == "nonlin":
        return _grid_products(*_flow_fields(case, seed), case["nm"])
    if kind == "cheb":
        state = prepare(case, seed)
        t, d, d2, to_coef = (a.to(torch.complex128) for a in _chebyshev(case["nr"]))
        scale = math.sqrt(2.0 / (case["nr"] - 1))  # the library's normalisation of coefficients
        spec = state["x"] @ to_coef.T / scale
        return [spec, scale * (spec @ d.T), scale * (spec @ d2.T)]
    instances = _instances(case)
    fields = _initial_temperature(case, seed)
    groups = {}
    for k, (nr, nm, scheme, ra, pr, dt) in enumerate(instances):
        steps = 1 + case["steps"] * (k + 1) // case["n"] if kind == "serve" else case["steps"]
        groups.setdefault((nr, nm, scheme, pr, dt, steps), []).append(k)
    found = [None] * len(instances)
    for (nr, nm, scheme, pr, dt, steps), members in groups.items():
        t0 = torch.as_tensor(np.stack([fields[k].T for k in members]), device=_device())
        a = _Annulus(nr, nm, scheme, np.array([instances[k][3] for k in members]), pr, dt, t0)
        for _ in range(steps):
            a.step()
        for j, k in enumerate(members):
            found[k] = [x[j].T.cpu().numpy().ravel() for x in (a.t, a.w, a.up, a.ur, a.psi)]
    names = ("T", "omg", "up", "ur") if kind == "serve" else ("T", "omg", "up", "ur", "psi")
    out = {name: np.concatenate([f[i] for f in found]) for i, name in enumerate(names)}
    return out if kind == "serve" else dict(out, diag=None)
