"""Workloads of the framework's public entry points, for timing and for checking results.

Each case is one call (or a short run of calls) that a user's program makes: the RK4 step
and rollout over the grid sizes, precisions, forcings and schemes that the solver is used
with, the RHS for a caller's own integrator, the rollout's adjoint, the 3-D transforms, the
spectral diagnostics, the coarse LES with the learned closure inside the step, and the
closure's training gradients.

``listed()`` names the fixed cases, ``draw(rng)`` gives more of the same ranges, ``prepare``
makes the inputs and what a program keeps (grid, RHS, parameters, model), ``run`` is one pass,
``exact`` the same outputs from plain torch in 64 bits, ``work`` the bytes and operations that
a pass cannot do without.  Fields are seeded random solenoidal velocities with the benchmark's
spectrum k^4 exp(-2 (k/4)^2) at u_rms = 1 on the 2 pi box, made by torch alone.
"""

import importlib
import math

import numpy as np
import torch

h3 = importlib.import_module("3dhit_b200")
closure = importlib.import_module("3dhit_b200.closure")
les = importlib.import_module("3dhit_b200.les")

DEVICE = "cuda"
LARGEST = 512**3  # points of the largest grid
STEPS_512 = 4     # steps of its rollout: the most expensive case


# ---------------------------------------------------------------------------
# cases
# ---------------------------------------------------------------------------

def listed():
    def flow(name, kind, n, steps, nu, forcing, dtype="float32", scheme="rk4"):
        nx, ny, nz = n
        return dict(name=name, kind=kind, nx=nx, ny=ny, nz=nz, steps=steps, nu=nu, forcing=forcing, dtype=dtype,
                    scheme=scheme)

    return [
        # a host loop over single steps on the smallest production grid (interactive use, a caller's
        # own time loop): every launch and every host call counts
        flow("step_32", "step", (32, 32, 32), 1, 0.02, "none"),
        # decaying turbulence on 32^3, the whole 100-step run as one rollout
        flow("rollout_32", "rollout", (32, 32, 32), 100, 0.02, "none"),
        # Lundgren forcing that holds the energy on 256^3: the 20 steps between two diagnostics
        flow("rollout_256_hold", "rollout", (256, 256, 256), 20, 1.5e-3, "hold"),
        # band-forced turbulence on 512^3, the headline throughput run, a few steps of it
        flow("rollout_512_band", "rollout", (512, 512, 512), STEPS_512, 6e-4, "band"),
        # a box with three different resolutions, linear forcing and the integrating-factor scheme
        flow("rollout_ragged_ifrk4", "rollout", (128, 64, 256), 13, 5e-3, "linear", scheme="ifrk4"),
        # the float64 run that a float32 result is checked against
        flow("rollout_f64_128", "rollout", (128, 128, 128), 5, 4e-3, "band", dtype="float64"),
        # one RHS for a caller's own integrator
        flow("rhs_256", "rhs", (256, 256, 256), 1, 1.5e-3, "band"),
        # the adjoint of a 20-step segment at 128^3 (one checkpoint interval of a long optimisation)
        flow("adjoint_128", "vjp", (128, 128, 128), 20, 4e-3, "linear"),
        # a field to the grid points and one back to its modes (initial fields, snapshots, statistics)
        flow("transforms_256", "transform", (256, 256, 256), 1, 0.0, "none"),
        # shell spectra and energy budget of a state, as a run samples them
        flow("diagnostics_256", "diagnostics", (256, 256, 256), 1, 1.5e-3, "band"),
        # the coarse LES with the learned closure evaluated inside the step, ten steps of its loop
        flow("les_64", "les", (64, 64, 64), 10, 1.5e-3, "hold"),
        # one training gradient of the closure on a batch of 16 snapshots of 64^3 points
        dict(name="closure_train", kind="train", points=16 * 64**3),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("rollout", "rollout", "rollout", "rollout", "step", "step", "rhs", "vjp", "vjp", "transform",
                       "diagnostics", "les", "train"))
    if kind == "train":
        return dict(kind=kind, points=16 * _log_int(rng, 64, 64**3))
    if kind == "les":
        n = rng.choice((32, 64, 128))
        shape = [n, n, n]
        if rng.random() < 0.4:
            shape[rng.randrange(2)] //= 2
        steps = _log_int(rng, 1, 20 if n <= 64 else 6)
        nu, scheme, dtype = _uniform_log(rng, 1e-3, 1e-2), "rk4", "float32"
        forcing = rng.choice(("hold", "linear", "none"))
    else:
        dtype = "float64" if rng.random() < 0.25 else "float32"
        largest = {"vjp": 2 * 128**3, "transform": 2 * 256**3}.get(kind, LARGEST)
        if dtype == "float64":
            largest = min(largest // 2, 256**3)
        base = 2 ** rng.randint(4, 9)
        shape = [base] * 3
        if rng.random() < 0.6:
            shape = [min(1024, max(8, int(base * rng.choice((0.25, 0.5, 1, 1, 2))))) for _ in range(3)]
        while shape[0] * shape[1] * shape[2] > largest:
            k = max(range(3), key=lambda i: (shape[i], rng.random()))
            shape[k] //= 2
        points = shape[0] * shape[1] * shape[2]
        most = {"rollout": 100, "vjp": 20}.get(kind, 1)
        cost = points * {"vjp": 16, "rollout": 1}.get(kind, 1) * (4 if dtype == "float64" else 1)
        most = max(1, min(most, STEPS_512 * LARGEST // cost))
        steps = _log_int(rng, 1, most) if most > 1 else 1
        nu = _uniform_log(rng, 6e-4, 2e-2)
        forcing = rng.choice(("none", "linear", "band", "hold") if kind != "vjp" else ("none", "linear", "band"))
        scheme = "ifrk4" if kind in ("rollout", "step") and rng.random() < 0.2 else "rk4"
    return dict(kind=kind, nx=shape[0], ny=shape[1], nz=shape[2], steps=steps, nu=nu, forcing=forcing, dtype=dtype,
                scheme=scheme)


def _uniform_log(rng, lo, hi):
    return float("%.3g" % math.exp(rng.uniform(math.log(lo), math.log(hi))))


# ---------------------------------------------------------------------------
# inputs (torch alone, from the seed)
# ---------------------------------------------------------------------------

def _rng(seed, salt):
    g = torch.Generator(device=DEVICE)
    g.manual_seed(int(seed) * 7919 + salt)
    return g


def _modes(case, dtype):
    """kx, ky, kz of the rfft layout, broadcast over it, and the 2/3 mask without k = 0."""
    ns = (case["nx"], case["ny"], case["nz"])
    ks = [torch.fft.fftfreq(n, 1.0 / n, device=DEVICE, dtype=dtype) for n in ns[:2]]
    ks.append(torch.arange(ns[2] // 2 + 1, device=DEVICE, dtype=dtype))
    kx, ky, kz = ks[0].view(-1, 1, 1), ks[1].view(1, -1, 1), ks[2].view(1, 1, -1)
    mask = (kx.abs() <= ns[0] // 3) & (ky.abs() <= ns[1] // 3) & (kz.abs() <= ns[2] // 3)
    mask[0, 0, 0] = False
    return kx, ky, kz, mask


def _weights(case, dtype):
    """How often an rfft plane stands in the full spectrum: 1 for kz = 0 and the Nyquist plane, else 2."""
    w = torch.full((case["nz"] // 2 + 1,), 2.0, device=DEVICE, dtype=dtype)
    w[0] = w[-1] = 1.0
    return w


def _real(case):
    return torch.float64 if case.get("dtype") == "float64" else torch.float32


def _field(case, seed, salt=0):
    """Solenoidal field in the 2/3 box, E(k) ~ k^4 exp(-2 (k/4)^2) of each wavenumber, u_rms = 1."""
    real = _real(case)
    shape = (3, case["nx"], case["ny"], case["nz"])
    u = torch.fft.rfftn(torch.rand(shape, generator=_rng(seed, salt), device=DEVICE, dtype=real) - 0.5, dim=(1, 2, 3))
    kx, ky, kz, mask = _modes(case, real)
    k2 = kx**2 + ky**2 + kz**2
    inv = torch.where(k2 > 0, 1.0 / k2, torch.zeros_like(k2))
    u *= mask * torch.sqrt(k2) * torch.exp(-k2 / 16.0)
    div = (kx * u[0] + ky * u[1] + kz * u[2]) * inv
    for c, k in enumerate((kx, ky, kz)):
        u[c] -= k * div
    n3 = float(case["nx"] * case["ny"] * case["nz"])
    a2 = sum((u[c].real.double() ** 2 + u[c].imag.double() ** 2).sum((0, 1)) for c in range(3))
    e = float((_weights(case, torch.float64) * a2).sum()) / (2 * n3 * n3)
    u *= math.sqrt(1.5 / e)
    return u


def _dt(case):
    # CFL 0.5 of a field whose largest |u| + |v| + |w| is 6 (u_rms = 1)
    return 0.5 * (2 * math.pi / max(case["nx"], case["ny"], case["nz"])) / 6.0


_A, _EPS, _BAND, _E = 0.1, 0.1, (1.0, 2.0), 1.5  # the forcings' settings


def _forcing(case):
    kind = case["forcing"]
    if kind == "linear":
        return h3.LinearForcing(A=_A)
    if kind == "band":
        return h3.BandForcing(eps=_EPS, kmin=_BAND[0], kmax=_BAND[1])
    if kind == "hold":
        return h3.HoldEnergyForcing(_E, case["nu"], tau=0.5)
    return h3.NoForcing()


def _mlp_weights(seed):
    """Initial weights of the closure (uniform in +-1/sqrt(fan in)), W1, b1 .. W4, b4."""
    g = torch.Generator().manual_seed(int(seed) + 17)
    out = []
    for i, o in ((9, 64), (64, 64), (64, 64), (64, 6)):
        b = 1.0 / math.sqrt(i)
        out.append(((torch.rand(i, o, generator=g) * 2 - 1) * b).to(DEVICE))
        out.append(((torch.rand(o, generator=g) * 2 - 1) * b).to(DEVICE))
    return out


# typical size of the filtered velocity gradients and of the subgrid stress
_X_SCALE, _Y_SCALE = 3.0, 0.02


def _model(seed):
    m = closure.ClosureMLP(torch.device(DEVICE, torch.cuda.current_device()))
    for p, w in zip(m.params, _mlp_weights(seed)):
        p.copy_(w)
    m.x_scale.fill_(_X_SCALE)
    m.y_scale.fill_(_Y_SCALE)
    return m


def _batch(case, seed):
    """Normalised gradients (P, 9) and stresses (P, 6) of a training batch."""
    g = _rng(seed, 5)
    x = torch.randn(case["points"], 9, generator=g, device=DEVICE)
    y = 0.4 * x[:, :6] * x[:, 3:9] + 0.8 * torch.randn(case["points"], 6, generator=g, device=DEVICE)
    return x, y


def _cotangent(case, seed, u):
    """dL/du of a loss on the final spectrum: a filter of a state-like field."""
    kx, ky, kz, _ = _modes(case, _real(case))
    n3 = float(case["nx"] * case["ny"] * case["nz"])
    return (u + 0.3 * _field(case, seed, salt=1)) * (_weights(case, _real(case)) / (1.0 + kx**2 + ky**2 + kz**2) / n3)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "train":
        x, y = _batch(case, seed)
        return dict(kind=kind, model=_model(seed), x=x, y=y)
    grid = h3.make_grid(case["nx"], case["ny"], case["nz"], dtype=_real(case))
    u = _field(case, seed)
    s = dict(kind=kind, grid=grid, u=u, dt=_dt(case), steps=case["steps"], scheme=case["scheme"],
             rhs=h3.make_ns_rhs(grid), params=h3.NSParams(nu=case["nu"], forcing=_forcing(case)))
    if kind == "vjp":
        s["ct"] = _cotangent(case, seed, u)
    elif kind == "transform":
        shape = (3, case["nx"], case["ny"], case["nz"])
        s["w"] = torch.rand(shape, generator=_rng(seed, 3), device=DEVICE, dtype=_real(case)) - 0.5
    elif kind == "les":
        s["step"] = les.FusedLESStep(grid, _model(seed), s["params"], s["dt"], fused=True)
    return s


def run(s):
    kind = s["kind"]
    if kind == "step":
        return h3.rk4_step(s["rhs"], s["u"], s["params"], s["dt"], 0.0, scheme=s["scheme"])
    if kind == "rollout":
        return h3.rollout(s["rhs"], s["u"], s["params"], s["dt"], s["steps"], scheme=s["scheme"])
    if kind == "rhs":
        return s["rhs"](s["u"], s["params"], 0.0)
    if kind == "vjp":
        return h3.rollout_vjp(s["rhs"], s["u"], s["params"], s["dt"], s["steps"], s["ct"])
    if kind == "transform":
        return h3.to_physical(s["u"], s["grid"]), h3.to_spectral(s["w"], s["grid"])
    if kind == "diagnostics":
        budget = h3.energy_budget(s["u"], s["grid"], s["params"].nu, s["params"].forcing)
        return budget, h3.energy_spectrum(s["u"], s["grid"]), h3.component_spectra(s["u"], s["grid"])
    if kind == "les":
        u = s["u"]
        for _ in range(s["steps"]):
            u = s["step"](u)
        return u
    m = s["model"]
    loss = m.loss_and_grads(s["x"], s["y"])
    return loss, [p.grad for p in m.params]


# ---------------------------------------------------------------------------
# the same outputs from plain torch in 64 bits
# ---------------------------------------------------------------------------

_DIMS = (-3, -2, -1)


class _Exact:
    """The solver in float64 with torch.fft."""

    def __init__(self, case):
        self.case = case
        self.shape = (case["nx"], case["ny"], case["nz"])
        self.n3 = float(case["nx"] * case["ny"] * case["nz"])
        self.kx, self.ky, self.kz, self.mask = _modes(case, torch.float64)
        self.k2 = self.kx**2 + self.ky**2 + self.kz**2
        self.inv = torch.where(self.k2 > 0, 1.0 / self.k2, torch.zeros_like(self.k2))
        self.w = _weights(case, torch.float64)
        # the band's edges are whole wavenumbers: exact in either precision
        self.band = (self.k2 >= _BAND[0] ** 2) & (self.k2 <= _BAND[1] ** 2)

    def phys(self, f):
        return torch.fft.irfftn(f, s=self.shape, dim=_DIMS)

    def spec(self, f):
        return torch.fft.rfftn(f, dim=_DIMS)

    def project(self, f):
        f = [c * self.mask for c in f]
        div = (self.kx * f[0] + self.ky * f[1] + self.kz * f[2]) * self.inv
        return [f[0] - self.kx * div, f[1] - self.ky * div, f[2] - self.kz * div]

    def sums(self, u, weight):
        return sum((weight * (c.real**2 + c.imag**2)).sum() for c in u) / (self.n3 * self.n3)

    def force(self, u, nu, A, eps):
        """The factor of u in the forcing term."""
        kind = self.case["forcing"]
        if kind == "linear":
            return A
        if kind == "band":
            return eps / self.sums(u, self.w * self.band) * self.band
        if kind == "hold":
            E, om = 0.5 * self.sums(u, self.w), 0.5 * self.sums(u, self.w * self.k2)
            return (2 * nu * om - (E - _E) / 0.5) / (2 * E)
        return None

    def rhs(self, u, nu, A=_A, eps=_EPS, viscous=True, f_ext=None):
        v = [self.phys(c) for c in u]
        curl = ((1, self.kz, 2, self.ky), (2, self.kx, 0, self.kz), (0, self.ky, 1, self.kx))
        w = [self.phys(1j * (kb * u[b] - ka * u[a])) for a, ka, b, kb in curl]
        n = [self.spec(v[(c + 1) % 3] * w[(c + 2) % 3] - v[(c + 2) % 3] * w[(c + 1) % 3]) for c in range(3)]
        del v, w
        f = self.force(u, nu, A, eps)
        if f is not None:
            n = [a + f * b for a, b in zip(n, u)]
        if f_ext is not None:
            n = [a + b for a, b in zip(n, f_ext)]
        n = self.project(n)
        return [a - nu * self.k2 * b for a, b in zip(n, u)] if viscous else n

    def step(self, u, dt, nu, A=_A, eps=_EPS, scheme="rk4", f_ext=None):
        def add(x, a, y):
            return [p + a * q for p, q in zip(x, y)]
        if scheme == "rk4":
            k = self.rhs(u, nu, A, eps, f_ext=f_ext)
            acc = k
            for a, b in ((0.5 * dt, 2.0), (0.5 * dt, 2.0), (dt, 1.0)):
                k = self.rhs(add(u, a, k), nu, A, eps, f_ext=f_ext)
                acc = add(acc, b, k)
            return add(u, dt / 6.0, acc)
        e = torch.exp(-0.5 * dt * nu * self.k2)
        k1 = self.rhs(u, nu, A, eps, viscous=False)
        eu = [e * c for c in u]
        k2 = self.rhs([a + 0.5 * dt * e * b for a, b in zip(eu, k1)], nu, A, eps, viscous=False)
        k3 = self.rhs(add(eu, 0.5 * dt, k2), nu, A, eps, viscous=False)
        k4 = self.rhs([e * (a + dt * b) for a, b in zip(eu, k3)], nu, A, eps, viscous=False)
        return [e * a + dt / 6.0 * (e * (e * b + 2 * c + 2 * d) + f) for a, b, c, d, f in zip(eu, k1, k2, k3, k4)]

    def sgs_force(self, u, weights):
        ks = (self.kx, self.ky, self.kz)
        x = torch.stack([self.phys(1j * k * c) for c in u for k in ks]).reshape(9, -1).T
        tau = _mlp(weights, x / _X_SCALE)[0].T * _Y_SCALE
        t = [self.spec(c.reshape(self.shape)) for c in tau]  # xx, yy, zz, xy, xz, yz
        rows = ((0, 3, 4), (3, 1, 5), (4, 5, 2))
        return self.project([-1j * sum(k * t[c] for k, c in zip(ks, row)) for row in rows])


def _mlp(weights, x):
    """Outputs of the closure (GELU in its tanh form) in float64."""
    a = x
    for i in range(4):
        z = a @ weights[2 * i] + weights[2 * i + 1]
        a = torch.nn.functional.gelu(z, approximate="tanh") if i < 3 else z
    return a, z


def _exact_train(case, seed):
    x, y = _batch(case, seed)
    w = [p.double().requires_grad_(True) for p in _mlp_weights(seed)]
    total = torch.zeros((), dtype=torch.float64, device=DEVICE)
    for xs, ys in zip(x.split(1 << 19), y.split(1 << 19)):
        loss = ((_mlp(w, xs.double())[0] - ys.double()) ** 2).sum() / y.numel()
        loss.backward()
        total += loss.detach()
    return total.reshape(1), [p.grad for p in w]


def _exact_vjp(case, ex, u, ct):
    from torch.utils.checkpoint import checkpoint
    u0 = u.clone().requires_grad_(True)
    scalars = [torch.tensor(v, dtype=torch.float64, device=DEVICE, requires_grad=True)
               for v in (case["nu"], _A, _EPS)]
    dt = _dt(case)

    def one(v, nu, A, eps):
        return torch.stack(ex.step(list(v), dt, nu, A, eps))

    v = u0
    for _ in range(case["steps"]):
        v = checkpoint(one, v, *scalars, use_reentrant=False)
    grads = torch.autograd.grad(v, [u0] + scalars, grad_outputs=ct, allow_unused=True)
    g = [0.0 if x is None else float(x.real) for x in grads[1:]]
    return grads[0], dict(zip(("nu", "A", "eps"), g))


def _exact_spectra(ex, u):
    smax = math.ceil(math.sqrt(3) * max(ex.shape) / 2) + 1
    shell = torch.floor(torch.sqrt(ex.k2) + 0.5).long().reshape(-1)
    comp = []
    for c in u:
        a2 = (ex.w * (c.real**2 + c.imag**2)).expand(ex.k2.shape).reshape(-1)
        comp.append(torch.bincount(shell, weights=a2, minlength=smax + 1)[1:smax + 1] / (2 * ex.n3 * ex.n3))
    comp = [c.cpu().numpy() for c in comp]
    ks = np.arange(1, smax + 1) * 1.0
    return (ks, comp[0] + comp[1] + comp[2]), (ks, *comp)


def exact(case, seed):
    kind = case["kind"]
    if kind == "train":
        return _exact_train(case, seed)
    ex = _Exact(case)
    u32 = _field(case, seed)
    if kind == "vjp":
        ct = _cotangent(case, seed, u32).to(torch.complex128)
        return _exact_vjp(case, ex, u32.to(torch.complex128), ct)
    u = [c.to(torch.complex128) for c in u32]
    nu, dt = case["nu"], _dt(case)
    with torch.no_grad():
        if kind == "transform":
            shape = (3, case["nx"], case["ny"], case["nz"])
            w = torch.rand(shape, generator=_rng(seed, 3), device=DEVICE, dtype=_real(case)) - 0.5
            return torch.stack([ex.phys(c) for c in u]), ex.spec(w.double())
        if kind == "diagnostics":
            E, om = 0.5 * ex.sums(u, ex.w), 0.5 * ex.sums(u, ex.w * ex.k2)
            f = ex.force(u, nu, _A, _EPS)
            if case["forcing"] == "band":
                P = torch.full_like(E, _EPS)
            else:
                P = torch.zeros_like(E) if f is None else 2.0 * f * E
            spec, comp = _exact_spectra(ex, u)
            return {"E": E, "eps": 2 * nu * om, "P": P}, spec, comp
        if kind == "rhs":
            return torch.stack(ex.rhs(u, nu))
        weights = [p.double() for p in _mlp_weights(seed)] if kind == "les" else None
        for _ in range(case["steps"]):
            f = ex.sgs_force(u, weights) if kind == "les" else None
            u = ex.step(u, dt, nu, scheme=case["scheme"], f_ext=f)
        return torch.stack(u)


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------

def work(case):
    """Inputs read once, outputs written once; the transforms at 2.5 N log2 N operations of a real
    3-D FFT and the pointwise arithmetic of each evaluation."""
    if case["kind"] == "train":
        p = case["points"]
        mults = 9 * 64 + 2 * 64 * 64 + 64 * 6
        return {"bytes": 4 * 15 * p, "flops": p * (3 * 2 * mults - 2 * 9 * 64)}
    n = case["nx"] * case["ny"] * case["nz"]
    real = 8 if case["dtype"] == "float64" else 4
    state = 3 * case["nx"] * case["ny"] * (case["nz"] // 2 + 1) * 2 * real
    fft = 2.5 * n * math.log2(n)
    rhs = 9 * fft + 60 * n
    kind, steps = case["kind"], case["steps"]
    if kind == "transform":
        return {"bytes": 2 * (state + 3 * n * real), "flops": 6 * fft}
    if kind == "diagnostics":
        return {"bytes": state, "flops": 10 * n}
    if kind == "rhs":
        return {"bytes": 2 * state, "flops": rhs}
    if kind == "vjp":  # forward and transpose of every stage
        return {"bytes": 3 * state, "flops": steps * 4 * (2 * rhs + 60 * n)}
    flops = steps * 4 * (rhs + 20 * n)
    if kind == "les":  # gradients, stress and closure once a step
        flops += steps * (15 * fft + n * 2 * (9 * 64 + 2 * 64 * 64 + 64 * 6))
    return {"bytes": 2 * state, "flops": flops}
