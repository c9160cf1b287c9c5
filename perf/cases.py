"""The workloads this library is timed on, through its Python entry points.

A case is a model on a grid: what is integrated (`kind`), the grid
(nx, ny[, nz]; nz = 0 for a 2D field), the precision and the number of time
steps of one pass.  A pass is what a simulation does between two looks at its
field: one call that advances it, then the field itself (and the energies
where the call measures them).  The field stays with the model from pass to
pass, as in a running simulation.

Kinds
  solve    energy, then one Strang step, per iteration (the solve driver)
  real     Strang steps in real time; `omega` != 0 rotates the frame
  ground   Strang steps in imaginary time with unit-mass renormalisation, and
           the energies of the result
  rk4      classical Runge-Kutta with the 2/3 filter on the product
  be       preconditioned backward Euler, from the same starting field each pass
  adjoint  loss and gradients (potential, starting field) of a real-time run
  batch    independent 2D runs of mixed sizes, advanced together

Physics
  box      periodic box [0, 2 pi]^d without a potential, a phase field of 64
           seeded modes: superfluid turbulence
  trap     harmonic trap, Gaussian with a seeded phase imprint (2D: [-8, 8]^2;
           3D: [-10, 10]^3, anisotropic): a trapped condensate

FP32 models hand their fields on in complex64 (their own precision), FP64
models in complex128.
"""
import math

import numpy as np
import torch

import __graft_entry__

sfd = __graft_entry__.load_package()


def listed():
    return [
        # the smallest call: a solve loop over a small 2D trap, as in the
        # examples and tests; launches and host work decide
        dict(name="solve_2d_64_fp64", kind="solve", physics="trap", nx=64, ny=64, nz=0, precision="fp64", steps=4),
        # the 2D trapped condensate of the parity run, default precision
        dict(name="trap_2d_128_fp64", kind="real", physics="trap", nx=128, ny=128, nz=0, precision="fp64", steps=100),
        # a 2D box whose sides are not powers of two, FP32
        dict(name="box_2d_480x360_fp32", kind="real", physics="box", nx=480, ny=360, nz=0, precision="fp32",
             steps=100),
        # superfluid turbulence at 256^3, the headline workload: compensated
        # FP32, plain FP32, and the default precision
        dict(name="box_3d_256_fp32c", kind="real", physics="box", nx=256, ny=256, nz=256, precision="fp32",
             compensated=True, steps=50),
        dict(name="box_3d_256_fp32", kind="real", physics="box", nx=256, ny=256, nz=256, precision="fp32", steps=50),
        dict(name="box_3d_256_fp64", kind="real", physics="box", nx=256, ny=256, nz=256, precision="fp64", steps=10),
        # a rotating trapped condensate on a ragged 3D grid
        dict(name="rot_3d_64x48x56_fp64", kind="real", physics="trap", nx=64, ny=48, nz=56, precision="fp64",
             omega=0.5, steps=10),
        # the 3D ground-state search in imaginary time
        dict(name="ground_3d_128_fp64", kind="ground", physics="trap", nx=128, ny=128, nz=128, precision="fp64",
             steps=20),
        # explicit Runge-Kutta and backward Euler on a 3D field
        dict(name="rk4_3d_64_fp64", kind="rk4", physics="box", nx=64, ny=64, nz=64, precision="fp64", steps=8),
        dict(name="be_3d_64_fp64", kind="be", physics="trap", nx=64, ny=64, nz=64, precision="fp64", steps=4),
        # the gradient workload at its grid, a tenth of its time steps
        dict(name="adjoint_2d_256_fp64", kind="adjoint", physics="trap", nx=256, ny=256, nz=0, precision="fp64",
             steps=200),
        # a parameter scan: many small 2D runs together
        dict(name="batch_2d_64_128_256", kind="batch", physics="trap", runs64=64, runs128=48, runs256=16, steps=100),
    ]


def _length(rng, lo, hi, pow2):
    """An axis length in [lo, hi], spread over its logarithm: a power of two,
    or any length whose prime factors are at most 31 (odd ones among them)."""
    if pow2:
        a, b = int(math.log2(lo)), int(math.log2(hi))
        return 1 << rng.randint(a, b)
    while True:
        n = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
        m = n
        for p in (2, 3, 5, 7, 11, 13, 17, 19, 23, 29, 31):
            while m % p == 0:
                m //= p
        if m == 1:
            return n


def draw(rng):
    kind = rng.choice(["solve", "real", "real", "real", "ground", "rk4", "be", "adjoint", "batch"])
    if kind == "batch":
        return dict(kind=kind, physics="trap", runs64=rng.randint(0, 96), runs128=rng.randint(1, 48),
                    runs256=rng.randint(0, 16), steps=rng.randint(20, 100))
    if kind == "adjoint":
        n = rng.choice([64, 128, 256])
        return dict(kind=kind, physics="trap", nx=n, ny=rng.choice([64, 128, 256]), nz=0, precision="fp64",
                    steps=rng.randint(50, 200))
    precision = "fp64" if kind == "be" else rng.choice(["fp64", "fp64", "fp32"])
    pow2 = rng.random() < 0.5
    three = rng.random() < 0.6
    c = dict(kind=kind, physics="trap" if kind in ("ground", "be") else rng.choice(["trap", "box"]))
    if kind in ("rk4", "be"):
        lo, hi = (32, 128 if kind == "rk4" else 64) if three else (32, 256)
    else:
        lo, hi = (32, 256) if three else (32, 512)
    if pow2:
        hi = min(hi, 256)
    c["nx"], c["ny"] = _length(rng, lo, hi, pow2), _length(rng, lo, hi, pow2)
    c["nz"] = _length(rng, lo, hi, pow2) if three else 0
    c["precision"] = precision
    if kind == "real" and rng.random() < 0.3:
        c["omega"], c["physics"] = 0.5, "trap"
    elif kind == "real" and precision == "fp32" and pow2 and rng.random() < 0.5:
        c["compensated"] = True
    # steps: bounded by the cells advanced in a pass, so that no drawn case
    # costs more than the largest listed one
    cells = c["nx"] * c["ny"] * max(1, c["nz"])
    budget = 256 ** 3 * (10 if precision == "fp32" else 2)
    per = {"solve": 2, "real": 1, "ground": 1, "rk4": 8, "be": 16}[kind] * (1 if pow2 else 4)
    most = {"solve": 8, "real": 100, "ground": 50, "rk4": 16, "be": 4}[kind]
    c["steps"] = max(1, min(most, budget // (cells * per)))
    return c


# ------------------------------------------------------------------ inputs --
def _dev():
    return torch.device("cuda", 0)


def _shape(case):
    return (case["nx"], case["ny"]) + ((case["nz"],) if case["nz"] else ())


def _bounds(case):
    nd = len(_shape(case))
    if case["physics"] == "box":
        return ((0.0, 2 * math.pi),) * nd
    return ((-8.0, 8.0),) * 2 if nd == 2 else ((-10.0, 10.0),) * 3


def _coeffs(case):
    """coeffD, beta, and the trap frequencies of each axis (none: no trap)."""
    if case["physics"] == "box":
        xi = 0.05
        return -xi / math.sqrt(2.0), 1.0 / (math.sqrt(2.0) * xi), None
    return (-0.5, 500.0, (1.0, 1.0)) if len(_shape(case)) == 2 else (-0.5, 2000.0, (1.0, 1.0, 4.0))


def _dt(case):
    """The workload's time step, smaller where the grid's largest wavenumber
    would leave the splitting's (for RK4: the scheme's) stable range."""
    cD, _, _ = _coeffs(case)
    kin = sum(abs(cD) * (math.pi * n / (b[1] - b[0])) ** 2 for n, b in zip(_shape(case), _bounds(case)))
    if case["kind"] == "rk4":
        return min(1e-3, 1.0 / kin)
    return min(2.5e-3 if case["physics"] == "box" else 1e-3, 2.0 / kin)


def _axes(shape, bounds):
    out = []
    for a, (n, b) in enumerate(zip(shape, bounds)):
        x = torch.from_numpy(sfd.grid_coords(n, *b)).to(_dev())
        out.append(x.reshape([-1 if i == a else 1 for i in range(len(shape))]))
    return out


def _theta(rng, shape, bounds, count, kmax, sigma):
    """A phase field: `count` seeded cosine modes with 0 < |k| <= kmax."""
    unit = [2 * math.pi / (b[1] - b[0]) for b in bounds]
    reach = [int(kmax / u) for u in unit]
    coef = torch.zeros(shape, dtype=torch.complex128)
    for _ in range(count):
        while True:
            p = [int(rng.integers(-r, r + 1)) for r in reach]
            if 0 < sum((q * u) ** 2 for q, u in zip(p, unit)) <= kmax * kmax + 1e-12:
                break
        a, phi = rng.normal(0.0, sigma), rng.uniform(0.0, 2 * math.pi)
        coef[tuple(q % n for q, n in zip(p, shape))] += a * complex(math.cos(phi), math.sin(phi))
    return torch.fft.ifftn(coef.to(_dev())).real * float(np.prod(shape))


def _unit_mass(psi, bounds):
    cell = float(np.prod([(b[1] - b[0]) / n for n, b in zip(psi.shape, bounds)]))
    return psi / math.sqrt(float((psi.real ** 2 + psi.imag ** 2).sum()) * cell)


def _inputs(case, seed):
    """psi0 and V (None without a trap) on the GPU, in 64 bits."""
    rng = np.random.default_rng(seed)
    shape, bounds = _shape(case), _bounds(case)
    if case["physics"] == "box":
        theta = _theta(rng, shape, bounds, 64, 4.0, 0.3)
        return torch.polar(torch.ones_like(theta), theta), None
    X, gam = _axes(shape, bounds), _coeffs(case)[2]
    V = 0.5 * sum(g * x ** 2 for g, x in zip(gam, X))
    env = torch.exp(-0.5 * sum(math.sqrt(g) * x ** 2 for g, x in zip(gam, X)) * 0.5)
    theta = _theta(rng, shape, bounds, 16, 3.0, 0.05)
    return _unit_mass(torch.polar(env.expand(shape).contiguous(), theta), bounds), V


def _target(shape, bounds, seed):
    """A vortex dipole at a seeded place, unit mass."""
    rng = np.random.default_rng(seed + 7)
    X, Y = _axes(shape, bounds)
    x0, y0 = rng.uniform(1.0, 2.0), rng.uniform(-0.5, 0.5)
    amp = torch.exp(-(X ** 2 + Y ** 2) / 4) * torch.tanh(torch.hypot(X - x0, Y - y0) / 0.5) \
        * torch.tanh(torch.hypot(X + x0, Y - y0) / 0.5)
    return _unit_mass(torch.polar(amp, torch.atan2(Y - y0, X - x0) - torch.atan2(Y - y0, X + x0)), bounds)


def _host(t):
    """A GPU tensor as the library takes it: a numpy array, x fastest."""
    return t.permute(*reversed(range(t.dim()))).contiguous().cpu().numpy().T


def _batch_sizes(case):
    return [64] * case["runs64"] + [128] * case["runs128"] + [256] * case["runs256"]


def _batch_inputs(case, seed):
    """Per size: psi and V of its runs, stacked, and their betas."""
    rng = np.random.default_rng(seed)
    bounds = ((-8.0, 8.0),) * 2
    out = {}
    for n in (64, 128, 256):
        psi, V, beta = [], [], []
        X, Y = _axes((n, n), bounds)
        for _ in range(_batch_sizes(case).count(n)):
            a, b = rng.uniform(0.5, 2.0, size=2)
            v = 0.5 * (a * X ** 2 + b * Y ** 2)
            for _ in range(8):
                h, cx, cy = rng.uniform(0.0, 2.0), rng.uniform(-6.0, 6.0), rng.uniform(-6.0, 6.0)
                v = v + h * torch.exp(-((X - cx) ** 2 + (Y - cy) ** 2) / 0.5)
            theta = _theta(rng, (n, n), bounds, 16, 3.0, 0.05)
            env = torch.exp(-0.5 * (math.sqrt(a) * X ** 2 + math.sqrt(b) * Y ** 2))
            psi.append(_unit_mass(torch.polar(env, theta), bounds))
            V.append(v)
            beta.append(rng.uniform(100.0, 1000.0))
        if psi:
            out[n] = (torch.stack(psi), torch.stack(V), beta)
    return out


# ------------------------------------------------------------------- a pass --
def prepare(case, seed):
    if case["kind"] == "batch":
        sizes = _batch_sizes(case)
        b = sfd.BatchSplit2(sizes, [((-8.0, 8.0),) * 2] * len(sizes), coeffD=-0.5)
        r = 0
        for n, (psi, V, beta) in _batch_inputs(case, seed).items():
            psi, V = psi.transpose(1, 2).contiguous().cpu().numpy(), V.transpose(1, 2).contiguous().cpu().numpy()
            for p, v, g in zip(psi, V, beta):
                b.set_run(r, g, v.T, p.T)
                r += 1
        b.set_tuning(1, 0, 1)  # a fixed launch choice, so that runs are reproducible
        return dict(case=case, batch=b)
    shape, bounds = _shape(case), _bounds(case)
    cD, beta, _ = _coeffs(case)
    psi, V = _inputs(case, seed)
    f = sfd.Field(sfd.Grid(shape, bounds))
    f.phi = _host(psi)
    pot = sfd.PotentialZero(f) if V is None else sfd.PotentialArray(f, _host(V))
    p = sfd.GrossPitaevskiiParameters(pot, coeffD=cD, beta=beta, Omega=case.get("omega", 0.0))
    args = (f, p, _dt(case), case["steps"], max(1, case["steps"]))
    if case["kind"] == "rk4":
        n = sfd.NumModelGPRK(*args, stepper="RK4", filter="product", precision=case["precision"])
    elif case["kind"] == "be":
        n = sfd.NumModelBackwardEuler(*args, precision=case["precision"])
    else:
        n = sfd.NumModelSplit2(*args, precision=case["precision"], compensated=case.get("compensated", False))
    s = dict(case=case, model=n)
    if case["kind"] == "be":
        s["start"] = f.phi.copy(order="F")
    if case["kind"] == "adjoint":
        s["target"] = _host(_target(shape, bounds, seed))
    return s


def _own(phi, precision):
    """The field in the model's own precision."""
    return phi if precision == "fp64" else torch.from_numpy(phi).to(torch.complex64)


def run(state):
    case = state["case"]
    if case["kind"] == "batch":
        b = state["batch"]
        mass = b.step(case["steps"], 1e-3)
        fields = [_own(b.download(r), "fp32") for r in range(len(b.sizes))]
        return {"mass": mass, "fields": {str(n): torch.stack([f for f, m in zip(fields, b.sizes) if m == n])
                                         for n in sorted(set(b.sizes))}}
    n = state["model"]
    if case["kind"] == "solve":
        rows = sfd.solve(n)
        return {"energies": np.array([r[2:] for r in rows]), "phi": _own(n.f.phi, case["precision"])}
    if case["kind"] == "ground":
        d = n.step(case["steps"], imag=True, diag=True)
        return {"mass": d["mass"], "energies": np.array(d["energy"]), "phi": _own(n.f.phi, case["precision"])}
    if case["kind"] == "adjoint":
        loss, dV, g = n.adjoint(state["target"], case["steps"], K=50)
        return {"loss": loss, "dV": dV, "dpsi0": g}
    if case["kind"] == "be":
        n.f.phi = state["start"]
    sfd.timeStep(n, case["steps"])
    return {"phi": _own(n.f.phi, case["precision"])}


# --------------------------------------------------------------------- work --
def work(case):
    """Per time step every field is read and written once (the field does not
    fit on the chip with its neighbours' columns), the potential read once; two
    transforms of 5 N log2 N and some 30 operations per cell besides.  Energies
    are one more read and one more transform; a Runge-Kutta stage is a step
    with two more transforms (the filter); a backward-Euler step at least two
    applications of its operator; a gradient three steps' work."""
    if case["kind"] == "batch":
        cells = sum(n * n for n in _batch_sizes(case))
        size, logn = 4, 14
        per = 1.0
    else:
        cells = int(np.prod(_shape(case)))
        size, logn = (8 if case["precision"] == "fp64" else 4), math.log2(cells)
        per = {"solve": 1.5, "real": 1, "ground": 1, "rk4": 8, "be": 4, "adjoint": 3}[case["kind"]]
    steps = case["steps"] + (1 if case["kind"] == "solve" else 0)
    field = 2 * size * cells
    pot = size * cells if case["physics"] == "trap" else 0
    return {"bytes": per * steps * (2 * field + pot), "flops": per * steps * cells * (10 * logn + 30)}


# -------------------------------------------------------------------- exact --
class _Flow:
    """The equation on a grid in plain 64-bit torch."""

    def __init__(self, shape, bounds, cD, beta, V, omega=0.0):
        self.cD, self.beta, self.V, self.omega = cD, beta, 0.0 if V is None else V, omega
        self.nd = len(shape)
        self.cell = float(np.prod([(b[1] - b[0]) / n for n, b in zip(shape, bounds)]))
        X = _axes(shape, bounds)
        self.xi = []
        for a, (n, b) in enumerate(zip(shape, bounds)):
            k = torch.fft.fftfreq(n, d=1.0 / n, dtype=torch.float64, device=_dev()) * (2 * math.pi / (b[1] - b[0]))
            self.xi.append(k.reshape([-1 if i == a else 1 for i in range(self.nd)]))
        # per axis: the multiplier of cD Lap - Omega Lz
        self.mult = [cD * x ** 2 for x in self.xi]
        if omega:
            self.mult[0] = self.mult[0] - omega * X[1] * self.xi[0]
            self.mult[1] = self.mult[1] + omega * X[0] * self.xi[1]

    def lin(self, q, f):
        """Per axis, in order: transform, multiply by f(multiplier), back."""
        for a in range(self.nd):
            q = torch.fft.ifft(f(self.mult[a]) * torch.fft.fft(q, dim=a), dim=a)
        return q

    def lap(self, q):
        return sum(torch.fft.ifft(m * torch.fft.fft(q, dim=a), dim=a) for a, m in enumerate(self.mult))

    def dens(self, q):
        return q.real ** 2 + q.imag ** 2

    def strang(self, q, dt):
        half = lambda m: torch.exp(0.5j * dt * m)  # noqa: E731
        q = self.lin(q, half)
        q = q * torch.exp(-1j * dt * (self.V + self.beta * self.dens(q)))
        return self.lin(q, half)

    def strang_imag(self, q, dt):
        half = lambda m: torch.exp(0.5 * dt * m)  # noqa: E731
        q = self.lin(q, half)
        q = self.lin(q * torch.exp(-dt * (self.V + self.beta * self.dens(q))), half)
        return q / math.sqrt(float(self.dens(q).sum()) * self.cell)

    def energy(self, q):
        """E_Omega, E_Delta, E_beta, E, mu."""
        d, F, n = self.dens(q), [torch.fft.fft(q, dim=a) for a in range(self.nd)], q.shape
        kin = -sum(float((self.cD * x ** 2 * self.dens(f)).sum()) / m for x, f, m in zip(self.xi, F, n))
        rot = sum(float(((m - self.cD * x ** 2) * self.dens(f)).sum()) / k
                  for m, x, f, k in zip(self.mult, self.xi, F, n)) if self.omega else 0.0
        kin, rot = kin * self.cell, rot * self.cell
        ed = kin + float((self.V * d).sum()) * self.cell if torch.is_tensor(self.V) else kin
        eb = 0.5 * self.beta * float((d * d).sum()) * self.cell
        return [rot, ed, eb, -rot + ed + eb, -rot + ed + 2 * eb]

    def rk4(self, q, dt):
        lim = 4.0 / 9.0 * min(float((x ** 2).max()) for x in self.xi)
        keep = sum(x ** 2 for x in self.xi) < lim

        def rhs(u):
            t = (self.V + self.beta * self.dens(u)) * u
            return 1j * (self.lap(u) - torch.fft.ifftn(keep * torch.fft.fftn(t)))
        k1 = rhs(q)
        k2 = rhs(q + 0.5 * dt * k1)
        k3 = rhs(q + 0.5 * dt * k2)
        k4 = rhs(q + dt * k3)
        return q + dt / 6 * (k1 + 2 * k2 + 2 * k3 + k4)

    def backward_euler(self, q, dt, tol=1e-8, most=70):
        """(1 - M L) x = M q / dt, M = 1 / (1/dt + V + beta |q|^2), by BiCGStab
        from q to the scheme's own tolerance; then unit mass."""
        M = 1.0 / (1.0 / dt + self.V + self.beta * self.dens(q))
        A = lambda u: u - M * self.lap(u)  # noqa: E731
        dot = lambda u, v: float((u * v.conj()).real.sum())  # noqa: E731
        b, x = M * q / dt, q
        nb, r = math.sqrt(dot(b, b)), b - A(q)
        r0, p = r, r
        for _ in range(most):
            Ap, rr = A(p), dot(r, r0)
            al = rr / dot(Ap, r0)
            s = r - al * Ap
            As = A(s)
            om = dot(As, s) / dot(As, As)
            x, r = x + al * p + om * s, s - om * As
            if math.sqrt(dot(r, r)) / nb < tol:
                break
            p = r + dot(r, r0) / rr * al / om * (p - om * Ap)
        return x / math.sqrt(float(self.dens(x).sum()) * self.cell)


def exact(case, seed):
    if case["kind"] == "batch":
        mass, fields = [], {}
        for n, (q, V, beta) in _batch_inputs(case, seed).items():
            fl = _Flow((n, n), ((-8.0, 8.0),) * 2, -0.5, 0.0, None)
            k2 = 0.5j * 1e-3 * (fl.mult[0] + fl.mult[1])
            g = torch.tensor(beta, dtype=torch.float64, device=_dev()).reshape(-1, 1, 1)
            for _ in range(case["steps"]):
                q = torch.fft.ifft2(torch.exp(k2) * torch.fft.fft2(q))
                q = q * torch.exp(-1e-3j * (V + g * (q.real ** 2 + q.imag ** 2)))
                q = torch.fft.ifft2(torch.exp(k2) * torch.fft.fft2(q))
            mass += (q.real ** 2 + q.imag ** 2).sum(dim=(1, 2)).tolist()
            fields[str(n)] = q.cpu()
        return {"mass": np.array(mass), "fields": fields}
    shape, bounds = _shape(case), _bounds(case)
    cD, beta, _ = _coeffs(case)
    q, V = _inputs(case, seed)
    fl = _Flow(shape, bounds, cD, beta, V, case.get("omega", 0.0))
    dt, kind = _dt(case), case["kind"]
    host = lambda t: t.detach().cpu().numpy()  # noqa: E731
    if kind == "adjoint":
        V = V.clone().requires_grad_(True)
        q0 = q.clone().requires_grad_(True)
        fl.V, q = V, q0
        for _ in range(case["steps"]):
            q = fl.strang(q, dt)
        z = (_target(shape, bounds, seed).conj() * q).sum() * fl.cell
        loss = 1.0 - z.real ** 2 - z.imag ** 2
        loss.backward()
        return {"loss": float(loss), "dV": host(V.grad), "dpsi0": host(q0.grad)}
    rows = []
    for _ in range(case["steps"] + (1 if kind == "solve" else 0)):
        if kind == "solve":
            rows.append(fl.energy(q)[:4])
        q = {"solve": fl.strang, "real": fl.strang, "ground": fl.strang_imag, "rk4": fl.rk4,
             "be": fl.backward_euler}[kind](q, dt)
    if kind == "solve":
        return {"energies": np.array(rows), "phi": host(q)}
    if kind == "ground":
        mass = float(fl.dens(q).sum()) * fl.cell
        return {"mass": mass, "energies": np.array(fl.energy(q)), "phi": host(q)}
    return {"phi": host(q)}
