"""FP64 fields above 2^18 cells, whose passes hold a whole, a half or a quarter
line per thread (smaller fields run others): every line length of the
register passes from 16 to 256 along x and along the strided axes."""
import numpy as np
import pytest

from helpers import random_field, run_model

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _lib(built_lib):
    return built_lib


BOUNDS = ((0.0, 3.0), (-1.0, 4.0), (-2.0, 2.0))
CD, DT = -0.31, 2.3e-3
SHAPES = [(16, 128, 256), (256, 32, 64), (64, 64, 128), (128, 256, 16), (32, 256, 64), (256, 16, 128), (2, 1024, 256),
          (256, 256, 8), (128, 4, 1024)]


def line_flow(v, n, b):
    """F^-1 exp(i cD xi^2 dt) F of one line, in long double."""
    xi = np.fft.fftfreq(n, d=1.0 / n) * ((6.283185307179586 / ((b[1] - b[0]) / n)) / n)
    return np.fft.ifft(np.fft.fft(v.astype(np.clongdouble)) * np.exp(np.clongdouble(1j) * (CD * (xi * xi) * DT)))


@pytest.mark.parametrize("shape", SHAPES)
def test_linear_step(sfd, shape):
    """One linear Strang step of a product of three random lines, whose flow is the
    product of theirs."""
    rng = np.random.default_rng(sum(shape))
    lines = [rng.standard_normal(n) + 1j * rng.standard_normal(n) for n in shape]
    lines[0] = lines[0] * 10.0 ** rng.uniform(-9, 0, shape[0])  # the strided lines differ in size
    psi = np.asfortranarray(np.einsum("i,j,k->ijk", *lines))
    got = run_model(sfd, shape, BOUNDS, psi, coeffD=CD, beta=0.0, dt=DT, nsteps=1)
    want = np.einsum("i,j,k->ijk", *[line_flow(v, n, b).astype(np.complex128) for v, n, b in zip(lines, shape, BOUNDS)])
    # six passes at 1.1e-16 + 0.45e-16 (1024-cell lines); the products of three
    # rounded lines here: five roundings of 1.6e-16 on either side
    assert np.linalg.norm(got - want) < (6 * 1.55e-16 + 2 * 5 * 1.6e-16) * np.linalg.norm(want)


@pytest.mark.parametrize("beta,vmax,dt", [(20.0, 0.0, 1e-3), (-20.0, 3.0, 0.4), (20.0, 3.0, -0.05)])
@pytest.mark.parametrize("shape", [(256, 256, 16), (256, 128, 32), (128, 128, 64), (256, 16, 128), (16, 128, 256)])
def test_nonlinear_flow(sfd, shape, beta, vmax, dt):
    """exp(-i (V + beta |psi|^2) dt) psi alone (coeffD = 0), in the last axis's
    pass: lines of 16 to 256 cells."""
    rng = np.random.default_rng(7 * sum(shape))
    psi = np.asfortranarray(rng.standard_normal(shape) + 1j * rng.standard_normal(shape))
    V = np.asfortranarray(rng.uniform(-vmax, vmax, shape)) if vmax else None
    got = run_model(sfd, shape, BOUNDS, psi, coeffD=0.0, beta=beta, V=V, dt=dt, nsteps=1)
    rho = np.abs(psi) ** 2
    theta = ((0.0 if V is None else V) + beta * rho) * dt
    want = psi * np.exp(-1j * theta)
    # six passes as above at 256 cells (1.27e-16); theta from |psi|^2 after three
    # of them (2 x 3 x 1.27e-16 of it) and from the FP64 expression here (5 x
    # 1.1e-16); exp and product here 4e-16
    w = np.abs(psi) / np.linalg.norm(psi)
    size = float(np.linalg.norm(w * np.abs(beta * dt) * rho)) + abs(vmax * dt)
    assert np.linalg.norm(got - want) < (6 * 1.27e-16 + 4e-16 + 1.4e-15 * size) * np.linalg.norm(want)


def test_rotation_step(sfd, O):
    """A rotating trap: passes with a phase row per line."""
    for shape in ((64, 128, 64), (256, 128, 16), (32, 16, 1024)):
        b = ((-5.0, 5.0), (-4.0, 4.0), (-3.0, 3.0))
        psi, V = random_field(shape, seed=5), O.quadratic_potential(shape, b)
        kw = dict(coeffD=-0.5, beta=4.0, omega=0.6, V=V, dt=1e-3, nsteps=2)
        for imag in (False, True):
            got = run_model(sfd, shape, b, psi, imag=imag, **kw)
            assert O.rel_l2(got, O.c_step(psi, b, imag=imag, **kw)) < 1e-12


@pytest.mark.parametrize("shape", [(128, 64, 64), (64, 128, 256), (32, 256, 64)])
def test_rk4_step_with_the_filter(sfd, O, shape):
    """Multiplier, accumulating, mask, forward and inverse passes."""
    b = ((-5.0, 5.0), (-4.0, 4.0), (-3.0, 3.0))
    psi, V = 0.5 * random_field(shape, seed=9), O.quadratic_potential(shape, b)
    for omega in (0.0, 0.4):
        f = sfd.Field(sfd.Grid(shape, b))
        f.phi = psi
        p = sfd.GrossPitaevskiiParameters(sfd.PotentialArray(f, V), coeffD=-0.5, beta=2.0, Omega=omega)
        n = sfd.NumModelGPRK(f, p, 1e-4, 2, 2, stepper="RK4", filter="product")
        n.step(2)
        got = f.phi.copy(order="F")
        n.close()
        want = O.c_rk_step(psi, b, V=V, coeffD=-0.5, beta=2.0, omega=omega, dt=1e-4, nsteps=2, stepper="RK4",
                           filter="product")
        assert O.rel_l2(got, want) < 1e-12


def test_energies(sfd, O):
    """The read-only passes, with rotation sums and without."""
    shape, b = (128, 64, 64), ((-5.0, 5.0), (-4.0, 4.0), (-3.0, 3.0))
    psi, V = random_field(shape, seed=11), O.quadratic_potential(shape, b)
    for omega in (0.0, 0.4):
        f = sfd.Field(sfd.Grid(shape, b))
        f.phi = psi
        p = sfd.GrossPitaevskiiParameters(sfd.PotentialArray(f, V), coeffD=-0.5, beta=2.0, Omega=omega)
        n = sfd.NumModelSplit2(f, p, 1e-3, 1, 1)
        got = np.array(n.energies())
        n.close()
        want = np.array(O.c_energy(psi, b, V=V, coeffD=-0.5, beta=2.0, omega=omega))
        assert np.max(np.abs(got - want)) < 1e-12 * np.max(np.abs(want))


@pytest.mark.parametrize("shape", [(64, 64, 128), (128, 16, 256)])
def test_adjoint(sfd, shape):
    """The gradients of two Strang steps against their FP64 adjoint written out with numpy's transforms."""
    b = ((-5.0, 5.0), (-4.0, 4.0), (-3.0, 3.0))
    cD, beta, dt, T = -0.5, 3.0, 1e-2, 2
    psi, tgt = random_field(shape, seed=12), random_field(shape, seed=13)
    V = np.asfortranarray(np.random.default_rng(1).uniform(0.0, 4.0, shape))
    dV = np.prod([(c[1] - c[0]) / n for n, c in zip(shape, b)])
    f = sfd.Field(sfd.Grid(shape, b))
    f.phi = psi
    p = sfd.GrossPitaevskiiParameters(sfd.PotentialArray(f, V), coeffD=cD, beta=beta)
    n = sfd.NumModelSplit2(f, p, dt, T, T)
    loss, gV, g0 = n.adjoint(tgt, T, K=2)
    n.close()

    xi2 = sum((np.fft.fftfreq(m, d=1.0 / m) * 2 * np.pi / (c[1] - c[0])).reshape([-1 if i == a else 1 for i in range(3)]) ** 2
              for a, (m, c) in enumerate(zip(shape, b)))
    half = np.exp(0.5j * dt * cD * xi2)

    def lin(q, h):
        return np.fft.ifftn(h * np.fft.fftn(q))
    pre, q = [], psi
    for _ in range(T):
        q = lin(q, half)
        pre.append(q)
        q = lin(q * np.exp(-1j * dt * (V + beta * np.abs(q) ** 2)), half)
    z = (tgt.conj() * q).sum() * dV
    g, wV = -2 * z * tgt * dV, np.zeros(shape)
    for s in reversed(pre):
        g = lin(g, half.conj())
        e = np.exp(-1j * dt * (V + beta * np.abs(s) ** 2))
        im = (g.conj() * e * s).imag
        wV += dt * im
        g = lin(g * e.conj() + 2 * beta * dt * im * s, half.conj())
    assert abs(loss - (1 - abs(z) ** 2)) < 1e-12 * max(1.0, abs(z) ** 2)
    assert np.linalg.norm(gV - wV) < 1e-12 * np.linalg.norm(wV)
    assert np.linalg.norm(g0 - g) < 1e-12 * np.linalg.norm(g)
