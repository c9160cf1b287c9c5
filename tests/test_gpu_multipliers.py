"""Multiplier tables of FP64 passes mode by mode: the factors of a table differ
by orders of magnitude (the Laplacian's by (n/2)^2, an imaginary-time factor
in a rotating frame by e^20 across the rows), and the small ones, where a
field's weight is, keep FP64's relative precision."""
import numpy as np
import pytest

from helpers import run_model

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _lib(built_lib):
    return built_lib


CD = -0.31


def xi_of(n, k, b):
    """The library's (and the reference's) Float64 wavenumber."""
    return np.fft.fftfreq(n, d=1.0 / n)[k] * ((6.283185307179586 / ((b[1] - b[0]) / n)) / n)


@pytest.mark.parametrize("mode", [1, 2, 3])
@pytest.mark.parametrize("shape,axis", [((256, 4), 0), ((4, 256), 1), ((512, 3), 0), ((6, 1000), 1), ((1024, 2), 0),
                                        ((64, 64, 128), 0), ((64, 64, 128), 2), ((256, 32, 64), 0),
                                        ((16, 256, 128), 1), ((8, 4, 2), 0), ((10, 1024, 32), 1)])
def test_laplacian_of_one_plane_wave(sfd, shape, axis, mode):
    """One explicit Euler step psi + i dt cD Lap psi of the plane wave of a low
    mode, with dt so long that the Laplacian is all of the result, projected on that mode."""
    n, nd = shape[axis], len(shape)
    bounds = ((0.0, 20.0),) * nd
    turns = (mode * np.arange(n)) % n  # exact
    wave = np.exp(np.clongdouble(2j) * np.longdouble(turns) / n * (4 * np.arctan(np.longdouble(1))))
    like = [-1 if a == axis else 1 for a in range(nd)]
    psi = np.asfortranarray(np.broadcast_to(wave.astype(np.complex128).reshape(like), shape))
    xi = xi_of(n, mode, bounds[axis])
    dt = float(2.0 ** np.round(np.log2(1e8 / abs(CD * xi * xi))))
    f = sfd.Field(sfd.Grid(shape, bounds))
    f.phi = psi
    p = sfd.GrossPitaevskiiParameters(sfd.PotentialZero(f), coeffD=CD, beta=0.0)
    m = sfd.NumModelGPRK(f, p, dt, 1, 1, stepper="RK1", filter="none")
    m.step(1)
    got = f.phi.copy(order="F")
    m.close()

    def project(q):  # of each line on the mode
        q = np.moveaxis(q, axis, -1).astype(np.clongdouble)
        return (q * wave.conj()).sum(axis=-1) / n

    exact = project(psi) * (1 + np.clongdouble(1j) * np.longdouble(dt) * np.longdouble(CD * (xi * xi)))
    # roundings to FP64 on the way: the multiplier, the pass's result, one
    # addition per further axis, and two in the stage update
    assert np.max(np.abs(project(got) / exact - 1)) < (4 + nd) * 2.0 ** -53


@pytest.mark.parametrize("scheme,nsteps", [(1, 1), (2, 2)])
@pytest.mark.parametrize("shape", [(64, 32), (16, 8), (48, 56), (256, 128), (31, 10), (512, 1024)])
def test_imaginary_time_with_growing_modes(sfd, shape, scheme, nsteps):
    """coeffD > 0: the factors of white noise reach e^10 per step."""
    bounds = ((0.0, 5.0),) * 2
    rng = np.random.default_rng(sum(shape))
    psi = np.asfortranarray(rng.standard_normal(shape) + 1j * rng.standard_normal(shape))
    xi = [np.array([xi_of(n, k, b) for k in range(n)]) for n, b in zip(shape, bounds)]
    dt, cD = 1e-2, 1000.0 / max(float((x * x).max()) for x in xi)
    got = run_model(sfd, shape, bounds, psi, coeffD=cD, beta=0.0, dt=dt, nsteps=nsteps, scheme=scheme, imag=True)
    q = psi.astype(np.clongdouble)
    for a in range(2):
        e = np.exp(np.longdouble(cD * (xi[a] * xi[a]) * dt) * nsteps).reshape([-1 if i == a else 1 for i in range(2)])
        q = np.fft.ifft(np.fft.fft(q, axis=a) * e, axis=a)
    dV = np.prod([(b[1] - b[0]) / n for n, b in zip(shape, bounds)])
    q = q / np.sqrt((np.abs(q) ** 2).sum() * dV)
    # per step up to four passes and the factor of the mass, at 1.6e-16 each
    # (1024-cell lines), and the mass itself; the rounded exponents at up to
    # 10 x 1.1e-16 twice
    err = np.linalg.norm((got - q).astype(np.complex128)) / np.linalg.norm(q.astype(np.complex128))
    assert err < nsteps * (6 * 1.6e-16 + 2 * 10 * 1.1e-16)


@pytest.mark.parametrize("shape", [(128, 128), (120, 120), (128, 100)])
def test_imaginary_time_in_a_rotating_frame(sfd, shape):
    """Lie steps of a field at rest in the middle of a box whose outer rows
    have factors up to e^20: the rows where the field lives stay below 1 and keep
    their precision."""
    bounds, cD, om, dt = ((-10.0, 10.0),) * 2, -0.5, 2.0, 0.1
    X = [np.array(sfd.grid_coords(n, *b)) for n, b in zip(shape, bounds)]
    psi = np.exp(-2.0 * (X[0][:, None] ** 2 + X[1][None, :] ** 2)) + 0j
    psi[np.abs(X[0]) > 4, :] = 0
    psi[:, np.abs(X[1]) > 4] = 0
    got = run_model(sfd, shape, bounds, np.asfortranarray(psi), coeffD=cD, beta=0.0, omega=om, dt=dt, nsteps=1,
                    scheme=1, imag=True)
    q = psi.astype(np.clongdouble)
    for a in range(2):
        xi = np.array([xi_of(shape[a], k, bounds[a]) for k in range(shape[a])])
        sign = -1.0 if a == 0 else 1.0
        e = cD * (xi * xi)[:, None] + sign * om * X[1 - a][None, :] * xi[:, None]  # (mode, row)
        e = np.exp(np.longdouble(e * dt))
        q = np.fft.ifft(np.fft.fft(q, axis=a) * (e if a == 0 else e.T), axis=a)
    dV = np.prod([(b[1] - b[0]) / n for n, b in zip(shape, bounds)])
    q = q / np.sqrt((np.abs(q) ** 2).sum() * dV)
    inner = np.ix_(*[np.abs(x) <= 3 for x in X])  # further out factors above 1 raise rounding itself
    d, w = (got - q)[inner].astype(np.complex128), q[inner].astype(np.complex128)
    # four roundings to FP64 (two passes, the mass, its factor) and what the
    # passes round on the way, twice for the parts that factors above 1 raise
    assert np.linalg.norm(d) < 2 * (4 * 1.1e-16 + 2 * 0.45e-16) * np.linalg.norm(w)
