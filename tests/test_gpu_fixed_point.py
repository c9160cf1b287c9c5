"""FP64 fields are transformed in 64-bit fixed point (csrc/fft_fix.cuh): one
linear Strang step (beta = 0, V = 0: two passes per axis) against the same
flow in long double, at every line length of the register passes, for lines
whose values differ widely in size, and no further off than numpy's FP64 FFT."""
import numpy as np
import pytest

from helpers import run_model

pytestmark = pytest.mark.gpu

BOUNDS = ((0.0, 3.0), (-1.0, 4.0))
CD, DT = -0.31, 2.3e-3


def linear_flow(psi, shape, dtype, dt=DT):
    """F^-1 exp(i cD xi^2 dt) F per axis, in the precision of dtype."""
    q = psi.astype(dtype)
    for a, (n, b) in enumerate(zip(shape, BOUNDS)):
        xi = np.fft.fftfreq(n, d=1.0 / n) * ((2 * np.pi / ((b[1] - b[0]) / n)) / n)
        ph = (np.clongdouble(1j) * (CD * (xi * xi) * dt)).astype(dtype)
        q = np.fft.ifft(np.fft.fft(q, axis=a) * np.exp(ph).reshape([-1 if i == a else 1 for i in range(2)]), axis=a)
    return q


def field(kind, shape, rng):
    z = rng.standard_normal(shape) + 1j * rng.standard_normal(shape)
    if kind == "tail":  # from 1 to 1e-40 across the field, as in a trap
        r2 = sum(np.linspace(-1, 1, n).reshape([-1 if i == a else 1 for i in range(2)]) ** 2
                 for a, n in enumerate(shape))
        z = z * np.exp(-46.0 * r2)
    elif kind == "spike":  # one cell far above the rest
        z = 1e-6 * z
        z[tuple(n // 2 for n in shape)] = 1.0
    elif kind == "tiny":
        z = 1e-200 * z
    elif kind == "huge":
        z = 1e150 * z
    return z


def rel(a, b):
    return float(np.linalg.norm((a - b).astype(np.complex128)) / np.linalg.norm(b.astype(np.complex128)))


@pytest.mark.parametrize("kind", ["random", "tail", "spike", "tiny", "huge"])
@pytest.mark.parametrize("shape", [(2, 4), (8, 16), (16, 8), (32, 64), (64, 32), (128, 2), (4, 128), (256, 32),
                                   (32, 256), (256, 256)])
def test_linear_step_is_at_least_as_close_as_fp64(sfd, shape, kind):
    psi = field(kind, shape, np.random.default_rng(sum(shape)))
    got = run_model(sfd, shape, BOUNDS, psi, coeffD=CD, beta=0.0, dt=DT, nsteps=1, precision="fp64")
    scale = 2.0 ** np.floor(np.log2(np.abs(psi).max()))  # exact, and norms of the extreme cases stay representable
    exact = linear_flow(psi / scale, shape, np.clongdouble)
    err = rel(got / scale, exact)
    # Four passes.  Each rounds its result to FP64, by at most 2^-53 of each
    # value (1.1e-16 in the norm), and its values on the way about six times at
    # 2^-57 of the line's rms or less (0.16e-16 rms): 4 (1.1e-16 + 0.16e-16).
    assert err < 5.1e-16
    # and against FP64 arithmetic on the same input (which rounds hardly at all
    # on the shortest lines: one ulp besides)
    fp64 = rel(linear_flow(psi / scale, shape, np.complex128), exact)
    assert err < fp64 + 2.3e-16
    print(f"{kind} {shape}: {err:.2e} against {fp64:.2e} in FP64 arithmetic")


@pytest.mark.parametrize("kind", ["random", "tail", "spike", "tiny", "huge"])
@pytest.mark.parametrize("shape", [(3, 5), (48, 56), (480, 36), (7, 45), (12, 343), (1000, 6), (10, 1024), (26, 31),
                                   (961, 4), (64, 486)])
def test_linear_step_of_other_lengths(sfd, shape, kind):
    """As above for lengths of the generic pass (radices 2 to 16 and the loop
    primes, one stage to six)."""
    psi = field(kind, shape, np.random.default_rng(sum(shape)))
    got = run_model(sfd, shape, BOUNDS, psi, coeffD=CD, beta=0.0, dt=DT, nsteps=1, precision="fp64")
    scale = 2.0 ** np.floor(np.log2(np.abs(psi).max()))
    exact = linear_flow(psi / scale, shape, np.clongdouble)
    err = rel(got / scale, exact)
    # up to 11 stages and products of a rounding each (a loop prime: sqrt(31)
    # of them) at 2^-61 or less of the largest possible value, 32 times the rms
    # at 1024 cells, 2 bits of slack in the quantum: 0.45e-16 rms per pass besides
    # the rounding of its result
    assert err < 4 * (1.1e-16 + 0.45e-16)
    fp64 = rel(linear_flow(psi / scale, shape, np.complex128), exact)
    assert err < fp64 + 2.3e-16
    print(f"{kind} {shape}: {err:.2e} against {fp64:.2e} in FP64 arithmetic")


@pytest.mark.parametrize("dt", [41.0, -3e5, 7e9])
@pytest.mark.parametrize("shape", [(64, 32), (48, 56)])
def test_linear_step_with_many_turns(sfd, shape, dt):
    """Phase tables (made in integer arithmetic on the host) of arguments up to
    1e14 radians: the bounds of the tests above."""
    psi = field("random", shape, np.random.default_rng(3))
    got = run_model(sfd, shape, BOUNDS, psi, coeffD=CD, beta=0.0, dt=dt, nsteps=1, precision="fp64")
    assert rel(got, linear_flow(psi, shape, np.clongdouble, dt)) < 4 * (1.1e-16 + 0.45e-16)


@pytest.mark.parametrize("bad", [np.nan, np.inf])
def test_nonfinite_cell_reaches_its_lines(sfd, bad):
    shape = (64, 32)
    psi = field("random", shape, np.random.default_rng(1))
    psi[3, 5] = bad
    got = run_model(sfd, shape, BOUNDS, psi, coeffD=CD, beta=0.0, dt=DT, nsteps=1, precision="fp64")
    assert not np.isfinite(got).any()


def test_zero_lines_stay_zero(sfd):
    shape = (64, 128)
    psi = np.zeros(shape, dtype=np.complex128)
    got = run_model(sfd, shape, BOUNDS, psi, coeffD=CD, beta=0.0, dt=DT, nsteps=1, precision="fp64")
    assert (got == 0).all()


@pytest.mark.parametrize("beta,vmax,dt", [(0.0, 3.0, 1e-3), (20.0, 0.0, 1e-3), (-20.0, 3.0, 0.4), (500.0, 1e4, 0.7),
                                          (1e-9, 1e-9, 1e-3), (20.0, 3.0, -0.05)])
@pytest.mark.parametrize("shape", [(4, 2), (16, 16), (8, 32), (32, 64), (16, 128), (64, 256), (5, 12), (16, 45), (8, 400)])
def test_nonlinear_flow(sfd, shape, beta, vmax, dt):
    """exp(-i (V + beta |psi|^2) dt) psi alone (coeffD = 0: the kinetic flows
    are the identity) against long double."""
    rng = np.random.default_rng(7 * sum(shape))
    psi = field("random", shape, rng)
    V = np.asfortranarray(rng.uniform(-vmax, vmax, shape)) if vmax else None
    got = run_model(sfd, shape, BOUNDS, psi, coeffD=0.0, beta=beta, V=V, dt=dt, nsteps=1, precision="fp64")
    q = psi.astype(np.clongdouble)
    rho = q.real ** 2 + q.imag ** 2
    b, d = np.longdouble(beta), np.longdouble(dt)
    exact = q * np.exp(np.clongdouble(-1j) * ((0 if V is None else V.astype(np.longdouble)) + b * rho) * d)
    # The passes as above.  theta: two of them come before the flow, so psi
    # enters |psi|^2 with 2 x 1.27e-16 of relative error at most and theta with
    # twice that; |psi|^2 itself carries 62 bits below the line's largest
    # possible value n rms^2 <= 2^8 rms^2, 4 units of 2^-54 rms^2 for its
    # rounding, its low product and the factor's (the potential's part is exact).
    w = np.abs(psi) / np.linalg.norm(psi)
    theta = abs(beta * dt) * float(np.linalg.norm(w * rho.astype(np.float64)))
    assert rel(got, exact) < 5.1e-16 + 5.1e-16 * theta + 4 * 2.0 ** -54 * abs(beta * dt) * float(rho.mean())


def test_nonlinear_flow_with_a_nonfinite_potential(sfd):
    shape = (32, 16)
    V = np.zeros(shape, order="F")
    V[3, 4] = np.nan
    got = run_model(sfd, shape, BOUNDS, field("random", shape, np.random.default_rng(2)), V=V, nsteps=1)
    assert not np.isfinite(got).any()


def test_time_steps_in_turn(sfd):
    """A model whose calls alternate between more time steps than it keeps
    potential tables for gives what models of one time step each give."""
    shape, rng = (32, 64), np.random.default_rng(5)
    psi, V = field("random", shape, rng), np.asfortranarray(rng.uniform(0.0, 50.0, shape))
    g = sfd.Grid(shape, BOUNDS)
    f = sfd.Field(g)
    f.phi = psi
    n = sfd.NumModelSplit2(f, sfd.GrossPitaevskiiParameters(sfd.PotentialArray(f, V), coeffD=CD, beta=2.0), 1e-3, 1, 1)
    want = psi
    for dt in [1e-3, 2e-3, 1e-3, 3e-3, 4e-3, 5e-3, 1e-3, 2e-3, 1e-3]:
        n.dt = dt
        n.step(70)
        got = f.phi.copy(order="F")
        want = run_model(sfd, shape, BOUNDS, want, coeffD=CD, beta=2.0, V=V, dt=dt, nsteps=70)
        assert np.array_equal(got, want)
    n.close()
