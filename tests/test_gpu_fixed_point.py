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


def linear_flow(psi, shape, dtype):
    """F^-1 exp(i cD xi^2 dt) F per axis, in the precision of dtype."""
    q = psi.astype(dtype)
    for a, (n, b) in enumerate(zip(shape, BOUNDS)):
        xi = np.fft.fftfreq(n, d=1.0 / n) * ((2 * np.pi / ((b[1] - b[0]) / n)) / n)
        ph = (np.clongdouble(1j) * (CD * (xi * xi) * DT)).astype(dtype)
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
