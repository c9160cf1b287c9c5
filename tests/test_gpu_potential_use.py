"""What a potential costs and does in the real-time flow of FP64 fields: no
memory beside its own, whatever the time steps, and a cell without a finite
value is NaN by itself."""
import numpy as np
import pytest

from helpers import random_field, run_model

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _lib(built_lib):
    return built_lib


BOUNDS = ((-3.0, 3.0), (-2.0, 2.0))


def model(sfd, shape, V):
    f = sfd.Field(sfd.Grid(shape, BOUNDS))
    f.phi = random_field(shape, seed=6)
    p = sfd.GrossPitaevskiiParameters(sfd.PotentialArray(f, V), beta=3.0)
    return f, sfd.NumModelSplit2(f, p, 1e-3, 1, 1)


@pytest.mark.parametrize("shape", [(512, 512), (256, 128), (360, 480)])
def test_time_steps_take_no_memory(sfd, shape):
    """Steps of several sizes need tables of a line or less each."""
    from sfd_gb300 import _lib
    V = np.asfortranarray(np.random.default_rng(2).uniform(0.0, 9.0, shape))
    f, n = model(sfd, shape, V)
    before = _lib.lib().gpss_device_bytes(n.handle)
    for dt in (1e-3, 2e-3, 3e-3, 4e-3, 5e-3):
        n.dt = dt
        n.step(1)
    # per time step: phase tables of n + 1 entries of 16 bytes per axis for dt,
    # dt / 2 and the sums of neighbouring halves; once 3 KB of roots of unity
    assert _lib.lib().gpss_device_bytes(n.handle) - before < 5 * 4 * 16 * (sum(shape) + 2) + 4096
    n.close()


@pytest.mark.parametrize("bad", [np.inf, -np.inf, np.nan])
@pytest.mark.parametrize("shape", [(64, 32), (48, 56), (512, 512), (256, 1024), (16, 8)])
def test_nonfinite_cell_of_the_potential(sfd, shape, bad):
    """The Lie step ends with the nonlinear flow: one cell is NaN after it, as
    exp(-i V dt) is, and every other cell what it is with a finite value there."""
    V = np.asfortranarray(np.random.default_rng(3).uniform(0.0, 9.0, shape))
    psi = random_field(shape, seed=7)
    kw = dict(beta=3.0, dt=1e-2, nsteps=1, scheme=1)
    want = run_model(sfd, shape, BOUNDS, psi, V=V, **kw)
    V[3, 5] = bad
    got = run_model(sfd, shape, BOUNDS, psi, V=V, **kw)
    assert np.isnan(got[3, 5].real) and np.isnan(got[3, 5].imag)
    got[3, 5] = want[3, 5]
    assert np.array_equal(got, want)


@pytest.mark.parametrize("shape", [(64, 32), (48, 56), (64, 64, 128)])
@pytest.mark.parametrize("scale", [1e-300, 1e-12, 1.0, 3e5, 2e14])
def test_potential_of_any_size(sfd, shape, scale):
    """exp(-i V dt) psi alone (coeffD = 0, beta = 0, Lie) against long double,
    from potentials that do nothing to 1e13 turns per step."""
    V = np.asfortranarray(np.random.default_rng(5).uniform(-scale, scale, shape))
    psi = random_field(shape, seed=8)
    dt = 0.37
    bounds = BOUNDS + ((0.0, 1.0),) * (len(shape) - 2)
    got = run_model(sfd, shape, bounds, psi, V=V, coeffD=0.0, beta=0.0, dt=dt, nsteps=1, scheme=1)
    # V dt in turns, exactly modulo one: V, dt and 1/(2 pi) to 190 bits as integers
    inv2pi = 0x28BE60DB9391054A7F09D5F47D4D377036D8A5664F10E410  # 2^192 / (2 pi)
    (dn, dd) = dt.as_integer_ratio()
    turns = np.empty(V.size)
    for i, v in enumerate(V.ravel()):
        (vn, vd) = float(v).as_integer_ratio()
        t = (vn * dn * inv2pi << 64) // (vd * dd << 192) & (2 ** 64 - 1)  # 2^-64 turns, floored
        turns[i] = (t - 2 ** 64 if t >= 2 ** 63 else t) * 2.0 ** -64
    exact = psi * np.exp(-2j * np.pi * turns.reshape(shape))
    # two or three passes at 1.6e-16 each, exp and the product here at 8e-16, and
    # dt / (2 pi) to 2^-62 of the angle
    theta = scale * dt * 2.0 ** -62
    assert np.linalg.norm(got - exact) < (len(shape) * 1.6e-16 + 8e-16 + 2 * np.pi * theta) * np.linalg.norm(exact)
