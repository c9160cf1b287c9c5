"""Hard walls: a potential of +inf in imaginary time.  exp(-(V + beta |psi|^2) dt)
is 0 there at every time step, in the prologue and the epilogue that the
passes carry it in (the merged and the step by step sequence)."""
import numpy as np
import pytest

from helpers import random_field, run_model

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _lib(built_lib):
    return built_lib


def walls(shape, bounds):
    """A harmonic well between walls of +inf, the outer sixth on each side."""
    V = np.zeros(shape, order="F")
    for a, (n, b) in enumerate(zip(shape, bounds)):
        x = np.linspace(b[0], b[1], n, endpoint=False).reshape([-1 if i == a else 1 for i in range(len(shape))])
        V += 0.5 * x ** 2 + np.where(np.abs(x) > b[1] * 2 / 3, np.inf, 0.0)
    return V


# the low part of dt / ln 2 is positive for the first time step, negative for the others
@pytest.mark.parametrize("dt", [1e-3, 2.5e-3, 1e-2, 0.1])
@pytest.mark.parametrize("scheme,merge", [(2, True), (2, False), (1, True)])
@pytest.mark.parametrize("shape", [(64, 32), (48, 56), (256, 16), (64, 64, 128), (16, 8, 4), (32, 45, 24)])
def test_infinite_potential_in_imaginary_time(sfd, shape, scheme, merge, dt):
    bounds = ((-3.0, 3.0),) * len(shape)
    kw = dict(V=walls(shape, bounds), beta=30.0, dt=dt, nsteps=4, scheme=scheme, imag=True)
    psi = random_field(shape, seed=4)
    got = run_model(sfd, shape, bounds, psi, merge=merge, **kw)
    want = run_model(sfd, shape, bounds, psi, form="plain", **kw)
    assert np.isfinite(got).all() and np.isfinite(want).all()
    # 4 steps of at most 6 passes and one exponential, each within 5e-16 of its
    # exact result in either form
    assert np.linalg.norm(got - want) < 2 * 4 * 7 * 5e-16 * np.linalg.norm(want)
