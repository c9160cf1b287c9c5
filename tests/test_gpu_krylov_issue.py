"""The host issues Krylov iterations ahead of the device's stopping test.  Where a
step's solves take what they took in the last step, as in a run that changes
slowly, it issues exactly those."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _lib(built_lib):
    return built_lib


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_no_iteration_is_issued_in_vain(sfd, precision):
    from sfd_gb300 import _lib
    shape, b = (64, 64), ((-8.0, 8.0),) * 2
    x, y = np.meshgrid(*[np.linspace(-8, 8, 64, endpoint=False)] * 2, indexing="ij")
    psi = np.exp(-0.25 * (x ** 2 + y ** 2) + 0.3j * x) * (1 + 0.1 * y)
    psi = np.asfortranarray(psi / np.linalg.norm(psi) * 4.0)
    newton = 3

    def model(**kw):
        f = sfd.Field(sfd.Grid(shape, b))
        f.phi = psi
        p = sfd.GrossPitaevskiiParameters(sfd.PotentialArray(f, np.asfortranarray(0.5 * (x ** 2 + y ** 2))),
                                          coeffD=-0.5, beta=50.0)
        # (a Newton tolerance that is never met: every step has `newton` solves)
        return sfd.NumModelCrankNicolson(f, p, 1e-3, 1, 1, nnewton=newton, tolnewton=1e-300, precision=precision, **kw)

    def launches(n):  # of one step
        before = _lib.lib().gpss_launch_count(n.handle)
        n.step(1)
        return _lib.lib().gpss_launch_count(n.handle) - before

    # a cap of k iterations that no solve gets below: k per solve
    per = {}
    for k in (1, 2):
        n = model(nkrylov=k, tolkrylov=1e-300)
        n.step(1)
        per[k] = launches(n)
        n.close()
    iteration = (per[2] - per[1]) // newton
    assert (per[2] - per[1]) % newton == 0 and iteration > 0
    n = model(tolkrylov=1e-8 if precision == "fp64" else 1e-5)
    for _ in range(3):
        n.step(1)
    same = 0
    for _ in range(12):
        last, got = n.last_krylov, launches(n)
        if n.last_krylov == last:
            # (the count leaves out the iteration that meets the tolerance, one per
            # solve; per[1] has one per solve)
            assert got == per[1] + iteration * n.last_krylov
            same += 1
    n.close()
    assert same >= 6
