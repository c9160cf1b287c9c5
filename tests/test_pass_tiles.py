"""The lines that a CTA of a pass holds, as counted on the host (the reductions'
partial sums are sized by them): FP64 fields of up to 2^18 cells run CTAs of
128 threads with four cells each, larger ones CTAs of 128 threads with 16 (8 on
lines of 32 and 64 cells).  No GPU needed."""
import ctypes

import pytest


@pytest.fixture(scope="module")
def lines(sfd, built_lib):
    from sfd_gb300 import _lib
    f = getattr(_lib.lib(), "_ZN4gpss22pass_lines_per_cta_f64Eibl")  # (int n, bool xl, long total)
    f.restype, f.argtypes = ctypes.c_int, [ctypes.c_int, ctypes.c_bool, ctypes.c_long]
    return f


@pytest.mark.parametrize("xl", [True, False])
@pytest.mark.parametrize("n", [16, 32, 64, 128, 256])
def test_lines_of_an_fp64_cta(lines, n, xl):
    for total in (n * n, 1 << 18):
        assert lines(n, xl, total) == 128 * 4 // n
    per_thread = 8 if n in (32, 64) else 16
    for total in ((1 << 18) + n, 1 << 24):
        assert lines(n, xl, total) == 128 * per_thread // n
