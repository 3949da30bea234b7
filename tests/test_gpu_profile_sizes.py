"""The profile solve at the edges of its warps and blocks of rows (1 to 64 unknowns), with components at the bound,
against the oracle's (scipy's NNLS). The systems have cond(A) below 1e2, so the normal equations are solved within
cond^2 n 2^-52 < 1e-9 of the largest component."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SOLVE_RTOL = 1e-8


def _system(n, seed):
    g = np.random.default_rng(seed)
    m = 6 * n + 12
    i, j = np.mgrid[0:m, 0:n]
    A = np.exp(-0.5 * ((i / m * n - j) / 0.7) ** 2) + 0.02 * g.random((m, n))
    x = g.random(n)
    x[g.random(n) < 0.3] = -0.3                              # (components that the constraint sets to zero)
    if n < 3:
        x[:] = 1.
    return A, A @ x + 0.01 * g.normal(size=m), 5. + 10. * np.arange(n)


@pytest.mark.parametrize("n", [1, 2, 3, 4, 9, 31, 32, 33, 40, 41, 63, 64])
@pytest.mark.parametrize("smooth, corr", [(0.0, 1.0), (0.3, 1.0), (1.0, 4.0)])
def test_solve_sizes(gpu_lib, n, smooth, corr):
    from bbarolo2_gb300 import profile as P
    from oracle import profile as O
    A, b, radii = _system(n, n)
    assert np.linalg.cond(A) < 100.
    got = P.solve_profile(A, b, radii, smooth, corr)
    want = O.solve_profile(A, b, radii, smooth, corr)
    np.testing.assert_allclose(got, want, rtol=SOLVE_RTOL, atol=SOLVE_RTOL * np.abs(want).max())
