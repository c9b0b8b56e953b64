"""The natural-spline k-integral against the same spline in 50 decimal digits, on grids whose points are far from evenly
spaced (two grids joined, with pairs of points close together)."""
from decimal import Decimal as D, getcontext

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _exact(ks, Y):
    """∫ of the natural cubic spline through (0, 0) and (ks, Y)."""
    getcontext().prec = 50
    X, Y = [D(0)] + [D(float(k)) for k in ks], [D(0)] + Y
    n = len(X)
    h = [X[i + 1] - X[i] for i in range(n - 1)]
    cp, d = [D(0)] * n, [D(0)] * n
    for i in range(1, n - 1):
        den = 2 * (h[i - 1] + h[i]) - h[i - 1] * cp[i - 1]
        cp[i] = h[i] / den
        d[i] = (6 * ((Y[i + 1] - Y[i]) / h[i] - (Y[i] - Y[i - 1]) / h[i - 1]) - h[i - 1] * d[i - 1]) / den
    z, s = D(0), D(0)
    for i in range(n - 2, -1, -1):
        zi = d[i] - cp[i] * z if i > 0 else D(0)
        s += h[i] * (Y[i] + Y[i + 1]) / 2 - h[i] ** 3 * (zi + z) / 24
        z = zi
    return float(s)


GRIDS = {
    "even": np.linspace(1.0, 2000.0, 301),
    "logarithmic": np.geomspace(1e-2, 5000.0, 257),
    "joined, 1e-6 apart": np.unique(np.r_[np.linspace(1, 2000, 300), np.linspace(1, 2000, 300)[100:200] + 1e-6]),
    "joined, 1e-9 apart": np.unique(np.r_[np.linspace(1, 2000, 300), np.linspace(1, 2000, 300)[100:200] + 1e-9]),
    "two points": np.array([1.0, 2.0]),
    "thirty-three": np.linspace(0.5, 9.0, 33),
}


@pytest.mark.parametrize("grid", list(GRIDS))
@pytest.mark.parametrize("nl", [1, 9])
def test_integral_of_the_natural_spline(grid, nl):
    import symboltz as S
    ks = GRIDS[grid]
    rng = np.random.default_rng(nl)
    c = rng.uniform(0, 6, nl)
    P0 = 2e-9 * ks ** -3 * (ks / 100) ** -0.03
    A = 1.5 + np.cos(0.003 * ks[:, None] + c)
    B = np.exp(-ks[:, None] / 900) * (1 + 0.2 * np.sin(0.004 * ks[:, None] + c))
    got = S.spectrum_cmb(A, B, P0, np.arange(2, 2 + nl), ks)
    two_over_pi = 2 / D("3.14159265358979323846264338327950288419716939937511")
    ref = [_exact(ks, [two_over_pi * D(float(k)) ** 2 * D(float(p)) * D(float(a)) * D(float(b)) for k, p, a, b in zip(ks, P0, A[:, i], B[:, i])])
           for i in range(nl)]
    # a positive integrand: some 60 roundings of 2^-53 on the way of each term, and a margin of 10
    np.testing.assert_allclose(got, ref, rtol=1e-13)
