"""The FP64 transforms at the largest degree a plan takes, 2048 at 4096 longitudes, where order 0 has 33
pieces of 64 degrees, and one degree below, where it has 32.

Tolerance: 1e-12 of the largest value at degree 512, the bar of the transforms' other tests, times the
degree: the recurrence over the degrees adds about three roundings (1.1e-16 each) a degree, here and in
the oracle, so its error grows with the degree (2 x 3 x 2048 x 1.1e-16 = 1.4e-12 at most).
"""

import numpy as np
import pytest

from oracle.sht import SQRT2_LEGACY, OracleSHT, gauss_nodes, legendre_rows

pytestmark = pytest.mark.gpu


def rel(lmax):
    return 1e-12 * max(1.0, lmax / 512)


def _legendre(nlat, lmax, orders):
    rows = {}
    for m, P in legendre_rows(gauss_nodes(nlat)[0][:nlat // 2], lmax):
        rows[m] = P
        if m == max(orders):
            return rows
    return rows


@pytest.mark.parametrize("lmax", [2047, 2048])
@pytest.mark.parametrize("nlat", [2, 64, 130, 256])   # one to four latitude groups per lane
def test_low_orders_at_the_largest_degrees(nlat, lmax):
    """Orders 0 to 2 with all their degrees, and the highest degree of order 0 alone."""
    import torch

    from slevolve_b200 import make_sht

    nlon, orders = 4096, (0, 1, 2)
    s, rows = make_sht("cuda", nlat, nlon, lmax), _legendre(nlat, lmax, orders)
    lon = 2.0 * np.pi * np.arange(nlon) / nlon
    parity = {m: (-1.0) ** np.arange(lmax + 1 - m)[:, None] for m in orders}

    def grid_of(c):
        g = np.zeros((nlat, nlon))
        for m in orders:
            north = SQRT2_LEGACY * (c[m:, m, None] * rows[m]).sum(axis=0)
            south = SQRT2_LEGACY * (c[m:, m, None] * rows[m] * parity[m]).sum(axis=0)
            e = np.exp(1j * m * lon) * (2.0 if m else 1.0)
            g += (np.concatenate([north, south[::-1]])[:, None] * e[None, :]).real
        return g

    rng = np.random.default_rng(nlat + lmax)
    top = np.zeros((lmax + 1, lmax + 1), complex)
    top[lmax, 0] = 1.0
    full = np.zeros_like(top)
    for m in orders:
        full[m:, m] = rng.standard_normal(lmax + 1 - m) + (1j * rng.standard_normal(lmax + 1 - m) if m else 0.0)
    for c in (top, full):
        want, got = grid_of(c), s.synthesis(torch.tensor(c, device="cuda")).cpu().numpy()
        assert np.abs(got - want).max() <= rel(lmax) * np.abs(want).max()
    g = rng.standard_normal((nlat, nlon))
    got = s.analysis(torch.tensor(g, device="cuda")).cpu().numpy()
    F = np.fft.rfft(g, axis=1)[:, :3] * (gauss_nodes(nlat)[1] / nlon)[:, None]
    nh = nlat // 2
    for m in orders:
        a, b = F[:nh, m], F[:nh - 1:-1, m]
        want = (rows[m] * (a + parity[m] * b)).sum(axis=1) / SQRT2_LEGACY
        assert np.abs(got[m:, m] - want).max() <= rel(lmax) * np.abs(got).max()


def test_every_order_at_the_largest_degree():
    import torch

    from slevolve_b200 import make_sht

    nlat, nlon, L = 64, 4096, 2048
    s, o = make_sht("cuda", nlat, nlon, L), OracleSHT(nlat, nlon, L)
    rng = np.random.default_rng(7)
    c = np.tril(rng.standard_normal((L + 1, L + 1)) + 1j * rng.standard_normal((L + 1, L + 1)))
    c[:, 0] = c[:, 0].real
    want = o.synthesis(c)
    got = s.synthesis(torch.tensor(c, device="cuda")).cpu().numpy()
    assert np.abs(got - want).max() <= rel(L) * np.abs(want).max()
    g = rng.standard_normal((nlat, nlon))
    want = o.analysis(g)
    got = s.analysis(torch.tensor(g, device="cuda")).cpu().numpy()
    assert np.abs(got - want).max() <= rel(L) * np.abs(want).max()
