"""Relaxed Love numbers against the sum over each degree's modes, one degree at a time, and the Earth models
whose tables end below the degree asked for, which are refused."""

import types

import numpy as np
import pytest

from slevolve_b200.init_topo import relaxed_love

KEYS = ("s", "r", "rprime")


def _model(ndeg, modes, rng):
    m = types.SimpleNamespace(he=rng.standard_normal(ndeg), ke=rng.standard_normal(ndeg),
                              nmod=rng.integers(0, modes + 1, ndeg))
    m.s, m.r, m.rprime = (0.01 + rng.random((modes, ndeg)) for _ in KEYS)
    return m


def _by_degree(m, lmax, tau):
    h, k = np.array(m.he[:lmax + 1], float), np.array(m.ke[:lmax + 1], float)
    for ll in range(1, lmax + 1):
        s = m.s[:m.nmod[ll], ll]
        f = 1.0 - np.exp(-s * tau)
        h[ll] += (m.r[:m.nmod[ll], ll] / s * f).sum()
        k[ll] += (m.rprime[:m.nmod[ll], ll] / s * f).sum()
    return h, k


@pytest.mark.parametrize("lmax", [0, 1, 2, 30, 31])
def test_equals_the_sum_over_modes(lmax):
    m = _model(32, 5, np.random.default_rng(lmax))
    for a, b in zip(relaxed_love(m, lmax, 7.5), _by_degree(m, lmax, 7.5)):
        # at most five terms below 1e2 / 1e-2, added in another order: a few roundings of 1.1e-16
        assert a.shape == b.shape and np.allclose(a, b, rtol=1e-13, atol=1e-13)


@pytest.mark.parametrize("short", ["all", "he", "ke", "nmod", *KEYS])
def test_tables_below_the_degree_are_refused(short):
    m = _model(32, 5, np.random.default_rng(1))
    m.nmod[:] = 3
    if short != "all":
        for key in ("he", "ke", "nmod", *KEYS):
            if key != short:
                a = getattr(m, key)
                setattr(m, key, np.concatenate([a, a], axis=-1))
    relaxed_love(m, 31, 7.5)
    with pytest.raises(IndexError):
        _by_degree(m, 32, 7.5)
    with pytest.raises(IndexError):
        relaxed_love(m, 32, 7.5)
