"""Eigen-emittances of anything that carries the second moments, one at a time or many."""
import collections
import types

import numpy as np

from ocelot_gb300 import envelope

NAMES = ("xx", "xpx", "pxpx", "yy", "ypy", "pypy", "xy", "pxpy", "xpy", "ypx")


def _moments(seed):
    z = np.random.default_rng(seed).standard_normal((4, 60)) * [[1e-4], [2e-5], [2e-4], [1e-5]]
    z[2] += 0.3 * z[0]
    s = np.cov(z)  # x, px, y, py
    return dict(xx=s[0, 0], xpx=s[0, 1], pxpx=s[1, 1], yy=s[2, 2], ypy=s[2, 3], pypy=s[3, 3], xy=s[0, 2],
                pxpy=s[1, 3], xpy=s[0, 3], ypx=s[1, 2])


def test_any_object_with_the_moments():
    m = _moments(1)
    want = envelope.eigen_emittances(types.SimpleNamespace(**m))
    assert 0 < want[1] < want[0]
    assert envelope.eigen_emittances(collections.namedtuple("Moments", NAMES)(**m)) == want
    assert envelope.eigen_emittances(type("Moments", (), dict(m, __slots__=()))()) == want


def test_many_at_once_equal_one_at_a_time():
    many = [types.SimpleNamespace(**_moments(k)) for k in range(5)]
    many[2].xpy = float("nan")
    one = [envelope.eigen_emittances(t) for t in many]
    assert np.isnan(one[2]).all() and np.isfinite(one[3]).all()
    assert np.array_equal(envelope._eigen_emittances(many), one, equal_nan=True)
