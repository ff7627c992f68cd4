"""The bound from below on the saturation mixing ratio that lets a cloudless cell skip the saturation adjustment."""
import numpy as np
import pytest

T0K = 273.15


def _exact(T, p):
    esl = 611.2 * np.exp(17.67 * (T - T0K) / (T - 29.65))
    esi = 611.2 * np.exp(21.8745584 * (T - 273.16) / (T - 7.66))
    f = np.clip((T0K - T) / 40.0, 0.0, 1.0)
    e = (1.0 - f) * esl + f * esi
    return 0.622 * e / np.maximum(p - e, 100.0)


@pytest.mark.parametrize("p", [100.0, 101.0, 611.2, 5.0e3, 3.0e4, 1.05e5])
def test_bound_is_below_the_saturation_value(p):
    """Over all temperatures that the skip accepts, with the 1 % that it leaves for its rounding still there."""
    T = np.unique(np.concatenate([np.linspace(100.001, 1000.0, 200001), T0K + np.linspace(-0.02, 0.02, 4001),
                                  T0K - 40.0 + np.linspace(-0.02, 0.02, 4001)]))
    ice = T < T0K
    x = np.where(ice, 21.8745584, 17.67) * (T - np.where(ice, 273.16, T0K)) / (T - np.where(ice, 7.66, 29.65))
    bound = 0.99 * 0.622 * 611.2 * np.exp(x) / p
    q = _exact(T, p)
    ok = np.isfinite(q)
    assert (bound[ok] <= q[ok] * (0.99 + 1e-12)).all()


def test_zero_vapour_and_limits():
    """The skip's own expression in single precision: never taken for a NaN, a low pressure or a low temperature."""
    def skip(T, p, qv):
        T, p, qv = np.float32(T), np.float32(p), np.float32(qv)
        a, t0, c = (21.8745584, 273.16, 7.66) if T < T0K else (17.67, T0K, 29.65)
        with np.errstate(all="ignore"):
            x = np.float32(a) * ((T - np.float32(t0)) / (T - np.float32(c)))
            return bool(p >= 100 and T > 100 and qv * p < np.float32(0.99 * 0.622 * 611.2) * np.exp(x))
    assert skip(300.0, 1.0e5, 0.001) and not skip(300.0, 1.0e5, 0.03)
    for bad in ((np.nan, 1e5, 0.0), (300.0, np.nan, 0.0), (300.0, 1e5, np.nan), (300.0, 99.0, 0.0), (99.0, 1e5, 0.0)):
        assert not skip(*bad)
