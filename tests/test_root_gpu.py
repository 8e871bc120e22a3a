"""The reciprocal root of gradient2d's FMA mode, seen through one step of the
time loop: a cell with value 0 beside one cell of value a has
s = eps + a^2 (each operation rounded) and becomes num / sqrt(s), num = 1.

Double: the hardware's estimate with one third-order step. Its rounding errors
are one of the product s y (at most half an ulp of the root, through e/2) and
that of the last operation (half an ulp), and the series' remainder is far
below: at most 1.1 ulp, over the whole range of s, the ends of the range that
the step serves (2^-100 and 2^100) and what lies beyond. Float: a pair rounded
once, so half an ulp but for a remainder near 2^-20 ulp."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def roots(a, dtype, eps):
    """(s, the engine's 1/sqrt(s)) for every value of a."""
    import torch
    from gbstencil.grid import DeviceGrid
    side = int(np.ceil(np.sqrt(a.size)))
    u = np.zeros((4 * side + 2, 4 * side + 2), dtype)
    cells = np.zeros(side * side, dtype)
    cells[:a.size] = a
    u[2:-1:4, 2:-1:4] = cells.reshape(side, side)
    g = DeviceGrid("gradient2d", dtype, [4 * side, 4 * side])
    for p in (0, 1):
        g.plane(p).copy_(torch.tensor(u))
    g.run(1, "fma", eps=eps)
    out = g.plane(1).cpu().numpy()[2:-1:4, 3:-1:4].reshape(-1)[:a.size]
    with np.errstate(over="ignore", under="ignore"):
        s = dtype(eps) + a * a
    return s, out


def error_in_ulps(got, s, wide):
    want = 1 / np.sqrt(s.astype(wide))
    ulp = np.spacing(want.astype(got.dtype)).astype(wide)
    return np.abs((got.astype(wide) - want) / ulp)


def test_double_root_over_the_whole_range():
    rng = np.random.default_rng(51)
    edges = [np.sqrt(2.0 ** e) * (1 + k * 2.0 ** -52) for e in (-100, 100) for k in range(-40, 41)]
    a = np.concatenate([np.exp2(rng.uniform(-500, 500, 60000)), np.exp2(rng.uniform(-50.5, -49.5, 5000)),
                        np.exp2(rng.uniform(49.5, 50.5, 5000)), rng.uniform(0.5, 2, 20000), np.array(edges)])
    s, got = roots(a, np.float64, 5e-324)
    assert np.isfinite(s).all() and (s > 0).all()
    assert error_in_ulps(got, s, np.longdouble).max() <= 1.1


def test_float_root():
    rng = np.random.default_rng(52)
    a = np.concatenate([np.exp2(rng.uniform(-45, 45, 60000)), rng.uniform(0.5, 2, 20000)]).astype(np.float32)
    s, got = roots(a, np.float32, 1e-30)
    assert error_in_ulps(got, s, np.float64).max() <= 0.5 + 2.0 ** -16


def test_double_root_of_infinity_and_nan():
    s, got = roots(np.array([np.finfo(np.float64).max, np.nan]), np.float64, 1.0)
    assert np.isinf(s[0]) and got[0] == 0 and np.isnan(got[1])
