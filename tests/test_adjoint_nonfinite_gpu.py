"""Non-finite cells reach exactly the gradients whose sums read them: a NaN or
an infinity in a cell of u_0 that no interior cell reads (a star's halo
corners) leaves every gradient as it was, and one that some terms read enters
those terms alone. Expected: the float64 numpy adjoint, which sums over the
cells that are read."""
import numpy as np
import pytest

import adjoint_ref as ar

pytestmark = pytest.mark.gpu


def gradients(name, u0, w, T):
    import torch
    from gbstencil.adjoint import Checkpointed
    gu, gc = Checkpointed(name, torch.tensor(u0, device="cuda"), T, 2).backward(torch.tensor(w, device="cuda"), True)
    return gu.cpu().numpy(), gc.cpu().numpy()


def inputs(name, dtype, n, seed):
    r = ar.BY_NAME[name]["rad"]
    rng = np.random.default_rng(seed)
    shape = [x + 2 * r for x in n]
    return r, rng.random(shape).astype(dtype), rng.standard_normal(shape).astype(dtype)


def corners(r, shape):
    lo, hi = [0, r - 1], [-1, -r]
    return [(i, j) for i in lo + hi for j in lo + hi]


@pytest.mark.parametrize("dtype", [np.float32, np.float64], ids=["f32", "f64"])
@pytest.mark.parametrize("name", ["star2d1r", "j2d9pt", "star2d3r"])
@pytest.mark.parametrize("n", [(1, 1), (9, 121), (70, 250)], ids=str)
@pytest.mark.parametrize("value", [np.nan, np.inf], ids=["nan", "inf"])
def test_halo_corners_are_not_read(name, dtype, n, value):
    T = 5  # launches of two steps and of one
    r, u0, w = inputs(name, dtype, n, 31)
    want = gradients(name, u0, w, T)
    for i, j in corners(r, u0.shape):
        u0[i, j] = value
    got = gradients(name, u0, w, T)
    assert all(np.array_equal(a, b) for a, b in zip(got, want))


@pytest.mark.parametrize("dtype", [np.float32, np.float64], ids=["f32", "f64"])
@pytest.mark.parametrize("name", ["star2d1r", "star2d2r", "box2d1r", "box2d2r"])
@pytest.mark.parametrize("value", [np.nan, np.inf, -np.inf], ids=str)
def test_a_cell_enters_the_terms_that_read_it(name, dtype, value):
    n = (12, 130)
    r, u0, w = inputs(name, dtype, n, 32)
    d0, d1 = u0.shape
    for cell in [(0, d1 // 2), (r - 1, r), (d0 - r, d1 - r - 1), (d0 // 2, 0), (5 + r, d1 - r), (r, r), (r, d1 // 2),
                 (d0 - r - 1, d1 - r - 1), (d0 // 2, d1 // 2), (0, 0)]:
        u = u0.copy()
        u[cell] = value
        _, gc = gradients(name, u, w, 1)
        lam = np.zeros(u.shape)
        lam[r:-r, r:-r] = w[r:-r, r:-r]
        _, ref = ar.adjoint(name, u.astype(np.float64), ar.default_coef(name), 1, lam)
        for kind in (np.isnan, np.isposinf, np.isneginf):
            assert np.array_equal(kind(gc), kind(ref)), (cell, gc, ref)


@pytest.mark.parametrize("dtype", [np.float32, np.float64], ids=["f32", "f64"])
@pytest.mark.parametrize("n", [(1, 1), (9, 121), (70, 250)], ids=str)
@pytest.mark.parametrize("value", [np.nan, np.inf], ids=["nan", "inf"])
def test_gradient2d_halo_corners_are_not_read(dtype, n, value):
    _, u0, w = inputs("gradient2d", dtype, n, 33)
    want = gradients("gradient2d", u0, w, 4)
    for i, j in corners(1, u0.shape):
        u0[i, j] = value
    got = gradients("gradient2d", u0, w, 4)
    assert all(np.array_equal(a, b) for a, b in zip(got, want))


@pytest.mark.parametrize("dtype", [np.float32, np.float64], ids=["f32", "f64"])
def test_gradient2d_a_cell_enters_its_neighbours_alone(dtype):
    n = (12, 130)
    _, u0, w = inputs("gradient2d", dtype, n, 34)
    d0, d1 = u0.shape
    for cell in [(0, d1 // 2), (d0 - 1, 1), (d0 // 2, 0), (5, d1 - 1), (1, 1), (6, 60), (0, 0)]:
        u = u0.copy()
        u[cell] = np.nan
        gu, gc = gradients("gradient2d", u, w, 1)
        lam = np.zeros(u.shape)
        lam[1:-1, 1:-1] = w[1:-1, 1:-1]
        ru, rc = ar.adjoint("gradient2d", u.astype(np.float64), ar.default_coef("gradient2d"), 1, lam)
        assert np.array_equal(np.isnan(gu), np.isnan(ru)), cell
        assert np.array_equal(np.isnan(gc), np.isnan(rc)), cell
