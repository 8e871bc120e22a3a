"""The streaming adjoint steps at the edges of their tiles: strips of one
column, a whole strip and one more, blocks of one row, grids smaller than a
window. Against the float64 numpy adjoint, at the tolerance of the other
adjoint tests (normwise 1e-9 double, 1e-4 float)."""
import numpy as np
import pytest

import adjoint_ref as ar

pytestmark = pytest.mark.gpu

SIZES = [(1, 1), (1, 60), (3, 61), (7, 120), (2, 121), (64, 59), (130, 5), (37, 241)]


def check(name, dtype, n, T, C, seed):
    import torch
    from gbstencil.adjoint import Checkpointed
    r = ar.BY_NAME[name]["rad"]
    rng = np.random.default_rng(seed)
    shape = [x + 2 * r for x in n]
    u0, w = rng.random(shape).astype(dtype), rng.standard_normal(shape).astype(dtype)
    run = Checkpointed(name, torch.tensor(u0, device="cuda"), T, C)
    gu, gc = run.backward(torch.tensor(w, device="cuda"), want_coef=True)
    inner = tuple(slice(r, -r) for _ in n)
    lam = np.zeros(shape)
    lam[inner] = w[inner]
    ru, rc = ar.adjoint(name, u0.astype(np.float64), ar.default_coef(name), T, lam)
    tol = 1e-4 if dtype == np.float32 else 1e-9
    for got, want in ((gu, ru), (gc, rc)):
        got = got.double().cpu().numpy()
        assert np.linalg.norm(got - want) <= tol * np.linalg.norm(want), (n, T)


@pytest.mark.parametrize("dtype", [np.float32, np.float64], ids=["f32", "f64"])
@pytest.mark.parametrize("n", SIZES, ids=str)
def test_gradient2d_step(n, dtype):
    check("gradient2d", dtype, n, 3, 2, 11)


@pytest.mark.parametrize("dtype", [np.float32, np.float64], ids=["f32", "f64"])
@pytest.mark.parametrize("name", ["star2d1r", "star2d2r", "star2d3r", "box2d1r", "box2d2r", "j2d5pt", "j2d9pt-gol"])
@pytest.mark.parametrize("n", [(1, 1), (2, 61), (5, 119), (9, 121), (70, 3), (33, 250)], ids=str)
def test_linear_steps(n, name, dtype):
    # 7 steps of one chunk: launches of 4, 2 and 1 steps where they are built
    check(name, dtype, n, 7, 7, 12)


@pytest.mark.parametrize("name", ["star2d1r", "j2d9pt", "box2d1r"])
@pytest.mark.parametrize("n", [(1, 1), (40, 118), (17, 130)], ids=str)
def test_linear_steps_without_coefficients(n, name):
    import torch
    from gbstencil.adjoint import Checkpointed
    r = ar.BY_NAME[name]["rad"]
    rng = np.random.default_rng(13)
    shape = [x + 2 * r for x in n]
    u0, w = rng.random(shape).astype(np.float32), rng.standard_normal(shape).astype(np.float32)
    gu, _ = Checkpointed(name, torch.tensor(u0, device="cuda"), 7, 3).backward(torch.tensor(w, device="cuda"), False)
    want, _ = ar.adjoint(name, u0.astype(np.float64), ar.default_coef(name), 7, w.astype(np.float64))
    got = gu.double().cpu().numpy()
    assert np.linalg.norm(got - want) <= 1e-4 * np.linalg.norm(want)
