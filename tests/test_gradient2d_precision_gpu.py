"""One adjoint step of float gradient2d is no further from 64 bits than the
step with the root in double (rounded once) and the sum of the differences in
double, which it replaced: that step is restated here in numpy float32."""
import numpy as np
import pytest

import adjoint_ref as ar

pytestmark = pytest.mark.gpu
F, D = np.float32, np.float64
N = 300


def fma(a, b, c):
    return (a.astype(D) * b + c).astype(F)


def shifted(a, off):
    return a[tuple(slice(1 + o, x - 1 + o) for o, x in zip(off, a.shape))]


def field(kind, seed):
    rng = np.random.default_rng(seed)
    noise = rng.random((N + 2, N + 2)).astype(F)
    y, x = np.linspace(0, 6, N + 2)[:, None], np.linspace(0, 9, N + 2)[None]
    smooth = (np.sin(x) * np.cos(y)).astype(F)
    u = {"random": noise, "smooth": smooth, "mixed": (smooth + F(1e-3) * noise).astype(F), "large": F(100) * noise}[kind]
    lam = np.zeros_like(u)
    lam[1:-1, 1:-1] = (rng.random((N, N)) - 0.5).astype(F)
    return u, lam


def restated(u, lam, num, eps, neighbours):
    c, inner = u[1:-1, 1:-1], (slice(1, -1), slice(1, -1))
    s = np.full(c.shape, eps)
    for o in neighbours:
        d = c - shifted(u, o)
        s = s + d * d
    q = np.zeros_like(u)
    q[inner] = (1.0 / np.sqrt(s.astype(D))).astype(F)
    sd = sum((c - shifted(u, o)).astype(D) for o in neighbours).astype(F)
    cube = ((num * q[inner]) * q[inner]) * q[inner]
    out = lam[inner] * fma(-cube, sd, np.ones_like(sd))
    w = ((lam * num) * q) * q * q
    for o in neighbours:
        back = [-x for x in o]
        out = fma(shifted(w, back), shifted(u, back) - c, out)
    return out


@pytest.mark.parametrize("kind", ["random", "smooth", "mixed", "large"])
@pytest.mark.parametrize("seed", [1, 2])
def test_float_step_error(kind, seed):
    import torch
    from gbstencil.adjoint import Checkpointed
    s = ar.BY_NAME["gradient2d"]
    num, eps = F(s["numerator"]), F(s["eps"])
    u, lam = field(kind, seed)
    gu, _ = Checkpointed("gradient2d", torch.tensor(u, device="cuda"), 1, 1).backward(torch.tensor(lam, device="cuda"))
    inner = (slice(1, -1), slice(1, -1))
    # the float64 adjoint with the same float eps and numerator
    c = u[inner].astype(D)
    acc = np.full(c.shape, D(eps))
    ds = [c - shifted(u.astype(D), o) for o in s["neighbours"]]
    for d in ds:
        acc += d * d
    g = D(num) * acc ** -1.5
    full = np.zeros(u.shape)
    full[inner] += lam[inner] * (1 - g * sum(ds))
    for o, d in zip(s["neighbours"], ds):
        shifted(full, o)[...] += lam[inner] * g * d
    want = full[inner]
    error = np.linalg.norm(gu.cpu().numpy()[inner] - want)
    assert error <= np.linalg.norm(restated(u, lam, num, eps, s["neighbours"]) - want)
