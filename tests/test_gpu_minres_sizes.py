"""Sector.minres on vectors where the host looks after fewer iterations than 16
(a million elements of work between looks: every 11, 4 and 1 here) and where
the passes stride over their grid, at iteration counts below, at and past a
look, against gradients.minres and against the residual of the solution.

e0 lies below the spectrum, so the system's condition number is below 10 and
two recurrences that round differently stay within 40 iterations x 10 x a few
2^-53 of each other: 1e-12 of |x|.  The residual P((H - e0) x - b) of MINRES
is what the recurrence says it is to the same accuracy, relative to |b|."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SHAPES = [(11, 3, 5), (11, 5, 5), (13, 6, 6)]      # 88,704, 221,760 and 2,965,248 elements: looks every 11, 4, 1


@pytest.mark.parametrize("shape", SHAPES)
def test_minres_between_looks(edlib, shape):
    import torch
    from pyhub_gb300.core import gradients as GR
    n, nu, nd = shape
    rng = np.random.default_rng(n + nu)
    t = np.zeros((n, n))
    for i in range(n):
        t[i, (i + 1) % n] = t[(i + 1) % n, i] = -rng.uniform(0.5, 1.0)
    sec = edlib.Sector(n, nu, nd, edlib.ED_HUBBARD, t=t, U=rng.uniform(1.0, 3.0, n))
    e0 = -4.0 * n          # |hopping part| < 2 n
    look = max(1, min(16, (1 << 20) // sec.n))
    assert look in (11, 4, 1)
    g = torch.Generator(device="cuda")
    g.manual_seed(9)
    psi = sec.from_ref(torch.randn(sec.dim, generator=g, dtype=torch.float64, device="cuda"))
    psi /= torch.linalg.vector_norm(psi)
    b = sec.from_ref(torch.randn(sec.dim, generator=g, dtype=torch.float64, device="cuda"))
    pb = b - psi * torch.dot(psi, b)
    work = torch.zeros_like(b)

    def apply(v):
        sec.hv(v, work)
        return work - e0 * v

    for maxiter in sorted({1, 2, 3, max(1, look - 1), look, look + 1, 2 * look, 2 * look + 1, 40}):
        x0, it0, rr0 = GR.minres(apply, b, psi, maxiter=maxiter, rtol=1e-9)
        x, it, rr = sec.minres(psi, e0, b, maxiter, 1e-9)
        scale = float(torch.linalg.vector_norm(x0))
        assert it == it0, maxiter
        assert float(torch.linalg.vector_norm(x - x0)) <= 1e-12 * scale, maxiter
        assert abs(float(torch.dot(psi, x))) <= 1e-12 * scale
        res = apply(x) - pb
        res -= psi * torch.dot(psi, res)
        bn = float(torch.linalg.vector_norm(pb))
        assert abs(float(torch.linalg.vector_norm(res)) / bn - rr) <= 1e-12, maxiter
    assert it < 40      # the last run converged
