"""Sector.minres (ed_minres) against gradients.minres, the same recurrence in
torch operations, and against the dense solution: Hubbard sectors with and
without row padding, a Heisenberg sector, runs cut off at maxiter before, at
and past the host's look (every 16 iterations on small sectors), b = 0, b along psi.

Both recurrences are the same to rounding; after k iterations they differ by
at most about k kappa 2^-53 relative to |x| (kappa the condition number of
H - E0 off psi, below 1e3 here): 1e-10.  A converged run is within
kappa * rtol of the dense solution."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _sector(edlib, name):
    rng = np.random.default_rng(5)
    if name == "heis":
        J = rng.uniform(0.5, 1.5, (8, 8))
        return edlib.Sector(8, 4, 0, edlib.ED_HEISENBERG, J=J + J.T)
    n, nu, nd = {"pad": (6, 3, 2), "nopad": (2, 1, 1), "eight": (8, 4, 3)}[name]
    t = np.zeros((n, n))
    for i in range(n - 1):
        t[i, i + 1] = t[i + 1, i] = -rng.uniform(0.5, 1.5)
    t[np.diag_indices(n)] = rng.normal(0.0, 0.3, n)
    return edlib.Sector(n, nu, nd, edlib.ED_HUBBARD, t=t, U=rng.uniform(2.0, 6.0, n))


@pytest.mark.parametrize("name", ["pad", "nopad", "eight", "heis"])
@pytest.mark.parametrize("maxiter", [1, 2, 15, 16, 17, 33, 2000])
def test_minres_matches_torch_recurrence_and_dense(edlib, name, maxiter):
    import torch
    from pyhub_gb300.core import gradients as GR
    sec = _sector(edlib, name)
    D = sec.dim
    cols = torch.zeros((D, sec.n), dtype=torch.float64, device="cuda")
    for i in range(D if D <= 400 else 0):
        e = torch.zeros(D, dtype=torch.float64, device="cuda")
        e[i] = 1.0
        sec.hv(sec.from_ref(e), cols[i])
    g = torch.Generator(device="cuda")
    g.manual_seed(3)
    b = sec.from_ref(torch.randn(D, generator=g, dtype=torch.float64, device="cuda"))
    if D <= 400:
        H = sec.to_ref(cols).T.cpu().numpy()
        val, vec = np.linalg.eigh(H)
        e0, psi = float(val[0]), sec.from_ref(torch.tensor(vec[:, 0].copy(), device="cuda"))
    else:
        from pyhub_gb300.core import lanczos as LZ
        gs = LZ.ground_state(sec, mode="f64", steps=200, rule=LZ.ResidualRule(1e-12, 10))
        e0, psi = gs.e0, gs.psi
    work = torch.zeros_like(b)

    def apply(v):
        sec.hv(v, work)
        return work - e0 * v

    x0, it0, rr0 = GR.minres(apply, b, psi, maxiter=maxiter, rtol=1e-12)
    x, it, rr = sec.minres(psi, e0, b, maxiter, 1e-12)
    scale = float(torch.linalg.vector_norm(x0))
    assert abs(it - it0) <= (0 if maxiter < 33 else 1)
    assert float(torch.linalg.vector_norm(x - x0)) <= 1e-10 * scale
    assert abs(rr - rr0) <= 1e-10 + 0.5 * rr0
    assert abs(float(torch.dot(psi, x))) <= 1e-12 * scale
    if D <= 400 and maxiter == 2000:
        d = val - e0
        bb = sec.to_ref(b).cpu().numpy()
        want = vec[:, 1:] @ ((vec[:, 1:].T @ bb) / d[1:])
        assert np.linalg.norm(sec.to_ref(x).cpu().numpy() - want) <= 1e-9 * np.linalg.norm(want)


def test_minres_zero_right_hand_side(edlib):
    import torch
    sec = _sector(edlib, "pad")
    psi = sec.from_ref(torch.ones(sec.dim, dtype=torch.float64, device="cuda") / sec.dim ** 0.5)
    x, it, rr = sec.minres(psi, -1.0, torch.zeros_like(psi), 50, 1e-10)
    assert it == 0 and rr == 0.0 and not x.any()
