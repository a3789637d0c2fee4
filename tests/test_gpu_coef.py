"""ed_lanczos_coef (the scalar work of a full-reorthogonalisation step) against
the same recurrences in numpy, at the step counts where the cluster's shares of
rows and columns change: 1, below and past one row per CTA (8), 32 rows per CTA
(256), one column per thread of the cluster (2048).

The Gram matrix is the identity with off-diagonals up to d, so Linv is within
d of it and every entry is a sum of at most 2k products of O(1) terms: the
difference from numpy is below 64 k 2^-53 (1 + d k)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("steps,d", [(1, 0.0), (7, 1e-3), (10, 1e-7), (33, 1e-3), (257, 1e-4), (300, 1e-7),
                                     (2100, 1e-7)])
def test_coef_matches_numpy(edlib, steps, d):
    import torch
    rng = np.random.default_rng(steps)
    ks = sorted({0, min(1, steps - 1), steps // 2, steps - 1})
    E = rng.uniform(-d, d, (steps, steps))
    G = np.eye(steps) + np.tril(E, -1) + np.tril(E, -1).T
    L = np.linalg.cholesky(G)
    Linv = np.linalg.inv(L)
    s = rng.uniform(0.5, 2.0, steps + 1)
    dev = lambda a: torch.tensor(a, dtype=torch.float64, device="cuda")   # noqa: E731
    mmax = steps + 2
    for k in ks:
        c = rng.standard_normal(k + 1)
        state = np.zeros(edlib.lanczos_state_doubles(mmax))
        state[2:2 + k] = s[:k]
        lin = np.zeros((mmax + 1, mmax + 1))
        lin[:k, :k] = Linv[:k, :k]
        state[3 + mmax: 3 + mmax + (mmax + 1) ** 2] = lin.ravel()
        sk = s[k]
        if k == 0:
            state[2] = sk
        dots = np.concatenate([c / (s[:k + 1] * sk), G[k, :k + 1] / (s[:k + 1] * sk)])
        st = dev(state)
        coef = dev(np.full(k + 2, np.nan))
        ab = dev(np.full((2, mmax), 1.0))
        edlib.lanczos_coef(k, mmax, dev(dots), dev([1.0 / sk ** 2]), st, coef, ab[0], ab[1])
        y = np.linalg.solve(G[:k + 1, :k + 1], c)
        tol = 64 * (k + 1) * 2.0 ** -53 * (1 + d * (k + 1))
        got = coef.cpu().numpy()
        assert np.abs(got[:k + 1] - y * s[:k + 1]).max() <= tol * 2 * max(1.0, np.abs(c).max()), k
        assert np.isnan(got[k + 1])
        out = st.cpu().numpy()
        row = out[3 + mmax:][k * (mmax + 1): k * (mmax + 1) + k + 1]
        assert np.abs(row - Linv[k, :k + 1]).max() <= tol
        assert out[0] == 0.0 and abs(out[2 + k] - sk) <= 4 * 2.0 ** -53 * sk
        assert abs(float(ab[0][k]) - c[k]) <= 8 * 2.0 ** -53 * abs(c[k])
        if k:
            assert abs(float(ab[1][k - 1]) - 1.0 / sk) <= 4 * 2.0 ** -53 / sk


def test_coef_stops_on_a_dependent_vector(edlib):
    """A vector inside the span of the basis (Gram pivot below half its norm) stops the run with zero coefficients."""
    import torch
    mmax, k = 12, 9
    state = torch.zeros(edlib.lanczos_state_doubles(mmax), dtype=torch.float64, device="cuda")
    state[2:2 + k] = 1.0
    lin = state[3 + mmax: 3 + mmax + (mmax + 1) ** 2].view(mmax + 1, mmax + 1)
    lin[:k, :k] = torch.eye(k, dtype=torch.float64, device="cuda")
    dots = torch.zeros(2 * (k + 1), dtype=torch.float64, device="cuda")
    dots[k + 1] = 0.8     # <v_0, v_k>: 1 - 0.64 < 1/2
    dots[2 * k + 1] = 1.0
    nrm = torch.ones(1, dtype=torch.float64, device="cuda")
    coef = torch.full((k + 1,), 3.0, dtype=torch.float64, device="cuda")
    ab = torch.ones((2, mmax), dtype=torch.float64, device="cuda")
    edlib.lanczos_coef(k, mmax, dots, nrm, state, coef, ab[0], ab[1])
    assert float(state[0]) == k and not coef.any()
    edlib.lanczos_coef(k + 1, mmax, dots.new_zeros(2 * (k + 2)), nrm, state, dots.new_full((k + 2,), 3.0), ab[0], ab[1])
    assert float(state[0]) == k and float(state[2 + k + 1]) == 0.0
