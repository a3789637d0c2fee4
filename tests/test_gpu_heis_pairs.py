"""Heisenberg pair sums (ed_rdm) for odd and even site counts down to one-site
halves, against the definition over all states in numpy:
pair lists with repeats, both orders, subsets, bra equal to and different from ket.

FP64: each sum is at most D products deep, |err| <= (D + 64) 2^-53 sum|b k|;
FP32 vectors round each product once more (2^-24)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _sums(n, h, bra, ket, J, K):
    """q0, q1 and the sum of magnitudes, sites 0-based; a set bit of h is a down spin."""
    b = bra * ket
    dJ, dK = (h >> J) & 1, (h >> K) & 1
    q1 = 0.25 * np.sum(np.where(dJ == dK, b, -b))
    if J == K:
        return 0.5 * b.sum(), q1, np.abs(b).sum()
    at = np.nonzero((dJ == 0) & (dK == 1))[0]
    to = np.searchsorted(h, h[at] ^ (1 << J) ^ (1 << K))
    p = bra[to] * ket[at]
    return (-1.0) ** (J + K) * p.sum(), q1, np.abs(b).sum() + np.abs(p).sum()


@pytest.mark.parametrize("n", [2, 3, 4, 5, 7, 8, 9, 12, 13])
@pytest.mark.parametrize("dt", ["f32", "f64"])
def test_pair_sums(edlib, n, dt):
    import torch
    nup = n // 2
    td = torch.float32 if dt == "f32" else torch.float64
    rng = np.random.default_rng(100 * n)
    h = np.array([x for x in range(1 << n) if bin(x).count("1") == n - nup], dtype=np.int64)
    D = len(h)
    J = rng.standard_normal((n, n))
    sec = edlib.Sector(n, nup, 0, edlib.ED_HEISENBERG, J=J + J.T)
    assert sec.dim == D
    allp = [(a, b) for a in range(1, n + 1) for b in range(1, n + 1)]
    some = [allp[int(i)] for i in rng.integers(0, len(allp), 5)] + [(n, 1), (1, n), (1, 1)]
    u = (D + 64) * 2.0 ** -53 + (2.0 ** -23 if dt == "f32" else 0.0)
    vec = [sec.from_ref(torch.tensor(rng.standard_normal(D), device="cuda").to(td)) for _ in range(2)]
    host = [sec.to_ref(v).double().cpu().numpy() for v in vec]
    for ket in (0, 1):
        for pairs in (allp, some, [(n, n)]):
            raw, _ = sec.rdm_raw(vec[0], None if ket == 0 else vec[1], pairs=pairs)
            for (a, b), (q0, q1) in zip(pairs, raw):
                w0, w1, mag = _sums(n, h, host[0], host[ket], a - 1, b - 1)
                assert abs(q0 - w0) <= u * mag and abs(q1 - w1) <= u * mag, (a, b, ket)


@pytest.mark.parametrize("n", [18, 20, 22, 25, 26])
@pytest.mark.parametrize("dt", ["f32", "f64"])
def test_pair_sums_of_wide_halves(edlib, n, dt):
    """B halves of 9 to 13 sites, sectors on both sides of 2^19 states: all pairs are summed, a pair of each
    kind (two A sites, two B sites, across, equal) and some others are compared."""
    import torch
    nup = n // 2
    td = torch.float32 if dt == "f32" else torch.float64
    rng = np.random.default_rng(n)
    x = np.arange(1 << n, dtype=np.uint32)
    pop = np.array([bin(i).count("1") for i in range(1 << 13)], dtype=np.uint8)
    h = x[pop[x & 0x1FFF] + pop[x >> 13] == n - nup].astype(np.int64)
    del x
    D = len(h)
    J = np.zeros((n, n))
    for i in range(n):
        J[i, (i + 1) % n] = J[(i + 1) % n, i] = 1.0
    sec = edlib.Sector(n, nup, 0, edlib.ED_HEISENBERG, J=J)
    assert sec.dim == D
    allp = [(a, b) for a in range(1, n + 1) for b in range(1, n + 1)]
    check = [(1, 2), (n // 2, 3), (n, n - 1), (1, n), (n, n // 2), (n // 2 + 2, 2), (3, 3), (n, n)]
    u = (D + 64) * 2.0 ** -53 + (2.0 ** -23 if dt == "f32" else 0.0)
    v = sec.from_ref(torch.tensor(rng.standard_normal(D), device="cuda").to(td))
    host = sec.to_ref(v).double().cpu().numpy()
    raw, _ = sec.rdm_raw(v, None, pairs=allp)
    for a, b in check:
        q0, q1 = raw[allp.index((a, b))]
        w0, w1, mag = _sums(n, h, host, host, a - 1, b - 1)
        assert abs(q0 - w0) <= u * mag and abs(q1 - w1) <= u * mag, (a, b)
