"""ed_rdm on Hubbard sectors where its launch changes form (one, two and four
rows at a time, by rows per SM and by bra = ket; one and several column tiles;
odd and even site counts; unequal fillings; 17 sites), every quantity against
its definition in FP64 torch.

Each sum is at most D products deep: |err| <= (D^(1/2) + 64) 2^-53 sum|b k| for
random signs of the partial sums' roundings; D below 9e5: 1e-13 sum|b k|.
FP32 vectors are widened exactly, so the same bound holds."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SECTORS = [(2, 1, 1), (3, 2, 1), (5, 2, 4), (6, 3, 3), (7, 7, 2), (9, 4, 5), (11, 3, 5), (12, 6, 6), (12, 2, 6),
           (17, 2, 3)]


@pytest.mark.parametrize("n,nu,nd", SECTORS)
@pytest.mark.parametrize("dt", ["f32", "f64"])
@pytest.mark.parametrize("same", [True, False])
def test_rdm_quantities(edlib, n, nu, nd, dt, same):
    import torch
    td = torch.float32 if dt == "f32" else torch.float64
    t = np.zeros((n, n))
    for i in range(n - 1):
        t[i, i + 1] = t[i + 1, i] = -1.0
    sec = edlib.Sector(n, nu, nd, edlib.ED_HUBBARD, t=t, U=np.full(n, 4.0))
    g = torch.Generator(device="cuda")
    g.manual_seed(n * 100 + nu * 10 + nd)
    vec = [sec.from_ref(torch.randn(sec.dim, generator=g, dtype=torch.float64, device="cuda")).to(td) for _ in range(2)]
    bra, ket = vec[0], (vec[0] if same else vec[1])
    b, k = (sec.to_ref(v).double().view(sec.nsdn, sec.nsup) for v in (bra, ket))
    us, ds = (torch.from_numpy(s.astype(np.int64)).cuda() for s in sec.strings())
    rng = np.random.default_rng(n)
    allp = [(J, K) for J in range(1, n + 1) for K in range(1, n + 1)]
    pairs = allp if n < 8 else [allp[int(i)] for i in rng.choice(len(allp), 12, replace=False)] + [(1, 1), (n, n), (n, 1)]
    raw, _ = sec.rdm_raw(bra, None if same else ket, pairs=pairs, flags=3)

    def bit(J):
        return 1 << (n - J)

    def hop(s, J, K):     # J occupied, K empty: where the particle moved to K lands, and the sign
        at = torch.nonzero(((s & bit(J)) != 0) & ((s & bit(K)) == 0))[:, 0]
        to = s[at] - bit(J) + bit(K)
        order = torch.argsort(s)
        to = order[torch.searchsorted(s[order], to)]
        par = torch.zeros_like(at)
        for P in range(min(J, K) + 1, max(J, K)):
            par += (s[at] & bit(P)) != 0
        return at, to, 1.0 - 2.0 * (par % 2).double()

    p = b * k
    for (J, K), q in zip(pairs, raw):
        nuJ, nuK = (((us & bit(x)) != 0).double() for x in (J, K))
        ndJ, ndK = (((ds & bit(x)) != 0).double() for x in (J, K))
        sz = 0.25 * (nuJ[None, :] - ndJ[:, None]) * (nuK[None, :] - ndK[:, None])
        want, mag = np.zeros(6), np.zeros(6)
        terms = {1: p * sz}
        if J == K:
            terms.update({0: p * nuJ[None, :], 2: p * ndJ[:, None], 3: p * nuJ[None, :] * ndJ[:, None]})
        else:
            at, to, sg = hop(us, J, K)
            dat, dto, dsg = hop(ds, J, K)
            rat, rto, rsg = hop(ds, K, J)
            terms.update({0: b[:, at] * k[:, to] * sg, 4: b[dat] * k[dto] * dsg[:, None],
                          5: -(b[rat][:, at] * k[rto][:, to] * sg * rsg[:, None])})
        for i, v in terms.items():
            want[i], mag[i] = float(v.sum()), float(v.abs().sum()) + (float(p.abs().sum()) if i in (1, 3) else 0.0)
        assert (np.abs(q - want) <= 1e-13 * mag + 1e-300).all(), ((J, K), q, want)
