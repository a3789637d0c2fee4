"""Row sums of the Hubbard densities where they are cut into parts (rows of 1,024
strings or more with one or two rows at a time) and where they are not, against
FP64 torch: the sums without up hops and the up hops beside them.  Bound as in test_gpu_rdm_sizes: 1e-13 sum|b k|."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# rows at a time: 1 (12, 5 and 3 parts), 2 (6 parts), 4 (whole)
SECTORS = [(15, 7, 0), (14, 6, 1), (13, 6, 3), (14, 7, 3), (13, 6, 4), (14, 7, 4), (12, 6, 5)]


@pytest.mark.parametrize("n,nu,nd", SECTORS)
@pytest.mark.parametrize("dt", ["f32", "f64"])
@pytest.mark.parametrize("npairs", [1, 2, 15, 16, 40])
@pytest.mark.parametrize("same", [True, False])
def test_row_sums(edlib, n, nu, nd, dt, npairs, same):
    import torch
    td = torch.float32 if dt == "f32" else torch.float64
    t = np.zeros((n, n))
    t[0, 1] = t[1, 0] = 1.0
    sec = edlib.Sector(n, nu, nd, edlib.ED_HUBBARD, t=t, U=np.zeros(n))
    g = torch.Generator(device="cuda")
    g.manual_seed(n * 100 + nu * 10 + nd)
    bra, ket = (sec.from_ref(torch.randn(sec.dim, generator=g, dtype=torch.float64, device="cuda")).to(td)
                for _ in range(2))
    if same:
        ket = bra
    p = (sec.to_ref(bra).double() * sec.to_ref(ket).double()).view(sec.nsdn, sec.nsup)
    b, k = (sec.to_ref(v).double().view(sec.nsdn, sec.nsup) for v in (bra, ket))
    us, ds = (torch.from_numpy(s.astype(np.int64)).cuda() for s in sec.strings())
    rng = np.random.default_rng(npairs)
    allp = [(J, K) for J in range(1, n + 1) for K in range(1, n + 1)]
    pairs = [(n, n)] + [allp[int(i)] for i in rng.choice(len(allp), npairs - 1, replace=False)]
    raw, _ = sec.rdm_raw(bra, None if same else ket, pairs=pairs, flags=0)
    order = torch.argsort(us)
    occ = lambda s, J: ((s >> (n - J)) & 1).double()      # noqa: E731
    mag = max(float(p.abs().sum()), float(b.norm() * k.norm()))      # at least sum|b k| of any one hop
    for (J, K), q in zip(pairs, raw):
        sJ, sK = (0.5 * (occ(us, x)[None, :] - occ(ds, x)[:, None]) for x in (J, K))
        want = [0.0, float((p * sJ * sK).sum()), 0.0, 0.0]
        if J == K:
            want[0] = float((p * occ(us, J)[None, :]).sum())
            want[2] = float((p * occ(ds, J)[:, None]).sum())
            want[3] = float((p * occ(us, J)[None, :] * occ(ds, J)[:, None]).sum())
        else:
            at = torch.nonzero((occ(us, J) == 1) & (occ(us, K) == 0))[:, 0]
            to = order[torch.searchsorted(us[order], us[at] - (1 << (n - J)) + (1 << (n - K)))]
            par = sum((occ(us[at], P) for P in range(min(J, K) + 1, max(J, K))), torch.zeros(len(at), device="cuda"))
            want[0] = float((b[:, at] * k[:, to] * (1.0 - 2.0 * (par % 2))).sum())
        assert (np.abs(q[:4] - np.array(want)) <= 1e-13 * mag).all(), ((J, K), q, want)
