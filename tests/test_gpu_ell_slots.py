"""FP32 products through the packed hop table (one word a slot where the hoppings have one or two magnitudes,
else two), whose slots without a hop read zero columns behind the staged ones: rows of every residue mod 8 and of whole slices, strings without a hop, few and many bonds,
each kernel that stages rows (one and four rows per CTA, batched 4, 8 and 16).

Integer t, U and x keep every sum below 2^24, so the FP32 products equal the FP64 ones; a NaN of x
reaches the same elements in both."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# (sites, N_up, N_dn, bonds): C(n, N_up) up strings
ROWS = [(12, 5, 6, 12), (12, 6, 5, 60), (13, 4, 5, 20), (13, 5, 4, 3), (17, 8, 2, 17), (17, 7, 2, 30), (17, 9, 3, 20)]


def _t(n, bonds, rng, mags):
    t = np.zeros((n, n))
    for _ in range(bonds):
        a, b = rng.choice(n, 2, replace=False)
        t[a, b] = t[b, a] = rng.choice([-1, 1]) * rng.integers(1, mags + 1)
    return t


@pytest.mark.parametrize("mags", [1, 2, 3])
@pytest.mark.parametrize("n,nu,nd,bonds", ROWS)
def test_row_products_equal_fp64(edlib, n, nu, nd, bonds, mags):
    import torch
    rng = np.random.default_rng(n + nu)
    sec = edlib.Sector(n, nu, nd, edlib.ED_HUBBARD, t=_t(n, bonds, rng, mags), U=rng.integers(0, 5, n).astype(float))
    x = torch.randint(-4, 5, (sec.nsdn * sec.nsup,), device="cuda").double()
    for nan in (False, True):
        if nan:
            x[rng.integers(0, x.numel(), 3)] = float("nan")
        ys = []
        for td in (torch.float32, torch.float64):
            y = sec.zeros(td)
            sec.hv(sec.from_ref(x.to(td)), y)
            ys.append(sec.to_ref(y).double())
        assert torch.equal(torch.isnan(ys[0]), torch.isnan(ys[1]))
        assert torch.equal(torch.nan_to_num(ys[0]), torch.nan_to_num(ys[1]))


@pytest.mark.parametrize("rows", [4, 8, 16])
def test_batched_products_equal_fp64(edlib, rows):
    import torch
    from pyhub_gb300 import _capi
    rng = np.random.default_rng(rows)
    shapes = [(4, 0, 2), (5, 1, 2), (8, 1, 3), (6, 3, 2), (6, 2, 3), (7, 3, 3), (8, 4, 1), (8, 3, 4), (12, 5, 2), (9, 3, 3)]
    secs = [edlib.Sector(n, nu, nd, edlib.ED_HUBBARD, t=_t(n, n, rng, 1 + i % 3), U=rng.integers(0, 5, n).astype(float))
            for i, (n, nu, nd) in enumerate(shapes)]
    b = _capi.Batch(secs, rows=rows)
    scratch = torch.empty(b.scratch_bytes() // 8 + 1, dtype=torch.float64, device="cuda")
    xs = [torch.randint(-4, 5, (s.nsdn * s.nsup,), device="cuda").double() for s in secs]
    ys = []
    for td in (torch.float32, torch.float64):
        x = torch.zeros(b.total, dtype=td, device="cuda")
        for i, s in enumerate(secs):
            b.view(x, i).copy_(s.from_ref(xs[i].to(td)))
        y = torch.full_like(x, float("nan"))
        b.hv(x, y, scratch)
        ys.append([s.to_ref(b.view(y, i)).double() for i, s in enumerate(secs)])
    for y32, y64 in zip(*ys):
        assert torch.equal(y32, y64)
