"""Heisenberg products where their passes change form: rows around one and two
128-column passes of the slab kernel (n = 16 to 22), no, few, 9 to 32 and more than
32 bonds between the halves, odd site counts, one-site halves, scale 1 and not, against the
definition over all states in FP64 torch.

Bound per element: 64 eps (|H||x|)_i (at most n(n-1)/2 + 2 terms, each rounded
twice); exact for integer J, x and scale."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _bonds(n, kind, rng):
    J = np.zeros((n, n))
    if kind == "halves":            # nothing crosses the middle
        pairs = [(a, a + 1) for a in range(n - 1) if a + 1 != n // 2]
    elif kind == "ring":
        pairs = [(a, (a + 1) % n) for a in range(n)]
    elif kind == "cross":           # 9 to 32 bonds between the halves
        h = n // 2
        pairs = [(a, (a + 1) % n) for a in range(n)] + [(a, h + b) for a in range(min(4, h)) for b in range(min(5, n - h))]
    else:
        pairs = [(a, b) for a in range(n) for b in range(a + 1, n)]
    for a, b in pairs:
        if a != b:
            J[a, b] = J[b, a] = rng.integers(1, 4)
    return J


@pytest.mark.parametrize("n", [2, 3, 5, 9, 16, 18, 19, 20, 22])
@pytest.mark.parametrize("kind", ["halves", "ring", "cross", "all"])
@pytest.mark.parametrize("dt", ["f32", "f64"])
def test_heisenberg_product(edlib, n, kind, dt):
    import torch
    if n == 22 and kind == "all":
        pytest.skip("covered by n = 20")
    td = torch.float32 if dt == "f32" else torch.float64
    rng = np.random.default_rng(n)
    Ji = _bonds(n, kind, rng)
    h = np.array([x for x in range(1 << n) if bin(x).count("1") == n - n // 2], dtype=np.int64)
    hd = torch.from_numpy(h).cuda()
    g = torch.Generator(device="cuda")
    g.manual_seed(n)
    for integer in (True, False):
        J = Ji if integer else Ji * 0.37
        sec = edlib.Sector(n, n // 2, 0, edlib.ED_HEISENBERG, J=J)
        x = torch.randint(-8, 9, (len(h),), generator=g, device="cuda").double()
        if not integer:
            x = torch.randn(len(h), generator=g, dtype=torch.float64, device="cuda")
        x = x.to(td).double()
        want, mag = torch.zeros_like(x), torch.zeros_like(x)
        for a in range(n):
            for b in range(a + 1, n):
                if J[a, b] == 0.0:
                    continue
                anti = ((hd >> a) ^ (hd >> b)) & 1
                at = torch.nonzero(anti)[:, 0]
                to = torch.searchsorted(hd, hd[at] ^ ((1 << a) | (1 << b)))
                want += 0.5 * J[a, b] * torch.where(anti == 1, -x, x)
                want[at] += -((-1.0) ** (a + b)) * J[a, b] * x[to]
                mag += 0.5 * abs(J[a, b]) * x.abs()
                mag[at] += abs(J[a, b]) * x[to].abs()
        xi = sec.from_ref(x.to(td))
        scratch = torch.empty(edlib.scratch_bytes(sec.n, 1) // 8 + 1, dtype=torch.float64, device="cuda")
        for scale in (1.0, 0.5):
            y = torch.full_like(xi, 3.0)
            dots = torch.zeros(2, dtype=torch.float64, device="cuda")
            sec.hv(xi, y, scale=scale, dots=dots, scratch=scratch)
            got = sec.to_ref(y).double()
            if integer:
                assert torch.equal(got, scale * want)
            else:
                eps = torch.finfo(td).eps
                assert bool(((got - scale * want).abs() <= 64 * eps * scale * mag + 1e-300).all())
            yx, yy = float((x * got).sum()), float((got * got).sum())
            tol = (1e-12 if dt == "f64" else 2e-5)
            assert abs(float(dots[0]) - yx) <= tol * float((x * got).abs().sum())
            assert abs(float(dots[1]) - yy) <= tol * yy


@pytest.mark.parametrize("norb", [8, 14, 20, 24, 30])
def test_fp64_equals_fp32_on_integers(edlib, norb):
    """The FP64 pass takes the columns by number of flips (in windows of 64 above 1e9 bytes: 30 sites), the
    FP32 pass in order: with couplings that are multiples of 4 and integer x every sum is an integer below
    2^24 and the products are equal."""
    import torch
    rng = np.random.default_rng(norb)
    J = np.zeros((norb, norb))
    for i in range(norb):
        for j in ((i + 1) % norb, (i + norb // 4) % norb):
            if i != j:
                J[i, j] = J[j, i] = 4.0 * rng.integers(1, 3)
    sec = edlib.Sector(norb, norb // 2, 0, edlib.ED_HEISENBERG, J=J)
    g = torch.Generator(device="cuda")
    g.manual_seed(norb)
    x = torch.randint(-2, 3, (sec.dim,), generator=g, device="cuda", dtype=torch.int8)
    ys = []
    for td in (torch.float32, torch.float64):
        y = sec.zeros(td)
        sec.hv(sec.from_ref(x.to(td)), y)
        ys.append(sec.to_ref(y).to(torch.float32))
    assert torch.equal(ys[0], ys[1])
