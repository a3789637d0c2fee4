"""Hubbard products where their form changes: the one-pass kernel (small sectors,
rows of at most 128 strings; one, two and four rows per CTA) and the two passes
(slabs of several widths, whole and partial passes, odd row strides), uniform
and per-site U, on-site energies, more than 8 sites (two bytes of the energy
table), scale and dots, against the definition in FP64 torch.

Bound per element: 64 eps (|H||x|)_i; exact for integer t, U, x."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SECTORS = [(1, 1, 1), (4, 2, 0), (5, 5, 2), (6, 3, 3), (9, 1, 7), (10, 5, 4), (11, 5, 5), (11, 6, 2), (12, 5, 4),
           (12, 2, 6), (13, 2, 6), (13, 6, 3), (17, 1, 3), (16, 3, 3), (16, 8, 1)]


class _Ref:
    def __init__(self, n, us, ds, t, U):
        import torch
        self.diag = torch.zeros(len(ds), len(us), dtype=torch.float64, device="cuda")
        self.hops = []
        for side, s in (("u", us), ("d", ds)):
            order = torch.argsort(s)
            for J in range(n):
                for K in range(n):
                    bJ, bK = 1 << (n - 1 - J), 1 << (n - 1 - K)
                    if J == K:
                        e = t[J, J] * ((s & bJ) != 0).double()
                        self.diag += e[None, :] if side == "u" else e[:, None]
                        continue
                    if t[K, J] == 0.0:
                        continue
                    at = torch.nonzero(((s & bJ) != 0) & ((s & bK) == 0))[:, 0]
                    to = order[torch.searchsorted(s[order], s[at] - bJ + bK)]
                    par = torch.zeros_like(at)
                    for P in range(min(J, K) + 1, max(J, K)):
                        par += (s[at] & (1 << (n - 1 - P))) != 0
                    self.hops.append((side, at, to, t[K, J] * (1.0 - 2.0 * (par % 2).double())))
        for J in range(n):
            b = 1 << (n - 1 - J)
            self.diag += U[J] * ((ds & b) != 0).double()[:, None] * ((us & b) != 0).double()[None, :]

    def __call__(self, x, mag=False):
        y = (self.diag.abs() if mag else self.diag) * x
        for side, at, to, c in self.hops:
            c = c.abs() if mag else c
            if side == "u":
                y.index_add_(1, to, x[:, at] * c)
            else:
                y.index_add_(0, to, x[at] * c[:, None])
        return y


@pytest.mark.parametrize("n,nu,nd", SECTORS)
@pytest.mark.parametrize("dt", ["f32", "f64"])
def test_hubbard_product_forms(edlib, n, nu, nd, dt):
    import torch
    td = torch.float32 if dt == "f32" else torch.float64
    eps = torch.finfo(td).eps
    rng = np.random.default_rng(n * 100 + nu * 10 + nd)
    g = torch.Generator(device="cuda")
    g.manual_seed(n)
    for kind in ("integer", "uniform", "sites"):
        t = np.zeros((n, n))
        pairs = [(i, (i + 1) % n) for i in range(n)] + [(0, n // 2), (1 % n, n - 1)]
        for a, b in pairs:
            if a != b:
                t[a, b] = t[b, a] = rng.integers(1, 4) if kind == "integer" else rng.uniform(-1.5, 1.5)
        U = np.full(n, 4.0)
        if kind == "integer":
            U = rng.integers(0, 5, n).astype(float)
            t[np.diag_indices(n)] = rng.integers(-2, 3, n)
        elif kind == "sites":
            U = rng.uniform(1.0, 6.0, n)
            t[np.diag_indices(n)] = rng.normal(0.0, 0.3, n)
        sec = edlib.Sector(n, nu, nd, edlib.ED_HUBBARD, t=t, U=U)
        us, ds = (torch.from_numpy(s.astype(np.int64)).cuda() for s in sec.strings())
        H = _Ref(n, us, ds, t, U)
        x = torch.randn(sec.nsdn, sec.nsup, generator=g, dtype=torch.float64, device="cuda")
        if kind == "integer":
            x = torch.round(4 * x)
        x = x.to(td).double()
        want, mag = H(x), H(x.abs(), mag=True)
        scratch = torch.empty(edlib.scratch_bytes(sec.n, 1) // 8 + 1, dtype=torch.float64, device="cuda")
        for ld, scale in ((sec.ld, 1.0), (sec.ld, 0.5), (sec.nsup + 1 - sec.nsup % 2, 1.0)):
            xi = torch.zeros(sec.nsdn, ld, dtype=td, device="cuda")
            xi[:, :sec.nsup] = x.to(td)
            y = torch.full_like(xi, 9.0)
            dots = torch.zeros(2, dtype=torch.float64, device="cuda")
            sec.hv(xi.view(-1), y.view(-1), scale=scale, dots=dots, scratch=scratch, ld=ld)
            got = y[:, :sec.nsup].double()
            assert bool((y[:, sec.nsup:] == 9.0).all())       # the padding is left as it was
            if kind == "integer":
                assert torch.equal(got, scale * want)
            else:
                assert bool(((got - scale * want).abs() <= 64 * eps * scale * mag + 1e-300).all())
            tol = 1e-12 if dt == "f64" else 2e-5
            assert abs(float(dots[0]) - float((x * got).sum())) <= tol * float((x * got).abs().sum()) + 1e-300
            assert abs(float(dots[1]) - float((got * got).sum())) <= tol * float((got * got).sum()) + 1e-300


@pytest.mark.parametrize("dt", ["f32", "f64"])
@pytest.mark.parametrize("U", ["uniform", "sites"])
def test_uijkl_drops_the_on_site_interaction(edlib, dt, U):
    """A sector built with an on-site U loses it when the U_ijkl interaction is set, as one built without."""
    import torch
    td = torch.float32 if dt == "f32" else torch.float64
    n = 6
    rng = np.random.default_rng(2)
    t = rng.integers(-2, 3, (n, n)).astype(float)
    t = np.triu(t) + np.triu(t, 1).T
    Ul = rng.integers(-2, 3, (n,) * 4).astype(float)
    u = np.full(n, 3.0) if U == "uniform" else np.arange(1.0, n + 1)
    x = torch.randint(-4, 5, (400,), device="cuda").to(td)
    ys = []
    for uu in (u, np.zeros(n)):
        sec = edlib.Sector(n, 3, 3, edlib.ED_HUBBARD, t=t, U=uu)
        sec.set_uijkl(Ul)
        y = sec.zeros(td)
        sec.hv(sec.from_ref(x), y)
        ys.append(sec.to_ref(y))
    assert torch.equal(ys[0], ys[1])
