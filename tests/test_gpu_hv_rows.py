"""Hubbard products of rows that are short against a pass of the slab kernel (256
columns): whole chunks, a short chunk, a column per lane, each in both types;
the sectors on both sides of the one-pass line for rows of 120 strings; per-site
U with few doubly occupied sites.

The definition in FP64 torch, with the bounds of test_gpu_hv_forms (64 eps (|H||x|)_i
per element, exact for integers)."""
import numpy as np
import pytest

from test_gpu_hv_forms import _Ref

pytestmark = pytest.mark.gpu

# strings per row: 120 (one pass, then two), 136, 153, 190, 210, 276, 364, 495, 715
SECTORS = [(16, 2, 5), (16, 2, 7), (17, 2, 5), (18, 2, 5), (20, 2, 4), (21, 2, 4), (24, 2, 3), (14, 3, 5), (12, 4, 5),
           (13, 4, 4), (25, 1, 3), (17, 15, 5)]


@pytest.mark.parametrize("n,nu,nd", SECTORS)
@pytest.mark.parametrize("dt", ["f32", "f64"])
@pytest.mark.parametrize("kind", ["integer", "uniform", "sites"])
def test_products_of_short_rows(edlib, n, nu, nd, dt, kind):
    import torch
    td = torch.float32 if dt == "f32" else torch.float64
    eps = torch.finfo(td).eps
    rng = np.random.default_rng(n * 100 + nu * 10 + nd)
    t = np.zeros((n, n))
    for a, b in [(i, (i + 1) % n) for i in range(n)] + [(0, n // 2), (1, n - 1)]:
        t[a, b] = t[b, a] = rng.integers(1, 4) if kind == "integer" else rng.uniform(-1.5, 1.5)
    U = np.full(n, 4.0) if kind == "uniform" else rng.integers(0, 5, n).astype(float)
    if kind == "sites":
        U = rng.uniform(1.0, 6.0, n)
    if kind != "uniform":
        t[np.diag_indices(n)] = rng.integers(-2, 3, n)
    sec = edlib.Sector(n, nu, nd, edlib.ED_HUBBARD, t=t, U=U)
    us, ds = (torch.from_numpy(s.astype(np.int64)).cuda() for s in sec.strings())
    H = _Ref(n, us, ds, t, U)
    g = torch.Generator(device="cuda")
    g.manual_seed(n)
    x = torch.randn(sec.nsdn, sec.nsup, generator=g, dtype=torch.float64, device="cuda")
    if kind == "integer":
        x = torch.round(4 * x)
    x = x.to(td).double()
    want, mag = H(x), H(x.abs(), mag=True)
    scratch = torch.empty(edlib.scratch_bytes(sec.n, 1) // 8 + 1, dtype=torch.float64, device="cuda")
    for ld, scale in ((sec.ld, 1.0), (sec.ld, 0.5), (sec.nsup + 1 - sec.nsup % 2, 1.0), (sec.nsup + sec.nsup % 2, 1.0)):
        xi = torch.full((sec.nsdn, ld), float("nan"), dtype=td, device="cuda")      # padding is not read into a result
        xi[:, :sec.nsup] = x.to(td)
        y = torch.full((sec.nsdn, ld), 9.0, dtype=td, device="cuda")
        dots = torch.zeros(2, dtype=torch.float64, device="cuda")
        sec.hv(xi.view(-1), y.view(-1), scale=scale, dots=dots, scratch=scratch, ld=ld)
        got = y[:, :sec.nsup].double()
        assert bool((y[:, sec.nsup:] == 9.0).all())
        if kind == "integer":
            assert torch.equal(got, scale * want)
        else:
            assert bool(((got - scale * want).abs() <= 64 * eps * scale * mag + 1e-300).all())
        tol = 1e-12 if dt == "f64" else 2e-5
        assert abs(float(dots[0]) - float((x * got).sum())) <= tol * float((x * got).abs().sum()) + 1e-300
        assert abs(float(dots[1]) - float((got * got).sum())) <= tol * float((got * got).sum()) + 1e-300
        y2 = torch.full_like(y, 9.0)
        sec.hv(xi.view(-1), y2.view(-1), scale=scale, ld=ld)
        assert torch.equal(y2, y)           # the dots change nothing
