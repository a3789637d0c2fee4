"""ed_multidot and ed_update over the sizes where their launch changes form:
below, at and past a tile, the switch from the split update to 4 and to 16
elements per thread, vector counts around the 8-vector groups.

Tolerances, from the order of summation (u = unit roundoff of the vectors):
  multi-dot  FP64: a thread's sum is at most n / 256 + 1 products long, then
             8 + 5 + 1024 / 32 additions: (n / 256 + 48) u sum|v w|.
             FP32: 16 products and 5 shuffles in FP32: 22 u sum|v w|.
  update     (nvec + 4) u (|ws w| + sum |c v|) per element; its norm over 16
             elements in u, then FP64: 17 u + n 2^-53, relative, and
             (FP64) (n + 48) 2^-53.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = [1, 127, 512, 513, 4095, 4100, 311_292, 311_300, 2_490_372]


@pytest.mark.parametrize("dt", ["f32", "f64"])
@pytest.mark.parametrize("n", SIZES)
@pytest.mark.parametrize("nvec", [1, 5, 8, 11, 33])
def test_multidot_update_sizes(edlib, dt, n, nvec):
    import torch
    td = torch.float32 if dt == "f32" else torch.float64
    u = 2.0 ** -24 if dt == "f32" else 2.0 ** -53
    ld = (n + 31) // 32 * 32
    g = torch.Generator(device="cuda")
    g.manual_seed(n + nvec)
    V = torch.randn((nvec, ld), generator=g, dtype=td, device="cuda")
    w = torch.randn(ld, generator=g, dtype=td, device="cuda")
    z = torch.randn(ld, generator=g, dtype=td, device="cuda")
    scratch = torch.empty(edlib.scratch_bytes(n, nvec) // 8 + 1, dtype=torch.float64, device="cuda")
    V64, w64, z64 = V[:, :n].double(), w[:n].double(), z[:n].double()
    rel = 22 * u if dt == "f32" else (n / 256 + 48) * u
    for zz in (None, z):
        m = nvec if zz is None else 2 * nvec
        out = torch.full((m + 1,), float("nan"), dtype=torch.float64, device="cuda")
        edlib.multidot(V, nvec, w, out, scratch, z=zz, n=n)
        for j in range(m):
            v, x = V64[j % nvec], (w64 if j < nvec else z64)
            bound = 1.05 * rel * float((v * x).abs().sum())
            assert abs(float(out[j]) - float((v * x).sum())) <= bound, (j, zz is None)
        assert torch.isnan(out[m])      # nothing past the sums
    coef = torch.randn(nvec, generator=g, dtype=torch.float64, device="cuda")
    ws = torch.tensor([0.75], dtype=torch.float64, device="cuda")
    for start, scale in ((w, ws), (w, None), (None, None)):
        out = torch.full((ld,), -7.0, dtype=td, device="cuda")
        nrm = torch.zeros(2, dtype=torch.float64, device="cuda")
        edlib.update(V, nvec, coef, start, out, norm2=nrm, scratch=scratch, n=n, wscale=scale)
        s = 1.0 if scale is None else 0.75
        head = 0.0 * w64 if start is None else s * w64
        c = coef.to(td).double()
        want = head - c @ V64
        mag = head.abs() + c.abs() @ V64.abs()
        assert bool(((out[:n].double() - want).abs() <= 1.05 * (nvec + 4) * u * mag).all())
        assert bool((out[n:] == -7.0).all())
        got = float((out[:n].double() ** 2).sum())
        tol = (17 * u + n * 2.0 ** -53) if dt == "f32" else (n + 48) * u
        assert abs(float(nrm[0]) - got) <= 1.05 * tol * got
