"""ed_multidot and ed_update with few vectors, where the number of vectors chooses
the form: 1 to 4 and more vectors of the FP64 multi-dot at the edges of their
steps (512 elements a step, 4 or 2 steps in flight past 77,824 elements), one
group's grid where it strides, and the first count of a second group.

Tolerances, from the order of summation (u = 2^-53): a thread's sum is at most
n / 512 products long, then 8 lanes' and warps' additions and at most 1,024
partial rows: (n / 256 + 48) u sum|v w|, and the same for a norm."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _vectors(n, nvec, td, seed):
    import torch
    ld = (n + 31) // 32 * 32
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    V = torch.randn((nvec, ld), generator=g, dtype=td, device="cuda")
    V[:, n:] = float("nan")           # what lies past a vector is never read into a sum
    w = torch.randn(ld, generator=g, dtype=td, device="cuda")
    z = torch.randn(ld, generator=g, dtype=td, device="cuda")
    return ld, V, w, z, g


@pytest.mark.parametrize("n", [1, 2, 511, 513, 1025, 2049, 77_824, 77_825, 79_871, 79_873, 80_897, 311_297, 622_593,
                               1_245_185])
@pytest.mark.parametrize("nvec", [1, 2, 3, 4, 5, 8, 9])
def test_multidot_few_vectors(edlib, n, nvec):
    import torch
    ld, V, w, z, _ = _vectors(n, nvec, torch.float64, 7 * n + nvec)
    scratch = torch.full((edlib.scratch_bytes(n, nvec) // 8 + 1,), float("nan"), dtype=torch.float64, device="cuda")
    for zz in (None, z):
        m = nvec if zz is None else 2 * nvec
        out = torch.full((m + 1,), float("nan"), dtype=torch.float64, device="cuda")
        edlib.multidot(V, nvec, w, out, scratch, z=zz, n=n)
        got = out.cpu().numpy()
        for j in range(m):
            p = V[j % nvec, :n] * (w if j < nvec else z)[:n]
            assert abs(got[j] - float(p.sum())) <= 1.05 * (n / 256 + 48) * 2.0 ** -53 * float(p.abs().sum()), (j, zz is None)
        assert np.isnan(got[m])


# (elements, vectors) on both sides of every line between the split, the 4 x 128 and the 16 x 256 form
UPDATE = [(38_912, 3), (38_912, 4), (38_913, 4), (38_913, 15), (63_488, 10), (63_488, 11), (63_488, 24), (63_488, 25),
          (200_000, 5), (200_000, 34), (200_000, 63), (200_000, 64), (311_296, 1), (311_296, 9), (311_296, 54),
          (311_297, 8), (311_297, 64), (853_888, 23), (853_888, 24), (1_048_576, 28), (1_048_576, 29),
          (1_048_577, 100), (1_048_577, 1)]


@pytest.mark.parametrize("n,nvec", UPDATE)
@pytest.mark.parametrize("dt", ["f32", "f64", "f32-f64", "f64-f32"])
def test_update_forms(edlib, n, nvec, dt):
    """Per element (nvec + 4) u (|ws w| + sum |c v|), u that of the accumulation, and one rounding to the output's
    type; the norm over 16 elements in FP32, then FP64: 17 u + n 2^-53 (FP64: (n / 256 + 48) 2^-53)."""
    import torch
    td = torch.float32 if dt.startswith("f32") else torch.float64
    od = torch.float32 if dt in ("f32", "f64-f32") else torch.float64
    u = 2.0 ** -24 if dt == "f32" else 2.0 ** -53
    uo = 2.0 ** -24 if od == torch.float32 else 2.0 ** -53
    ld, V, w, z, g = _vectors(n, nvec, td, n + nvec)
    w = w.to(od)
    coef = torch.randn(nvec, generator=g, dtype=torch.float64, device="cuda")
    scratch = torch.full((edlib.scratch_bytes(n, nvec) // 8 + 1,), float("nan"), dtype=torch.float64, device="cuda")
    V64, c = V[:, :n].double(), coef.to(torch.float32).double() if dt == "f32" else coef
    ws = torch.tensor([0.75], dtype=torch.float64, device="cuda")
    for start, in_place in ((w, False), (w.clone(), True), (None, False)):
        head = 0.75 * start[:n].double() if start is not None else torch.zeros(n, dtype=torch.float64, device="cuda")
        want, mag = head - c @ V64, head.abs() + c.abs() @ V64.abs()
        out = start if in_place else torch.full((ld,), -7.0, dtype=od, device="cuda")
        tail = out[n:].clone()
        nrm = torch.zeros(2, dtype=torch.float64, device="cuda")
        edlib.update(V, nvec, coef, start, out, norm2=nrm, scratch=scratch, n=n, wscale=None if start is None else ws)
        assert bool(((out[:n].double() - want).abs() <= 1.05 * ((nvec + 4) * u * mag + uo * want.abs())).all())
        assert torch.equal(out[n:], tail)
        got = float((out[:n].double() ** 2).sum())
        tol = 17 * uo + n * 2.0 ** -53 if od == torch.float32 else (n / 256 + 48) * 2.0 ** -53
        assert abs(float(nrm[0]) - got) <= 1.05 * tol * got


@pytest.mark.parametrize("n,nvec", [(36, 1), (38_912, 1), (38_913, 2), (77_824, 7), (77_824, 8), (77_825, 1),
                                    (131_072, 6), (131_072, 48), (200_000, 10), (311_296, 47), (311_297, 3),
                                    (1_048_576, 3), (1_048_577, 3), (1_245_185, 3), (1_245_185, 4)])
@pytest.mark.parametrize("dt", ["f32", "f64"])
def test_update_forms_without_a_norm(edlib, n, nvec, dt):
    """The lines lie elsewhere where no norm is asked for; same bound per element."""
    import torch
    td = torch.float32 if dt == "f32" else torch.float64
    u = 2.0 ** -24 if dt == "f32" else 2.0 ** -53
    ld, V, w, z, g = _vectors(n, nvec, td, n - nvec)
    coef = torch.randn(nvec, generator=g, dtype=torch.float64, device="cuda")
    c = coef.to(td).double()
    want, mag = w[:n].double() - c @ V[:, :n].double(), w[:n].double().abs() + c.abs() @ V[:, :n].double().abs()
    out = torch.full((ld,), -7.0, dtype=td, device="cuda")
    edlib.update(V, nvec, coef, w, out, n=n)
    assert bool(((out[:n].double() - want).abs() <= 1.05 * (nvec + 5) * u * mag).all())
    assert bool((out[n:] == -7.0).all())
