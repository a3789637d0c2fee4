"""ed_multidot and ed_update with few vectors, where the number of vectors chooses
the form: 1, 2, 3-4 and more vectors of the FP64 multi-dot at the edges of their
steps (512 elements a step, 4 or 2 steps in flight), one group's grid where it
strides, and the first count of a second group.

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


@pytest.mark.parametrize("n", [1, 2, 511, 513, 1023, 1025, 2047, 2048, 2049, 4097, 311_297, 622_593, 1_245_185])
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
