"""ed_sector_set_uijkl against products on other streams: a product enqueued (or
captured in a graph) before the call keeps the on-site U it was enqueued with,
one enqueued after it has none, whatever the streams' order of execution.

Both are compared bit for bit with the products of sectors that are only ever
one or the other.  The streams are held up by a bounded spin of torch's own, so
that the first product runs after the call, and work on the default stream
after the second."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

N, NU, ND = 6, 3, 2


def _case(edlib, dt, U):
    import torch
    td = torch.float32 if dt == "f32" else torch.float64
    rng = np.random.default_rng(7)
    t = rng.integers(-2, 3, (N, N)).astype(float)
    t = np.triu(t) + np.triu(t, 1).T
    u = np.full(N, 3.0) if U == "uniform" else np.arange(1.0, N + 1)
    mk = lambda uu: edlib.Sector(N, NU, ND, edlib.ED_HUBBARD, t=t, U=uu)   # noqa: E731
    sec, with_u, without = mk(u), mk(u), mk(np.zeros(N))
    x = sec.from_ref(torch.randint(-4, 5, (sec.dim,), device="cuda").to(td))
    want = []
    for s in (with_u, without):
        y = s.zeros(td)
        s.hv(x, y)
        want.append(y)
    torch.cuda.synchronize()
    assert not torch.equal(*want)
    return sec, x, want[0], want[1], rng


@pytest.mark.parametrize("dt", ["f32", "f64"])
@pytest.mark.parametrize("U", ["uniform", "sites"])
def test_enqueued_product_keeps_its_interaction(edlib, dt, U):
    import torch
    sec, x, with_u, without, _ = _case(edlib, dt, U)
    y1, y2 = torch.zeros_like(x), torch.zeros_like(x)
    torch.cuda.synchronize()
    side = torch.cuda.Stream()
    with torch.cuda.stream(side):
        torch.cuda._sleep(100_000_000)     # ~50 ms
        sec.hv(x, y1)
    sec.set_uijkl(np.zeros((N,) * 4))
    with torch.cuda.stream(side):
        sec.hv(x, y2)
    torch.cuda.synchronize()
    assert torch.equal(y1, with_u)
    assert torch.equal(y2, without)


@pytest.mark.parametrize("dt", ["f32", "f64"])
@pytest.mark.parametrize("U", ["uniform", "sites"])
def test_product_ahead_of_the_default_stream(edlib, dt, U):
    import torch
    sec, x, _, without, _ = _case(edlib, dt, U)
    y = torch.zeros_like(x)
    torch.cuda.synchronize()
    side = torch.cuda.Stream()
    torch.cuda._sleep(100_000_000)
    sec.set_uijkl(np.zeros((N,) * 4))
    with torch.cuda.stream(side):
        sec.hv(x, y)
    side.synchronize()
    assert torch.equal(y, without)
    torch.cuda.synchronize()


@pytest.mark.parametrize("dt", ["f32", "f64"])
@pytest.mark.parametrize("U", ["uniform", "sites"])
def test_captured_product_keeps_its_interaction(edlib, dt, U):
    import torch
    sec, x, with_u, without, rng = _case(edlib, dt, U)
    y = torch.zeros_like(x)
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        sec.hv(x, y)
    sec.set_uijkl(np.zeros((N,) * 4))
    g.replay()
    torch.cuda.synchronize()
    assert torch.equal(y, with_u)
    sec.hv(x, y)
    assert torch.equal(y, without)
    Ul = rng.integers(-2, 3, (N,) * 4).astype(float)
    sec.set_uijkl(Ul)                       # terms, then none again
    sec.hv(x, y)
    assert not torch.equal(y, without)
    sec.set_uijkl(np.zeros((N,) * 4))
    sec.hv(x, y)
    assert torch.equal(y, without)
