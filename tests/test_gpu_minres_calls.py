"""ed_minres as a call: what it promises its caller about streams and buffers."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _case(edlib, n=8, nu=4, nd=4):
    """A sector, a unit vector psi and a right-hand side (psi need not be an eigenvector)."""
    import torch
    rng = np.random.default_rng(11)
    t = np.zeros((n, n))
    for i in range(n):
        t[i, (i + 1) % n] = t[(i + 1) % n, i] = -rng.uniform(0.5, 1.5)
    sec = edlib.Sector(n, nu, nd, edlib.ED_HUBBARD, t=t, U=rng.uniform(2.0, 6.0, n))
    g = torch.Generator(device="cuda")
    g.manual_seed(4)
    psi = sec.from_ref(torch.randn(sec.dim, generator=g, dtype=torch.float64, device="cuda"))
    psi /= torch.linalg.vector_norm(psi)
    b = sec.from_ref(torch.randn(sec.dim, generator=g, dtype=torch.float64, device="cuda"))
    return sec, psi, b


@pytest.mark.parametrize("shape", [(8, 4, 4), (11, 5, 5), (12, 6, 6)])
@pytest.mark.parametrize("maxiter", [0, 3])
def test_the_stream_is_idle_when_the_call_returns(edlib, shape, maxiter):
    import torch
    sec, psi, b = _case(edlib, *shape)
    torch.cuda.synchronize()
    side = torch.cuda.Stream()
    for _ in range(5):
        with torch.cuda.stream(side):
            sec.minres(psi, -30.0, b, maxiter, 1e-10)
            assert side.query()


@pytest.mark.parametrize("kind", ["stream", "handle"])
def test_a_stream_of_its_own_waits_for_the_current_one(edlib, kind):
    """The current stream is held up by a bounded spin: what Sector.minres enqueues there (x, b's last write) comes first."""
    import torch
    sec, psi, b = _case(edlib)
    want, it0, rr0 = sec.minres(psi, -30.0, b, 6, 0.0)
    late = torch.zeros_like(b)
    torch.cuda.synchronize()
    side = torch.cuda.Stream()
    torch.cuda._sleep(100_000_000)      # ~50 ms
    late.copy_(b)
    x, it, rr = sec.minres(psi, -30.0, late, 6, 0.0, stream=side if kind == "stream" else side.cuda_stream)
    torch.cuda.synchronize()
    assert torch.equal(x, want) and (it, rr) == (it0, rr0)


def test_the_default_streams_handle(edlib):
    import torch
    sec, psi, b = _case(edlib)
    want, it0, rr0 = sec.minres(psi, -30.0, b, 6, 0.0)
    torch.cuda.synchronize()
    with torch.cuda.stream(torch.cuda.Stream()):
        x, it, rr = sec.minres(psi, -30.0, b, 6, 0.0, stream=0)
    assert torch.equal(x, want) and (it, rr) == (it0, rr0)


def test_overlapping_buffers_are_refused(edlib):
    import ctypes
    import torch
    sec, psi, b = _case(edlib)
    L = edlib.lib()
    nb = int(L.ed_minres_scratch_bytes(sec.handle, sec.ld))
    scratch = torch.empty(nb // 8 + 1, dtype=torch.float64, device="cuda")
    x = torch.full_like(b, 3.0)
    wide = torch.zeros(2 * sec.n, dtype=torch.float64, device="cuda")
    it, rr = ctypes.c_int(), ctypes.c_double()

    def call(p, r, xx, sc):
        return L.ed_minres(sec.handle, None, sec.ld, p, -30.0, r, xx, 3, 1e-10, ctypes.byref(it), ctypes.byref(rr),
                           sc, nb)

    P, B, X, S, W = (v.data_ptr() for v in (psi, b, x, scratch, wide))
    keep = (psi.clone(), b.clone())
    for args in ((P, B, B, S), (P, B, P, S), (P, W, W + 8 * (sec.n - 1), S), (P, W + 8 * (sec.n - 1), W, S),
                 (P, B, S, S), (S, B, X, S), (P, S + 8, X, S)):
        assert call(*args) == edlib.ED_ERR_ARG
        assert "alias" in L.ed_last_error().decode()
    torch.cuda.synchronize()
    assert torch.equal(psi, keep[0]) and torch.equal(b, keep[1]) and bool((x == 3.0).all())
    # side by side and b = psi are fine
    assert call(P, W, W + 8 * sec.n, S) == edlib.ED_OK
    assert call(P, P, X, S) == edlib.ED_OK


@pytest.mark.parametrize("maxiter,rtol", [(0, 1e-10), (-3, 1e-10), (4, -1.0), (4, float("nan"))])
def test_odd_limits_run_as_the_torch_recurrence(edlib, maxiter, rtol):
    """No iterations for maxiter <= 0 (x = 0, residual 1); a tolerance that cannot be met runs to maxiter."""
    import torch
    from pyhub_gb300.core import gradients as GR
    sec, psi, b = _case(edlib)
    work = torch.zeros_like(b)

    def apply(v):
        sec.hv(v, work)
        return work + 30.0 * v

    x0, it0, rr0 = GR.minres(apply, b, psi, maxiter=maxiter, rtol=rtol)
    x, it, rr = sec.minres(psi, -30.0, b, maxiter, rtol)
    assert it == it0 and abs(rr - rr0) <= 1e-10
    # both recurrences agree to rounding: a few iterations of a system of condition ~10
    assert float(torch.linalg.vector_norm(x - x0)) <= 1e-12 * float(torch.linalg.vector_norm(x0))
