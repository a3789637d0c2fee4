"""ed_hv_launches against the kernels that a product enqueues, counted in a
captured graph, and the launch count of a timed Lanczos run."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _kernel_nodes(call):
    """Kernel nodes of what `call(stream)` enqueues (libcudart's capture; nothing runs)."""
    import torch
    rt = ctypes.CDLL(f"libcudart.so.{torch.version.cuda.split('.')[0]}")
    side = torch.cuda.Stream()
    st, graph, n = ctypes.c_void_p(side.cuda_stream), ctypes.c_void_p(), ctypes.c_size_t()
    assert rt.cudaStreamBeginCapture(st, 1) == 0
    call(side)
    assert rt.cudaStreamEndCapture(st, ctypes.byref(graph)) == 0
    assert rt.cudaGraphGetNodes(graph, None, ctypes.byref(n)) == 0
    nodes = (ctypes.c_void_p * n.value)()
    assert rt.cudaGraphGetNodes(graph, nodes, ctypes.byref(n)) == 0
    kinds = []
    for v in nodes:
        k = ctypes.c_int()
        assert rt.cudaGraphNodeGetType(ctypes.c_void_p(v), ctypes.byref(k)) == 0
        kinds.append(k.value)
    assert rt.cudaGraphDestroy(graph) == 0
    return kinds.count(0)      # cudaGraphNodeTypeKernel


@pytest.mark.parametrize("case", [(1, 1, 0), (6, 3, 3), (11, 5, 5), (12, 6, 5), (16, 2, 5), (16, 2, 8), (20, 1, 5), "heis",
                                  "uijkl"])
@pytest.mark.parametrize("dt", ["f32", "f64"])
def test_launches_of_a_product(edlib, case, dt):
    import torch
    td = torch.float32 if dt == "f32" else torch.float64
    if case == "heis":
        J = np.ones((8, 8)) - np.eye(8)
        sec = edlib.Sector(8, 4, 0, edlib.ED_HEISENBERG, J=J)
    else:
        n, nu, nd = (5, 2, 2) if case == "uijkl" else case
        t = np.ones((n, n)) - np.eye(n)
        sec = edlib.Sector(n, nu, nd, edlib.ED_HUBBARD, t=t, U=np.full(n, 2.0))
        if case == "uijkl":
            sec.set_uijkl(np.ones((n,) * 4))
    x = torch.zeros(sec.n, dtype=td, device="cuda")
    y = torch.zeros_like(x)
    sec.hv(x, y)
    torch.cuda.synchronize()
    assert sec.hv_launches(td) == _kernel_nodes(lambda s: sec.hv(x, y, stream=s))


def test_timed_run_counts_the_sectors_launches(edlib):
    import torch
    from pyhub_gb300.core import lanczos as LZ
    n = 6
    t = np.diag(np.ones(n - 1), 1)
    sec = edlib.Sector(n, 3, 3, edlib.ED_HUBBARD, t=t + t.T, U=np.full(n, 2.0))
    timer = LZ.KernelTimer()
    LZ.lanczos_full(sec, LZ.start_vector(sec, 0), 7, timer=timer)
    torch.cuda.synchronize()
    assert sec.hv_launches(torch.float64) == 1
    s = timer.summary()
    assert s["hv"]["launches"] == 7 and s["multidot"]["launches"] == 14 and s["coef"]["launches"] == 7
    assert timer.launches() == sum(v["launches"] for v in s.values())
