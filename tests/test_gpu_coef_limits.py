"""ed_lanczos_coef where its dynamic shared memory meets the default limit of
48 KB (k = 2,707 to 2,719 leave no room for the kernel's static arrays), each in
a process of its own, in which no larger step has raised the limit; and the
largest |G - I| entry that a step records.

The step of an orthonormal basis is exact: g = e_k, c arbitrary, Linv = I give
alpha_k = c_k and coef = c, with scales 1."""
import os
import subprocess
import sys

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

ONE_STEP = """
import sys
sys.path.insert(0, {root!r})
import torch
from pyhub_gb300 import _capi as C
k, close = {k}, {close}
m = k + 1
st = torch.zeros(C.lanczos_state_doubles(m), dtype=torch.float64, device="cuda")
st[2:2 + k] = 1.0
lin = st[3 + m:3 + m + (m + 1) ** 2].view(m + 1, m + 1)
lin[:k, :k] = torch.eye(k, dtype=torch.float64, device="cuda")
dots = torch.zeros(2 * (k + 1), dtype=torch.float64, device="cuda")
dots[:k + 1] = torch.arange(k + 1, dtype=torch.float64, device="cuda") % 7 - 3
dots[2 * k + 1] = 1.0
nrm = torch.ones(1, dtype=torch.float64, device="cuda")
coef = torch.full((k + 1,), 9.0, dtype=torch.float64, device="cuda")
ab = torch.ones(2, m, dtype=torch.float64, device="cuda")
C.lanczos_coef(k, m, None if close else dots, nrm, st, None if close else coef, ab[0], ab[1])
torch.cuda.synchronize()
assert float(st[0]) == 0.0 and float(st[2 + k]) == 1.0 and float(ab[1][k - 1]) == 1.0
if not close:
    assert torch.equal(coef, dots[:k + 1]) and float(ab[0][k]) == float(dots[k])
print("step ok")
"""


@pytest.mark.parametrize("k", [2555, 2706, 2707, 2719, 2720])
@pytest.mark.parametrize("close", [False, True])
def test_step_in_a_fresh_process(edlib, k, close):
    r = subprocess.run([sys.executable, "-c", ONE_STEP.format(root=ROOT, k=k, close=close)], capture_output=True,
                       text=True, timeout=300)
    assert r.returncode == 0 and "step ok" in r.stdout, r.stderr[-2000:]


@pytest.mark.parametrize("k", [1, 9, 300])
def test_largest_gram_entry(edlib, k):
    """state[1] holds the largest |G_k - I| entry of the steps so far: off the diagonal, on it, and kept when smaller
    ones follow.  An entry is (s_j b_j) s_k, one rounding each for scales of 1: equal to the last bit."""
    import torch
    m = k + 2
    rng = np.random.default_rng(k)
    for where in ("off", "diagonal"):
        st = torch.zeros(edlib.lanczos_state_doubles(m), dtype=torch.float64, device="cuda")
        st[2:2 + k] = 1.0
        lin = st[3 + m:3 + m + (m + 1) ** 2].view(m + 1, m + 1)
        lin[:k, :k] = torch.eye(k, dtype=torch.float64, device="cuda")
        g = rng.uniform(-1e-9, 1e-9, k + 1)
        g[k] = 1.0 + g[k]
        if where == "off":
            g[k // 2] = -3e-6
        else:
            g[k] = 1.0 - 2e-5
        want = np.abs(g - np.eye(k + 1)[k]).max()
        dots = torch.tensor(np.concatenate([np.ones(k + 1), g]), device="cuda")
        nrm = torch.ones(1, dtype=torch.float64, device="cuda")
        coef = torch.zeros(k + 2, dtype=torch.float64, device="cuda")
        ab = torch.ones(2, m, dtype=torch.float64, device="cuda")
        edlib.lanczos_coef(k, m, dots, nrm, st, coef, ab[0], ab[1])
        assert float(st[0]) == 0.0 and float(st[1]) == want
        nxt = torch.zeros(2 * (k + 2), dtype=torch.float64, device="cuda")
        nxt[2 * k + 3] = 1.0
        edlib.lanczos_coef(k + 1, m, nxt, nrm, st, coef, ab[0], ab[1])
        assert float(st[0]) == 0.0 and float(st[1]) == want


@pytest.mark.parametrize("k", [0, 1, 40])
@pytest.mark.parametrize("case", ["healthy", "breakdown", "non-finite", "stopped"])
def test_closing_call_is_part_one_of_the_step(edlib, k, case):
    """A closing call writes what the step's first part writes, bit for bit, and nothing else; a step after it agrees."""
    import torch
    m = 48
    nb = {"healthy": 2.3, "breakdown": 1e-28, "non-finite": float("inf"), "stopped": 2.3}[case]
    got = []
    for close_first in (False, True):
        st = torch.zeros(edlib.lanczos_state_doubles(m), dtype=torch.float64, device="cuda")
        st[2:3 + k] = 0.7
        if case == "stopped":
            st[0] = 3.0
        lin = st[3 + m:3 + m + (m + 1) ** 2].view(m + 1, m + 1)
        lin[:k, :k] = torch.eye(k, dtype=torch.float64, device="cuda")
        nrm = torch.tensor([nb], dtype=torch.float64, device="cuda")
        ab = torch.ones(2, m, dtype=torch.float64, device="cuda")
        if close_first:
            before = st.clone()
            edlib.lanczos_coef(k, m, None, nrm, st, None, ab[0], ab[1])
            same = torch.ones_like(st, dtype=torch.bool)
            same[0] = same[2 + k] = False
            assert torch.equal(st[same], before[same])
            first = (st[0].clone(), st[2 + k].clone(), ab.clone())
        dots = torch.zeros(2 * (k + 1), dtype=torch.float64, device="cuda")
        dots[2 * k + 1] = 1.0 / (0.49 if k == 0 else 1.0 / 2.3)
        coef = torch.full((k + 1,), 9.0, dtype=torch.float64, device="cuda")
        edlib.lanczos_coef(k, m, dots, nrm, st, coef, ab[0], ab[1])
        got.append((st.clone(), coef, ab.clone()))
    for a, b in zip(*got):
        assert torch.equal(a, b)
    st, _, ab = got[0]
    assert torch.equal(first[0], st[0]) and torch.equal(first[1], st[2 + k])
    if k:
        assert torch.equal(first[2][1], ab[1])
    want = {"healthy": 0.0, "breakdown": float(k), "non-finite": -float(k), "stopped": 3.0}[case]
    assert float(st[0]) == (want if k else (3.0 if case == "stopped" else 0.0))
