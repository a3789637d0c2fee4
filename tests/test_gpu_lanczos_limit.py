"""lanczos_full at the largest basis that a step takes (1,600 vectors): a run that
converges at the last check before it ends there, although the steps enqueued
ahead of that check would pass the limit; a run that needs more is refused."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _sector(edlib):
    n = 8
    rng = np.random.default_rng(3)
    t = np.triu(rng.normal(size=(n, n)))
    return edlib.Sector(n, 4, 4, edlib.ED_HUBBARD, t=t + t.T, U=rng.uniform(1.0, 5.0, n))


def _rule(stop_at):
    def rule(val, step):
        return step >= stop_at
    return rule


@pytest.mark.parametrize("lookahead", [True, False])
def test_converges_at_the_last_check_before_the_limit(edlib, lookahead):
    from pyhub_gb300.core import lanczos as LZ
    sec = _sector(edlib)
    r = LZ.lanczos_full(sec, LZ.start_vector(sec, 1), 1700, rule=_rule(1596), check_every=7, min_steps=1590,
                        lookahead=lookahead)
    assert r.steps == 1596 and r.converged and not r.breakdown
    # 1,596 of 4,900 dimensions: the lowest pair has converged
    y = sec.zeros(r.psi.dtype)
    sec.hv(r.psi, y)
    assert float((y - r.ritz[0] * r.psi).norm()) <= 1e-10


def test_a_longer_run_is_refused(edlib):
    from pyhub_gb300.core import lanczos as LZ
    sec = _sector(edlib)
    with pytest.raises(edlib.EDError, match="too large"):
        LZ.lanczos_full(sec, LZ.start_vector(sec, 1), 1700, rule=_rule(1650), check_every=7, min_steps=1590)
