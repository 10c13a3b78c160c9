"""Which kernels run a call: the rule is applied at every call, also where the
step graph of the call before could run again."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _case(n=800):
    from gb300dem import workloads
    m = max(4, int(round(n ** (1 / 3))))
    c = workloads.lattice_case(5, m, m, -(-n // (m * m)), 2.05e-3, radius=(0.9e-3, 1.1e-3), jitter=5e-5, vmax=1.0,
                               wmax=300.0, dt=2e-6, skin=2e-4)
    c["atoms"] = {k: v[:n] for k, v in c["atoms"].items()}
    return c


def _launches(g, steps):
    k0, r0 = g.kernel_times()["kernel_launches"], g.nrebuilds
    g.step(steps)
    return g.kernel_times()["kernel_launches"] - k0, g.nrebuilds - r0


def test_rule_at_every_call(monkeypatch):
    from gb300dem.api import DemSystem
    case = _case()
    monkeypatch.setenv("LIGGGHTS_GB300_FUSED_STEPS", "0")
    ref = DemSystem(case)
    ref.setup()
    g = DemSystem(case)
    g.setup()
    for fused in ("1", "0", "1", "0"):
        ref.step(20)
        monkeypatch.setenv("LIGGGHTS_GB300_FUSED_STEPS", fused)
        k, reb = _launches(g, 20)
        monkeypatch.setenv("LIGGGHTS_GB300_FUSED_STEPS", "0")
        # separate kernels: at least two a step; k_steps: one, and one more with each build's some thirty
        assert (k >= 40) if fused == "0" else (k <= 2 + 50 * reb), (fused, k, reb)
    a, b = g.atoms(), ref.atoms()
    for q in a:
        assert np.array_equal(a[q], b[q]), q
