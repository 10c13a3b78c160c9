"""Short calls of small systems, which launch the fused kernel without a graph,
against the separate kernels in a graph: rebuilds on any step of a call, a list
that outgrows its capacity, a moving mesh, bonds; short and long calls mixed.
The bits and the counts are the same."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _case(name):
    from gb300dem import workloads
    from golden_io import load_golden
    if name in ("mixer_rotate", "fibre_press"):
        return load_golden(name)[0]
    c = workloads.lattice_case(7, 8, 8, 8, 2.05e-3, radius=(0.9e-3, 1.1e-3), jitter=5e-5, vmax=1.0, wmax=300.0, dt=2e-6,
                               skin=2e-4)
    if name == "every2":
        c["neigh"] = (2, 0, 0)
    return c


def _run(case, calls):
    from gb300dem.api import DemSystem
    g = DemSystem(case)
    g.setup()
    for k in calls:
        g.step(k)
    out = {k: np.array(v) for k, v in g.atoms().items()}, g.stats()
    g.close()
    return out


@pytest.mark.parametrize("small_list", [False, True])
@pytest.mark.parametrize("name", ["plain", "every2", "mixer_rotate", "fibre_press"])
def test_short_calls(name, small_list, monkeypatch):
    case = _case(name)
    for calls in ([1] * 60, [8] * 15, [3, 9] * 10, [1, 40, 2, 30, 7, 40]):
        monkeypatch.setenv("LIGGGHTS_GB300_FUSED_STEPS", "0")
        ref, sr = _run(case, calls)
        monkeypatch.setenv("LIGGGHTS_GB300_FUSED_STEPS", "1")
        if small_list:
            monkeypatch.setenv("LIGGGHTS_GB300_PAIRS_PER_ATOM", "0")
        got, s = _run(case, calls)
        monkeypatch.delenv("LIGGGHTS_GB300_PAIRS_PER_ATOM", raising=False)
        for k in ref:
            assert np.array_equal(got[k], ref[k]), (k, calls)
        for k in ("ntimestep", "nrebuilds", "npairs", "natoms"):
            assert s[k] == sr[k], (k, calls)
