"""Where the fused kernel's cooperative launch is refused (at the residency
query, in the graph, at a short call, behind a rebuild, at the graph's launch),
the separate kernels take over, with their bits; other handles are not
concerned."""
import numpy as np
import pytest

from test_gpu_short_calls import _case, _run

pytestmark = pytest.mark.gpu

GRID, IN_GRAPH, DIRECT, RESUME, GRAPH_LAUNCH = 1, 2, 4, 8, 16


@pytest.mark.parametrize("small_list", [False, True])
@pytest.mark.parametrize("refuse", [GRID, IN_GRAPH, DIRECT, RESUME, GRAPH_LAUNCH, DIRECT | IN_GRAPH, 31])
@pytest.mark.parametrize("name", ["every2", "mixer_rotate", "fibre_press"])
def test_refused(name, refuse, small_list, monkeypatch):
    case = _case(name)
    for calls in ([1, 8, 3, 37, 2, 60], [40, 1, 1], [8] * 12):
        monkeypatch.setenv("LIGGGHTS_GB300_FUSED_STEPS", "0")
        ref, sr = _run(case, calls)
        monkeypatch.setenv("LIGGGHTS_GB300_FUSED_STEPS", "1")
        monkeypatch.setenv("LIGGGHTS_GB300_COOP_REFUSE", str(refuse))
        if small_list:
            monkeypatch.setenv("LIGGGHTS_GB300_PAIRS_PER_ATOM", "0")
        got, s = _run(case, calls)
        monkeypatch.delenv("LIGGGHTS_GB300_PAIRS_PER_ATOM", raising=False)
        monkeypatch.delenv("LIGGGHTS_GB300_COOP_REFUSE")
        for k in ref:
            assert np.array_equal(got[k], ref[k]), (k, calls)
        for k in ("ntimestep", "nrebuilds", "npairs", "natoms"):
            assert s[k] == sr[k], (k, calls)


def test_refusal_belongs_to_the_handle(monkeypatch):
    from gb300dem.api import DemSystem
    case = _case("plain")
    monkeypatch.setenv("LIGGGHTS_GB300_COOP_REFUSE", "31")
    a = DemSystem(case)
    a.setup()
    a.step(20)
    monkeypatch.delenv("LIGGGHTS_GB300_COOP_REFUSE")
    b = DemSystem(case)
    b.setup()
    n = b.kernel_times()["kernel_launches"], b.nrebuilds
    b.step(20)
    assert b.kernel_times()["kernel_launches"] - n[0] <= 2 + 50 * (b.nrebuilds - n[1])
    x, y = a.atoms(), b.atoms()
    for k in x:
        assert np.array_equal(x[k], y[k]), k
