"""Handles stepped from several threads at the same time give the bits that they
give alone, whichever kernels run them; so does a long call of the fused kernel
that returns to the host in between."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fused", [(True, True), (True, False)])
def test_two_threads(fused):
    """Two handles (the second also of a size that runs in the separate kernels) stepped at the same time."""
    from gb300dem import workloads
    from gb300dem.api import DemSystem
    big = dict(radius=(0.9e-3, 1.1e-3), jitter=5e-5, vmax=1.0, wmax=300.0, dt=2e-6, skin=2e-4)
    cases = [workloads.lattice_case(5, 20, 20, 20, 2.05e-3, **big),
             workloads.lattice_case(6, 20, 20, 25, 2.05e-3, **big) if fused[1] else
             workloads.lattice_case(6, 50, 50, 50, 2.05e-3, **big)]

    def steps(g):
        g.setup()
        for k in (1, 30, 2, 8, 40, 1):
            g.step(k)
        return {k: np.array(v) for k, v in g.atoms().items()}

    alone = []
    for c in cases:
        g = DemSystem(c)
        alone.append(steps(g))
        g.close()
    gs, got, bad = [DemSystem(c) for c in cases], [None, None], []

    def work(i):
        try:
            for _ in range(3):
                gs[i].upload(cases[i]["atoms"])
                got[i] = steps(gs[i])
        except Exception as e:
            bad.append(e)

    th = [threading.Thread(target=work, args=(i,)) for i in range(2)]
    for t in th:
        t.start()
    for t in th:
        t.join()
    assert not bad
    for i in range(2):
        for k in alone[i]:
            assert np.array_equal(got[i][k], alone[i][k]), (i, k)


@pytest.mark.parametrize("turn", ["1", "3", "8", "36", "37"])
@pytest.mark.parametrize("name", ["plain", "every2", "mixer_rotate", "fibre_press"])
def test_turns(name, turn, monkeypatch):
    """Calls of more steps than a turn, fewer and as many; rebuilds on a turn's last step."""
    from test_gpu_short_calls import _case, _run
    case, calls = _case(name), [37, 9, 1, 73, 8, 40]
    monkeypatch.setenv("LIGGGHTS_GB300_FUSED_STEPS", "0")
    ref, sr = _run(case, calls)
    monkeypatch.setenv("LIGGGHTS_GB300_FUSED_STEPS", "1")
    monkeypatch.setenv("LIGGGHTS_GB300_TURN", turn)
    got, s = _run(case, calls)
    for k in ref:
        assert np.array_equal(got[k], ref[k]), k
    for k in ("ntimestep", "nrebuilds", "npairs", "natoms"):
        assert s[k] == sr[k], k
