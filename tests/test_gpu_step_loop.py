"""The step loop of the separate kernels, unrolled in its graph.

A step that decides to rebuild holds the rest of the loop's iteration until the
next one's rebuild, and the last step holds it to the end.  Whatever falls
together (a rebuild on every step, on the first or last of an iteration or of
a call, calls shorter and longer than an iteration), a run gives the bits of
the host's loop and as many steps and rebuilds."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _run(case, calls):
    from gb300dem.api import DemSystem
    g = DemSystem(case)
    g.setup()
    for k in calls:
        g.step(k)
    out = {k: np.array(v) for k, v in g.atoms().items()}, g.stats()
    g.close()
    return out


@pytest.mark.parametrize("moving", [False, True])
@pytest.mark.parametrize("every", [1, 2, 3, 4, 5, 9])
def test_holds_at_every_place(every, moving, monkeypatch):
    from gb300dem import workloads
    from golden_io import load_golden
    if moving:
        case = dict(load_golden("mixer_rotate")[0], neigh=(every, 0, 0))
    else:
        case = workloads.lattice_case(7, 7, 7, 7, 2.05e-3, radius=(0.9e-3, 1.1e-3), jitter=5e-5, vmax=1.0, wmax=300.0,
                                      dt=2e-6, skin=2e-4)
        case["neigh"] = (every, 0, 0)
    calls = [1, 2, 3, 4, 5, 6, 8, 9, 13]
    monkeypatch.setenv("LIGGGHTS_GB300_FUSED_STEPS", "0")
    a, sa = _run(case, calls)
    monkeypatch.setenv("LIGGGHTS_GB300_NO_GRAPH", "1")
    b, sb = _run(case, calls)
    for k in a:
        assert np.array_equal(a[k], b[k]), k
    for k in ("ntimestep", "nrebuilds", "npairs", "natoms"):
        assert sa[k] == sb[k], k
    assert sa["ntimestep"] == sum(calls) and sa["nrebuilds"] >= 1 + sum(calls) // every
