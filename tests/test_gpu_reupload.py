"""Uploads into a handle that has run before: its arrays are kept where they
fit and the step graph where nothing that it holds has changed, and every run
gives the bits of a new handle's, whatever ran before it (as many atoms, fewer,
more, other radii and so another cutoff, a list that outgrew its capacity)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _case(n, rmax=1.1e-3, seed=5):
    from gb300dem import workloads
    m = 12
    c = workloads.lattice_case(seed, m, m, 14, 2.25e-3, radius=(0.9e-3, rmax), jitter=5e-5, vmax=1.0, wmax=300.0,
                               dt=2e-6, skin=2e-4)
    c["atoms"] = {k: v[:n] for k, v in c["atoms"].items()}
    return c


def _steps(g):
    g.setup()
    g.step(3)
    g.step(60)
    s = g.stats()
    return {k: np.array(v) for k, v in g.atoms().items()}, (s["npairs"], s["nrebuilds"], s["ntimestep"])


def _fresh(case):
    from gb300dem.api import DemSystem
    g = DemSystem(case)
    out = _steps(g)
    g.close()
    return out


@pytest.mark.parametrize("fused", ["0", "1"])
@pytest.mark.parametrize("small_list", [False, True])
def test_any_sequence_of_uploads(fused, small_list, monkeypatch):
    from gb300dem.api import DemSystem
    monkeypatch.setenv("LIGGGHTS_GB300_FUSED_STEPS", fused)
    if small_list:
        monkeypatch.setenv("LIGGGHTS_GB300_PAIRS_PER_ATOM", "1")
    cases = [_case(*a) for a in ((700,), (700,), (700, 1.1e-3, 6), (700, 1.0e-3), (33,), (2000,), (1200,), (700,))]
    g = DemSystem(cases[0])
    for c in cases:
        g.upload(c["atoms"])
        got, count = _steps(g)
        ref, rcount = _fresh(c)
        assert count == rcount
        for k in ref:
            assert np.array_equal(got[k], ref[k]), k
    g.close()


@pytest.mark.parametrize("name", ["hopper_mesh_cdt", "mixer_rotate", "fibre_press"])
def test_meshes_and_bonds_again(name, monkeypatch):
    from gb300dem.api import DemSystem
    from golden_io import load_golden
    case = load_golden(name)[0]
    static = not any(m.get("move") for m in case["meshes"]) and name == "hopper_mesh_cdt"
    ref, rcount = _fresh(case)
    g = DemSystem(case)
    _steps(g)
    if static:  # a moved mesh stays where it is
        g.upload(case["atoms"])
        got, count = _steps(g)
        assert count == rcount
        for k in ref:
            assert np.array_equal(got[k], ref[k]), k
    else:
        g.upload(case["atoms"])
        _steps(g)
    g.close()
