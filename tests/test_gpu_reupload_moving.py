"""Uploads into a handle with moving-mesh walls, and with bonds: the kept
arrays (mesh slots, bond histories) and the kept graph give a new handle's bits.
The meshes have movers that leave them in place, so that the second run
starts where the first did."""
import numpy as np
import pytest

from golden_io import load_golden
from test_gpu_reupload import _fresh, _steps

pytestmark = pytest.mark.gpu


def _case(name):
    case = load_golden(name)[0]
    for m in case["meshes"]:
        if m.get("rotate") is not None:  # the quaternion of a step is the identity
            m["rotate"] = dict(m["rotate"], origin=(0.0, 0.0, 0.0), period=1e300)
        if m.get("vel") is not None:
            m["vel"] = (0.0, 0.0, 0.0)
    return case


@pytest.mark.parametrize("fused", ["0", "1"])
@pytest.mark.parametrize("small_list", [False, True])
@pytest.mark.parametrize("name", ["mixer_rotate", "fibre_press", "fibre_bond_stress"])
def test_again(name, small_list, fused, monkeypatch):
    from gb300dem.api import DemSystem
    monkeypatch.setenv("LIGGGHTS_GB300_FUSED_STEPS", fused)
    if small_list:
        monkeypatch.setenv("LIGGGHTS_GB300_PAIRS_PER_ATOM", "1")
    case = _case(name)
    first = dict(case["atoms"])  # another state to run before
    first["v"] = np.ascontiguousarray(first["v"][::-1]) * 3.0
    ref, rcount = _fresh(case)
    g = DemSystem(case)
    g.upload(first)
    g.setup()
    g.step(150)
    for _ in range(2):
        g.upload(case["atoms"])
        got, count = _steps(g)
        assert count == rcount
        for k in ref:
            assert np.array_equal(got[k], ref[k]), k
    g.close()
