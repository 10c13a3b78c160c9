"""Positions that only the upper end of the FP32 range holds: an atom that
drifts there is finite and lost at that step's build, as any that left the box;
one beyond FP32 is reported as non-finite."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fused", ["0", "1"])
@pytest.mark.parametrize("x,ok", [(1e30, True), (1.6e38, True), (-1.75e38, True), (3.4028e38, True), (-3.41e38, False),
                                  (1e200, False)])
def test_far_drift(x, ok, fused, monkeypatch):
    from gb300dem import workloads
    from gb300dem.api import DemError, DemSystem
    monkeypatch.setenv("LIGGGHTS_GB300_FUSED_STEPS", fused)
    c = workloads.lattice_case(7, 4, 4, 4, 2.2e-3, periodic=(0, 0, 0))
    c["atoms"]["v"][17, 0] = x / c["dt"]
    g = DemSystem(c)
    g.setup()
    if not ok:
        with pytest.raises(DemError, match="DEM_ERR_NAN"):
            g.step(3)
        return
    g.step(3)
    assert g.natoms() == 63 and g.stats()["nlost"] == 1
    assert 18 not in g.atoms()["tag"] and np.isfinite(g.atoms()["x"]).all()
