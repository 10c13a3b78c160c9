"""Wall history of a restart against the oracle."""
import numpy as np
import pytest

from golden_io import FORCE_RTOL, max_rel, sort_by_tag
from test_gpu_wall_params import _case

pytestmark = pytest.mark.gpu


def test_wall_history_with_a_normal_part():
    """A restart's wall history is taken as it is in the setup pass, whatever
    its direction; the first step's update makes it tangential."""
    from gb300dem.api import DemSystem
    from oracle.binding import Oracle
    case = _case("plane")
    n = len(case["atoms"]["tag"])
    case["atoms"] = dict(case["atoms"], x=case["atoms"]["x"] * [1, 1, 0] + [0, 0, 0.89e-3])
    hist = np.random.default_rng(1).uniform(-1e-7, 1e-7, (n, 3))
    g, o = DemSystem(case), Oracle(case)
    for s in (g, o):
        s.set_restart([], [], np.zeros((0, 3)), [hist])
        s.setup()
    a, b = sort_by_tag(g.atoms()), sort_by_tag(o.atoms())
    assert max_rel(a["f"], b["f"]) < FORCE_RTOL and max_rel(a["torque"], b["torque"]) < FORCE_RTOL
    for s in (g, o):
        s.run(3)
    a, b = sort_by_tag(g.atoms()), sort_by_tag(o.atoms())
    assert max_rel(a["f"], b["f"]) < FORCE_RTOL and max_rel(a["torque"], b["torque"]) < FORCE_RTOL

