"""As many primitive walls as a handle takes, against the oracle."""
import numpy as np
import pytest

from golden_io import FORCE_RTOL, max_rel, sort_by_tag
from test_gpu_wall_params import _case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("last", [0, 3, 7])
def test_eight_planes(last):
    """The wall that an atom is near may be any of the eight."""
    from gb300dem.api import DemSystem
    from oracle.binding import Oracle
    case = _case("none")
    far = [(2, -0.5 - 0.01 * k, 1, 0) for k in range(7)]
    case["planes"] = far[:last] + [(2, 0.0, 1, 0)] + far[last:]
    g, o = DemSystem(case), Oracle(case)
    g.setup()
    o.setup()
    for steps in (1, 9):
        g.step(steps)
        o.run(steps)
        a, b = sort_by_tag(g.atoms()), sort_by_tag(o.atoms())
        assert max_rel(a["f"], b["f"]) < FORCE_RTOL and max_rel(a["torque"], b["torque"]) < FORCE_RTOL
    assert np.count_nonzero(np.abs(b["f"][:, 2]) > 1e-3) > 5
