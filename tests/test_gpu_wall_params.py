"""dem_set_pair_params on a running handle: the wall contacts of the next step
take the new tables (pairs keep their constants until the next build), as the
oracle's do, whose systems here have no touching pairs."""
import numpy as np
import pytest

from golden_io import FORCE_RTOL, TRAJ_RTOL, max_rel, sort_by_tag

pytestmark = pytest.mark.gpu

KEYS = ("Yeff", "Geff", "betaeff", "coeffFrict", "coeffRollFrict", "coeffRestLog")


def _floor(L):
    a, b, c, d = (-L, -L, 0.0), (2 * L, -L, 0.0), (2 * L, 2 * L, 0.0), (-L, 2 * L, 0.0)
    return np.asarray([(a, b, c), (a, c, d)])


def _case(wall, **law):
    from gb300dem import workloads
    L = 6 * 3e-3
    c = workloads.lattice_case(7, 6, 6, 1, 3e-3, radius=(0.9e-3, 1.05e-3), z0=0.93e-3, jitter=5e-5, vmax=0.2,
                               wmax=100.0, periodic=(0, 0, 0), plane_z=0.0 if wall == "plane" else None, **law)
    c["boxlo"], c["boxhi"] = (-3e-3,) * 3, (L + 3e-3, L + 3e-3, 0.02)
    if wall == "mesh":
        c["meshes"] = [dict(nodes=_floor(L), wall_type=1, rolling=0)]
    elif wall == "cylinder":
        c["cylinders"] = [(1, 1.0, 1.0, L / 2, 1, 0)]  # axis y at z = 1, x = L/2: nearly the floor
    return c


@pytest.mark.parametrize("fused", ["0", "1"])
@pytest.mark.parametrize("law", ["hertz", "hooke"])
@pytest.mark.parametrize("wall", ["plane", "mesh", "cylinder"])
def test_walls_take_new_tables_at_once(wall, law, fused, monkeypatch):
    from gb300dem import api, workloads
    from oracle import binding
    monkeypatch.setenv("LIGGGHTS_GB300_FUSED_STEPS", fused)
    kw = dict(normal_model=1, charVel=2.0) if law == "hooke" else {}
    case = _case(wall, rest=((0.9,),), **kw)
    new = workloads.derive_tables((3e6,), (0.3,), ((0.4,),), ((0.3,),))
    vel = 1.3 if law == "hooke" else 0.0
    g, o = api.DemSystem(case), binding.Oracle(case)
    g.setup()
    o.setup()
    for steps in (5, 1, 20):
        g.step(steps)
        o.run(steps)
        a, b = sort_by_tag(g.atoms()), sort_by_tag(o.atoms())
        assert max_rel(a["f"], b["f"]) < FORCE_RTOL * steps
        assert max_rel(a["x"], b["x"]) < TRAJ_RTOL
        assert g.nrebuilds == o.nrebuilds  # no build between the call and the step
        if steps == 5:
            tabs = [np.ascontiguousarray(new[k], dtype=np.float64) for k in KEYS]
            g._check(api.load().dem_set_pair_params(g.h, 1, *[api._p(t) for t in tabs], vel))
            binding.lib().orc_set_pair_params(o.h, 1, *[binding._p(t) for t in tabs], vel)
    assert np.count_nonzero(np.abs(b["f"][:, 2]) > 1e-3) > 5  # touching the wall
