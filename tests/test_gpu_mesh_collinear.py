"""Mesh triangles whose nodes lie on one line, against the oracle.  Their
barycentric coordinates are infinities and NaN; a NaN lies in no region of the
closest feature, whatever its sign, so the region and the contact follow from
the others."""
import numpy as np
import pytest

from golden_io import FORCE_RTOL, max_rel, sort_by_tag

pytestmark = pytest.mark.gpu


def _case(inner):
    """One sphere per triangle; inner: the node that lies between the others."""
    from gb300dem import workloads
    m = 14
    c = workloads.lattice_case(3, m, m, 1, 5e-3, radius=(0.9e-3, 1.0e-3), z0=4e-3, vmax=0.1, wmax=50.0,
                               periodic=(0, 0, 0), plane_z=None, zhi=9e-3)
    rng = np.random.default_rng([7, inner])
    tri = []
    for x in c["atoms"]["x"]:
        d = rng.integers(-4, 5, 3).astype(float)
        while np.count_nonzero(d) < 2:
            d = rng.integers(-4, 5, 3).astype(float)
        d /= np.linalg.norm(d)
        off = np.cross(d, rng.normal(size=3))
        mid = x + off * 0.6e-3 / np.linalg.norm(off) + d * rng.uniform(-1.3e-3, 1.3e-3)
        ends = (mid - 0.7e-3 * d, mid, mid + rng.uniform(0.3e-3, 0.9e-3) * d)
        order = {0: (1, 0, 2), 1: (0, 1, 2), 2: (0, 2, 1)}[inner]
        tri.append([ends[k] for k in order])
    c["meshes"] = [dict(nodes=np.asarray(tri), wall_type=1, rolling=0)]
    return c


@pytest.mark.parametrize("flags", [False, True])
@pytest.mark.parametrize("inner", [0, 1, 2])
def test_collinear_triangles_match_oracle(inner, flags):
    from gb300dem.api import DemSystem
    from oracle.binding import Oracle
    case = _case(inner)
    if flags:  # every edge and corner active (of a line's own corners none would be)
        one = np.ones((len(case["meshes"][0]["nodes"]), 3), np.uint8)
        case["meshes"][0].update(edge_active=one, corner_active=one.copy())
    g, o = DemSystem(case), Oracle(case)
    g.setup()
    o.setup()
    for steps in (0, 1, 9):
        if steps:
            g.step(steps)
            o.run(steps)
        a, b = sort_by_tag(g.atoms()), sort_by_tag(o.atoms())
        p, q = g.mesh_contacts(0), o.mesh_contacts(0)
        assert (sorted(zip(p["tag"].tolist(), p["tri"].tolist())) ==
                sorted(zip(q["tag"].tolist(), q["tri"].tolist())))
        assert max_rel(a["f"], b["f"]) < FORCE_RTOL
    assert len(q["tag"]) > 0
