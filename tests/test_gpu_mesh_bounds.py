"""The wall kernel's FP32 triangle bounds and warp tiles against the oracle.

The bounds may only leave out triangles that the exact closest-feature
resolution would not touch, so the contact sets and slots equal the oracle's
on meshes where they are hardest: slivers (50:1), triangles too thin for the
edge bounds (1e6:1), large triangles far from the origin (FP32 rounding of
the coordinates), and squares far smaller than the contact's own radius.  The
atoms near the floor number 31, 32, 33 and 97 (tiles of 32).  A rotating mesh
with an odd number of triangles keeps the oracle's node positions bit for bit.
"""
import numpy as np
import pytest

from golden_io import FORCE_RTOL, TRAJ_RTOL, max_rel, sort_by_tag

pytestmark = pytest.mark.gpu


def _floor(x0, x1, nx, y0, y1, ny):
    gx, gy = np.linspace(x0, x1, nx + 1), np.linspace(y0, y1, ny + 1)
    tri = []
    for i in range(nx):
        for j in range(ny):
            a, b = (gx[i], gy[j], 0.0), (gx[i + 1], gy[j], 0.0)
            c, d = (gx[i + 1], gy[j + 1], 0.0), (gx[i], gy[j + 1], 0.0)
            tri += [(a, b, c), (a, c, d)]
    return np.asarray(tri)


def _case(mesh, natoms, shift):
    from gb300dem import workloads
    n = int(np.ceil(natoms ** 0.5))
    c = workloads.lattice_case(7, n, n, 1, 2.1e-3, radius=(0.9e-3, 1.05e-3), z0=0.93e-3, jitter=5e-5, vmax=0.2,
                               wmax=100.0, periodic=(0, 0, 0), plane_z=None)
    c["atoms"] = {k: v[:natoms] for k, v in c["atoms"].items()}
    L = n * 2.1e-3
    tri = {"sliver": lambda: _floor(0.0, L, max(1, n // 4), 0.0, L, 50 * max(1, n // 4)),
           "thin": lambda: np.concatenate([_floor(0.0, L, 2, 0.0, L / 2, 2),
                                           _floor(0.0, L, 1, L / 2, L / 2 + 1e-6 * L, 1),
                                           _floor(0.0, L, 2, L / 2 + 1e-6 * L, L, 2)]),
           "large": lambda: _floor(-0.3, 0.4, 2, -0.2, 0.5, 2),
           "fine": lambda: _floor(0.0, L, int(L / 0.4e-3), 0.0, L, int(L / 0.4e-3))}[mesh]()
    sh = np.asarray(shift)
    c["boxlo"], c["boxhi"] = tuple(sh - 3e-3), tuple(sh + np.array([L, L, 0.02]) + 3e-3)
    c["atoms"]["x"] = c["atoms"]["x"] + sh
    c["meshes"] = [dict(nodes=tri + sh, wall_type=1, rolling=0)]
    return c


@pytest.mark.parametrize("natoms", [1, 31, 32, 33, 97])
@pytest.mark.parametrize("mesh,shift", [("sliver", (0.0, 0.0, 0.0)), ("thin", (0.0, 0.0, 0.0)),
                                        ("large", (0.7, -0.9, 0.3)), ("fine", (0.05, 0.02, 0.1))])
def test_floor_contacts_match_oracle(mesh, shift, natoms):
    from gb300dem.api import DemSystem
    from oracle.binding import Oracle
    case = _case(mesh, natoms, shift)
    g, o = DemSystem(case), Oracle(case)
    g.setup()
    o.setup()
    for steps in (1, 9, 40):
        g.step(steps)
        o.run(steps)
        a, b = sort_by_tag(g.atoms()), sort_by_tag(o.atoms())
        assert max_rel(a["x"], b["x"]) < TRAJ_RTOL
        assert max_rel(a["f"], b["f"]) < (FORCE_RTOL if steps == 1 else 1e-9)
        m, p = g.mesh_contacts(0), o.mesh_contacts(0)
        km = sorted(zip(m["tag"].tolist(), m["tri"].tolist(), m["slot"].tolist()))
        kp = sorted(zip(p["tag"].tolist(), p["tri"].tolist(), p["slot"].tolist()))
        assert km == kp and (len(km) > 0 or natoms == 1)  # (the single atom floats above the floor)


def test_rotating_mesh_of_odd_size_matches_oracle():
    from gb300dem import workloads
    from gb300dem.api import DemSystem
    from oracle.binding import Oracle
    c = workloads.mixer_case(3, 8, 8, 2, 2.2e-3, (0.95e-3, 1.0e-3), blade_half_len=6e-3, blade_height=5e-3,
                             period=0.01, z0=1.0e-3, jitter=2e-5, vmax=0.5, wmax=50.0)
    m = c["meshes"][0]
    fan = [m["nodes"][0]]
    for k in range(32):  # a strip of small triangles in the paddle's plane beside it
        a = np.array([m["nodes"][0][0][0], m["nodes"][0][0][1], 1e-4 * (k + 1)])
        fan.append(np.array([a, a + [1e-4, 0, 0], a + [0, 0, 1e-4]]) - [2e-4 * (k + 1), 0, 0])
    m["nodes"] = np.asarray(fan)
    g, o = DemSystem(c), Oracle(c)
    g.setup()
    o.setup()
    g.step(60)
    o.run(60)
    assert np.array_equal(g.mesh_nodes(0), o.mesh_nodes(0))
    assert g.nrebuilds == o.nrebuilds
