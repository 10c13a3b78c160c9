"""The adjoint engine's lists at the edges of their kernels' tiles.

Nine lanes of a warp search one atom's stencil rows (three atoms per warp) and
keep up to eight entries a row for the fill pass; a block of the law kernels
queues up to eight runs of 128 entries.  A wide skin overflows the kept rows
and lengthens the list without changing the contacts, so the trajectory and
the gradient stay what they are with the narrow one, and the trajectory is the
system's own: both to rounding over a few steps (30 steps of some ten
operations of relative error 1e-16 on sums of order one, amplified by the
contacts' stiffness: 1e-9 is kept)."""
import numpy as np
import pytest

from golden_io import max_rel, sort_by_tag

pytestmark = pytest.mark.gpu

RTOL = 1e-9
STEPS, SEG = 30, 10


def _case(n, skin):
    from gb300dem import workloads
    m = max(8, int(np.ceil(n ** (1 / 3))))
    c = workloads.lattice_case(seed=3, nx=m, ny=m, nz=max(3, -(-n // (m * m))), spacing=1.97e-3, radius=(0.99e-3, 1.0e-3),
                               z0=0.985e-3, jitter=2e-6, vmax=5e-3, wmax=50.0, E=(1e7,), nu=(0.3,), rest=((0.6,),),
                               frict=((0.5,),), dt=1e-6, skin=skin)
    c["atoms"] = {k: v[:n] for k, v in c["atoms"].items()}
    c["planes"] = [(2, 0.0, 1, 0)]
    c["neigh"] = (SEG, 0, 0)
    return c


def _run(case):
    from gb300dem.adjoint import DemAdjoint, make_loss
    e = DemAdjoint(case)
    _, g = e.gradient(1e7, 0.6, 0.5, nsteps=STEPS, segment=SEG, loss=make_loss(w_ke=1.0))
    s = {k: np.array(v) for k, v in e.final_state().items()}
    e.close()
    return s, {k: np.array(v) for k, v in g.items()}


@pytest.mark.parametrize("n", [1, 2, 3, 4, 31, 128, 385, 4097, 20001])
def test_wide_skin_changes_nothing(n):
    from gb300dem.api import DemSystem
    narrow, gn = _run(_case(n, 2e-4))
    wide, gw = _run(_case(n, 3.2e-3))
    g = DemSystem(_case(n, 2e-4))
    g.setup()
    g.step(STEPS)
    a = sort_by_tag(g.atoms())
    if n == 20001:  # several runs a block
        assert g.stats()["npairs"] > 3 * n / 2
    g.close()
    for k in ("x", "v", "omega"):
        assert max_rel(wide[k], narrow[k]) < RTOL, k
        assert max_rel(wide[k], a[k]) < RTOL, k
    for k in gn:
        assert max_rel(gw[k], gn[k]) < RTOL, k
