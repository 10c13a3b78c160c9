"""The force gather of the per-atom kernel against that of the fused kernel.

k_particle adds one component of one atom per lane, from a list of up to 16
contacts kept in shared memory and beyond it one lane per atom; k_steps gathers
with one lane per atom.  Both add in the reference's order, so a sphere with
any number of contacts moves by the same bits: a large one in a shell of k
small ones, k around the list's length and around the 32 entries of the masks,
as first and as last atom (own entries, partner entries)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _case(k, first):
    from gb300dem import workloads
    c = workloads.lattice_case(4, 12, 12, 12, 2.05e-3, radius=(0.9e-3, 1.1e-3), dt=1e-6, skin=2e-4,
                               periodic=(0, 0, 0))
    R, r = 4e-3, 1e-3
    t = np.arange(k) + 0.5
    phi, z = np.pi * (1 + 5 ** 0.5) * t, 1 - 2 * t / k
    s = np.sqrt(1 - z * z)
    u = np.stack([s * np.cos(phi), s * np.sin(phi), z], 1)
    centre = np.array([0.0123, 0.0123, 0.0123])
    x = centre + (R + r - 2e-5 * (1 + t[:, None] / k)) * u
    x = np.concatenate([[centre], x] if first else [x, [centre]])
    rad = np.concatenate([[R], np.full(k, r)] if first else [np.full(k, r), [R]])
    rng = np.random.default_rng(k)
    n = k + 1
    c["atoms"] = dict(tag=np.arange(1, n + 1, dtype=np.int32), type=np.ones(n, np.int32), x=x,
                      v=rng.normal(0, 0.05, (n, 3)), omega=rng.normal(0, 30.0, (n, 3)), radius=rad,
                      rmass=workloads.sphere_mass(rad, c["material"]["density"]))
    return c


@pytest.mark.parametrize("first", [True, False])
@pytest.mark.parametrize("k", [1, 4, 5, 15, 16, 17, 32, 33, 50])
def test_any_number_of_contacts(k, first, monkeypatch):
    from gb300dem.api import DemSystem
    out = []
    for fused in "01":
        monkeypatch.setenv("LIGGGHTS_GB300_FUSED_STEPS", fused)
        g = DemSystem(_case(k, first))
        g.setup()
        g.step(1)
        assert g.diagnostics()["ncontacts"] >= k
        g.step(29)
        out.append({a: np.array(v) for a, v in g.atoms().items()})
        g.close()
    for a in out[0]:
        assert np.array_equal(out[0][a], out[1][a]), a
