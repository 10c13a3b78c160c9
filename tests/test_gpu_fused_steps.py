"""The fused step kernel against the separate kernels and the host loop.

k_steps runs the tiles of the separate kernels between grid barriers, so a
run gives the same bits either way: for every contact path (touching pairs
only, contact distance factor above 1, bonds), with and without rolling
friction, with planes, static, translating and rotating meshes, across
neighbour rebuilds (by displacement, by a moving mesh, every few steps
without a check), whatever the split into calls, after a list that outgrew
its capacity, after an insertion, and for systems of one warp up to several
tiles per warp.  A grid barrier that gives up returns DEM_ERR_TIMEOUT, and the
handle works again after the next upload.
"""
import numpy as np
import pytest

from golden_io import load_golden

pytestmark = pytest.mark.gpu


def _lattice(n, **kw):
    from gb300dem import workloads
    m = max(4, int(round(n ** (1 / 3))))
    base = dict(radius=(0.9e-3, 1.1e-3), jitter=5e-5, vmax=1.0, wmax=300.0, dt=2e-6, skin=2e-4)
    base.update(kw)
    c = workloads.lattice_case(5, m, m, -(-n // (m * m)), 2.05e-3, **base)
    c["atoms"] = {k: v[:n] for k, v in c["atoms"].items()}
    return c


def _cases():
    roll = dict(rolling_model=1, rollfrict=((0.3,),))
    hooke = dict(normal_model=1, charVel=2.0, ntypes=2, E=(5e6, 2e7), nu=(0.45, 0.3), rest=((0.9, 0.7), (0.7, 0.5)),
                 frict=((0.5, 0.4), (0.4, 0.3)))
    return {
        "one_atom": lambda: _lattice(1), "one_warp": lambda: _lattice(32), "two_warps": lambda: _lattice(33),
        "touch": lambda: _lattice(700), "rolling": lambda: _lattice(1500, **roll), "hooke": lambda: _lattice(900, **hooke),
        "band": lambda: dict(_lattice(800), cdf=1.1), "many_tiles": lambda: _lattice(90000, **roll),
        "every3": lambda: dict(_lattice(600), neigh=(3, 6, 0)),
        "hopper": lambda: load_golden("hopper_mesh_cdt")[0], "mixer": lambda: load_golden("mixer_rotate")[0],
        "press": lambda: load_golden("fibre_press")[0], "silo": lambda: load_golden("silo_cyl")[0],
    }


def _run(case, calls, monkeypatch, env, insert=None):
    from gb300dem.api import DemSystem
    for k, v in env.items():
        monkeypatch.setenv(k, v)
    g = DemSystem(case)
    g.setup()
    for n, k in enumerate(calls):
        if insert is not None and n == 1:
            g.insert(insert)
        g.step(k)
    out = (g.atoms(), g.pairs(), [g.mesh_contacts(k) for k in range(len(case.get("meshes", [])))], g.stats())
    out = ({k: np.array(v) for k, v in out[0].items()},) + out[1:]
    g.close()
    for k in env:
        monkeypatch.delenv(k)
    return out


def _same(a, b):
    for x, y in zip((a[0], a[1], *a[2]), (b[0], b[1], *b[2])):
        for k in x:
            assert np.array_equal(x[k], y[k]), k
    for k in ("ntimestep", "nrebuilds", "npairs", "natoms", "nlost"):
        assert a[3][k] == b[3][k], k


FUSED, APART, HOST = ({"LIGGGHTS_GB300_FUSED_STEPS": "1"}, {"LIGGGHTS_GB300_FUSED_STEPS": "0"},
                      {"LIGGGHTS_GB300_NO_GRAPH": "1"})


@pytest.mark.parametrize("name", list(_cases()))
def test_fused_steps_give_the_separate_kernels_bits(name, monkeypatch):
    case = _cases()[name]()
    calls = [1, 2, 37, 160]
    ref = _run(case, calls, monkeypatch, APART)
    _same(_run(case, calls, monkeypatch, FUSED), ref)
    _same(_run(case, calls, monkeypatch, HOST), ref)
    assert ref[3]["nrebuilds"] > 1 or name in ("one_atom", "silo", "hopper", "press")


@pytest.mark.parametrize("name", ["touch", "press"])
def test_list_overflow_resumes(name, monkeypatch):
    case = _cases()[name]()
    ref = _run(case, [90], monkeypatch, APART)
    for env in (FUSED, APART):
        _same(_run(case, [90], monkeypatch, dict(env, LIGGGHTS_GB300_PAIRS_PER_ATOM="0")), ref)


def test_insertion(monkeypatch):
    case = _lattice(400)
    case["capacity"] = (420, 0.9e-3, 1.1e-3)
    n = 12
    top = float(case["boxhi"][2]) - 1.5e-3
    x = np.array([[0.002 + 0.0011 * k, 0.004, top] for k in range(n)])
    new = dict(tag=np.arange(401, 401 + n, dtype=np.int32), type=np.ones(n, np.int32), x=x, v=np.zeros((n, 3)),
               omega=np.zeros((n, 3)), radius=np.full(n, 1e-3), rmass=np.full(n, 1e-5))
    ref = _run(case, [20, 1, 40], monkeypatch, APART, new)
    _same(_run(case, [20, 1, 40], monkeypatch, FUSED, new), ref)
    _same(_run(case, [20, 1, 40], monkeypatch, HOST, new), ref)


def test_barrier_that_gives_up(monkeypatch):
    from gb300dem.api import DemError, DemSystem
    case = _lattice(2000)
    monkeypatch.setenv("LIGGGHTS_GB300_FUSED_STEPS", "1")
    monkeypatch.setenv("LIGGGHTS_GB300_BARRIER_POLLS", "1")
    g = DemSystem(case)
    g.setup()
    with pytest.raises(DemError, match="DEM_ERR_TIMEOUT"):
        g.step(50)
    monkeypatch.delenv("LIGGGHTS_GB300_BARRIER_POLLS")
    g.upload(case["atoms"])
    g.setup()
    g.step(50)
    h = DemSystem(case)
    h.setup()
    h.step(50)
    a, b = g.atoms(), h.atoms()
    for k in a:
        assert np.array_equal(a[k], b[k]), k
