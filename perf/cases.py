"""Timed cases of the sphere-DEM timestep: what a user of this framework has it do.

A case names a kind of granular system, its size and how many timesteps one
call advances.  Every pass goes through the public API: ``DemSystem.step(K)``
and ``DemSystem.atoms(out)`` on a resident system (a run between two outputs,
or one exchange interval of a coupled code), the whole life of a run from host
arrays (upload, setup, steps, download), a batched ensemble, or an adjoint
gradient.  The systems are the ones of this repository's benchmark and tests
(the 10,000-sphere pour, the conical hopper, the settling column, the fibre
bed, the paddle mixer, the settling ensemble, the adjoint's column), at their
sizes and at smaller and larger ones.

Systems with CDT rolling friction start in motion (spins of v/r): from rest,
CDT's torque of fixed size turns the last bits of a zero spin into its
direction, so that no two correct programs agree on it.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "liggghts-inl_gb300", "python"))

from gb300dem import api, ensemble, workloads  # noqa: E402

# kind of system -> smallest and largest number of atoms, most steps of a call
RANGES = {
    "pour": (500, 200_000, 200),     # Hertz, monodisperse, floor plane: the CPU build's demo case once spheres meet
    "column": (1_000, 1_000_000, 50),  # Hertz + CDT rolling, polydisperse, periodic column
    "hooke": (1_000, 400_000, 50),   # Hooke, two materials, periodic column
    "bed": (2_000, 500_000, 50),     # dense: about 2.4 touching contacts per sphere, Hertz + CDT
    "hopper": (5_000, 1_000_000, 50),  # triangle-mesh cone, open outlet, Hertz + CDT on pairs and wall
    "mixer": (2_000, 200_000, 100),  # rotating paddle mesh
    "fibres": (2_000, 200_000, 50),  # bonded fibres, closed box, moving mesh lid
    "ensemble": (20_000, 700_000, 100),  # many independent systems in one handle
    "adjoint": (500, 20_000, 200),   # gradient of the final kinetic energy
}


def listed():
    return [
        # a coupled code (CFD-DEM) that exchanges the particles' state every step: the smallest call
        dict(name="pour_500_step", kind="pour", n=500, steps=1, whole=False),
        # the 10,000-sphere pour, 200 steps between outputs
        dict(name="pour_10k", kind="pour", n=10_000, steps=200, whole=False),
        # a stirred vessel: rotating mesh, an odd number of spheres
        dict(name="mixer_21k", kind="mixer", n=21_437, steps=100, whole=False),
        # two materials, Hooke's law, a periodic column of ragged extents
        dict(name="hooke_99k", kind="hooke", n=99_405, steps=50, whole=False),
        # hopper discharge at laboratory size and at the benchmark's size, its default workload
        dict(name="hopper_100k", kind="hopper", n=100_000, steps=50, whole=False),
        dict(name="hopper_1m", kind="hopper", n=1_000_000, steps=50, whole=False),
        # a dense packing: list and contact work per sphere at its highest
        dict(name="bed_400k", kind="bed", n=400_000, steps=50, whole=False),
        # bonded fibres pressed by a lid
        dict(name="fibres_200k", kind="fibres", n=200_000, steps=50, whole=False),
        # parameter study: independent columns in one handle
        dict(name="ensemble_48", kind="ensemble", n=500_000, steps=100, whole=False),
        # calibration: gradients at test size and at the benchmark's size
        dict(name="adjoint_1k", kind="adjoint", n=1_000, steps=100, whole=True),
        dict(name="adjoint_20k", kind="adjoint", n=20_000, steps=200, whole=True),
        # a whole short run from host arrays: upload, setup, steps, download
        dict(name="column_300k_whole", kind="column", n=300_000, steps=20, whole=True),
    ]


def draw(rng):
    kind = rng.choice(["pour", "pour", "column", "column", "hooke", "bed", "hopper", "hopper", "mixer", "fibres",
                       "ensemble", "adjoint"])
    lo, hi, most = RANGES[kind]
    n = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    steps = int(round(math.exp(rng.uniform(math.log(10 if kind in ("adjoint", "ensemble") else 1), math.log(most)))))
    whole = kind == "adjoint" or (kind != "ensemble" and rng.random() < 0.2)
    return dict(kind=kind, n=n, steps=steps, whole=whole)


# ----------------------------------------------------------------------------
# the systems
# ----------------------------------------------------------------------------

def _first(c, n):
    c["atoms"] = {k: v[:n] for k, v in c["atoms"].items()}
    return c


def _in_motion(c, seed, vmax, wmax):
    rng = np.random.default_rng([seed, 1])
    n = len(c["atoms"]["tag"])
    c["atoms"]["v"] = rng.uniform(-vmax, vmax, (n, 3))
    c["atoms"]["omega"] = rng.uniform(-wmax, wmax, (n, 3))
    return c


# r U[0.8, 1.2] mm, rho 1500, E 1e7, e 0.5, mu 0.6, CDT 0.3, dt 5e-7: the benchmark's material
_HOPPER_MATERIAL = dict(density=1500.0, E=(1e7,), rest=((0.5,),), frict=((0.6,),), rollfrict=((0.3,),),
                        rolling_model=1, dt=5e-7, skin=5e-4)


def _pour(n, seed):
    sp = 2.04e-3
    side = 0.1 if n >= 2000 else 0.03
    m = int(side / sp)
    if n > 40_000:
        m = int(math.ceil((n / 15.0) ** 0.5))
        side = m * sp + 1e-3
    c = workloads.lattice_case(seed, m, m, -(-n // (m * m)), sp, radius=(1e-3, 1e-3), density=2500.0, z0=1.0e-3,
                               jitter=5e-5, vmax=0.3, wmax=50.0, E=(5e6,), nu=(0.45,), rest=((0.9,),), frict=((0.5,),),
                               dt=1e-6, skin=5e-4, pad=(side - m * sp, side - m * sp))
    return _first(c, n)


def _column(n, seed):
    m = max(6, int(round(n ** (1.0 / 3.0))))
    c = workloads.lattice_case(seed, m, m, -(-n // (m * m)), 2.2e-3, radius=(0.8e-3, 1.2e-3), nu=(0.3,), z0=1.2e-3,
                               jitter=5e-5, **_HOPPER_MATERIAL)
    return _in_motion(_first(c, n), seed, 0.5, 800.0)


def _hooke(n, seed):
    m = max(6, int(round((n / 1.2) ** (1.0 / 3.0))))
    c = workloads.lattice_case(seed, m, m + 1, -(-n // (m * (m + 1))), 2.1e-3, radius=(0.9e-3, 1.1e-3), z0=1.0e-3,
                               jitter=5e-5, vmax=0.3, wmax=100.0, ntypes=2, E=(5e6, 2e7), nu=(0.45, 0.3),
                               rest=((0.9, 0.7), (0.7, 0.5)), frict=((0.5, 0.4), (0.4, 0.3)), normal_model=1,
                               charVel=2.0, dt=1e-6, skin=5e-4)
    return _first(c, n)


def _bed(n, seed):
    nz = 25 if n >= 40_000 else 10
    m = max(4, int(math.ceil((n / (4.0 * nz)) ** 0.5)))
    c = workloads.packed_bed_case(seed, m, m, nz, dnn=2.002e-3, radius=(0.99e-3, 1.01e-3), nu=(0.45,),
                                  **_HOPPER_MATERIAL)
    return _in_motion(_first(c, n), seed, 0.2, 1000.0)


def _hopper(n, seed):
    r_out, ta, sp = 0.03, math.tan(math.radians(30.0)), 2.2e-3
    h, held = 0.0, 0.0
    while held < 1.1 * n + 2000 and h < 0.37:  # fill height whose lattice holds n spheres
        held += math.pi * (r_out + h * ta - 1.2e-3) ** 2 / sp ** 2
        h += sp
    c = workloads.hopper_case(seed, r_out, 0.25, 30.0, 256, 64, sp, radius=(0.8e-3, 1.2e-3), nu=(0.45,), jitter=1e-4,
                              fill_height=h + 4e-3, max_atoms=n, clearance=-1e-4, z_below=-0.02, **_HOPPER_MATERIAL)
    return _in_motion(c, seed, 0.5, 1000.0)


def _mixer(n, seed):
    m = max(8, int(round((n / 0.4) ** (1.0 / 3.0))))
    nz = -(-n // (m * m))
    c = workloads.mixer_case(seed, m, m, nz, 2.2e-3, (0.95e-3, 1.1e-3), blade_half_len=0.35 * m * 2.2e-3,
                             blade_height=0.8 * nz * 2.2e-3, period=0.5, z0=1.0e-3, jitter=2e-5, vmax=0.5, wmax=50.0)
    return _first(c, n)


def _fibres(n, seed):
    r = 0.5e-3
    side = 45e-3 if n > 40_000 else 23e-3
    bond = workloads.elastoplastic_bond_params(
        2, [1], E=1e9, yield_strain=0.01, hardening=0.1, radius=r, lam=0.5, nu=0.3, tsCreate=1.0, damp_fn=0.05,
        damp_ft=0.05, damp_tn=0.05, damp_tt=0.05, maxDistance=2 * r * 1.0035, maxSigma=6e6, maxTau=6e6, ratioTC=0.5,
        createDistance=2 * r * 1.002)
    return workloads.fibre_bed_case(seed, n // 10 * 10, radius=r, box_xy=(side, side), bond=bond, dt=1e-7, skin=2e-4,
                                    vmax=0.05, plate_vel=(0.0, 0.0, -0.05), plate_gap=0.0)


def _ensemble(n, seed):
    # about 2,000 to 20,000 spheres each; the systems' sizes and materials belong to the case, the state to the seed
    systems = ensemble.settling_systems(n, max(4, int(round(n / 11_000.0))))
    for k, c in enumerate(systems):
        _in_motion(c, seed + 1000 * k, 0.3, 50.0)
    return systems


def _adjoint(n, seed):
    sp = 2.2e-3
    side = 0.05 if n >= 5000 else 0.02
    m = int(side / sp)
    c = workloads.lattice_case(seed, m, m, -(-n // (m * m)), sp, radius=(0.9e-3, 1.1e-3), z0=1.32e-3, jitter=0.05 * sp,
                               E=(1e7,), nu=(0.3,), rest=((0.6,),), frict=((0.5,),), dt=1e-6, skin=5e-4, zhi=0.3,
                               pad=(side - m * sp, side - m * sp))
    return _first(c, n)


_SYSTEMS = dict(pour=_pour, column=_column, hooke=_hooke, bed=_bed, hopper=_hopper, mixer=_mixer, fibres=_fibres,
                ensemble=_ensemble, adjoint=_adjoint)


def _system(case, seed):
    return _SYSTEMS[case["kind"]](case["n"], seed)


# ----------------------------------------------------------------------------
# prepare, run
# ----------------------------------------------------------------------------

def _pinned(n):
    """The caller's page-locked arrays for DemSystem.atoms(out=...)."""
    ints = {k: torch.zeros(n, dtype=torch.int32).pin_memory().numpy() for k in ("tag", "type")}
    vecs = {k: torch.zeros((n, 3), dtype=torch.float64).pin_memory().numpy() for k in ("x", "v", "omega", "f", "torque")}
    return {**ints, **vecs, **{k: torch.zeros(n, dtype=torch.float64).pin_memory().numpy() for k in ("radius", "rmass")}}


def prepare(case, seed):
    c = _system(case, seed)
    if case["kind"] == "adjoint":
        from gb300dem.adjoint import DemAdjoint, make_loss
        mat = c["material"]
        return dict(case=case, engine=DemAdjoint(c), spec=make_loss(w_ke=1.0),
                    at=(mat["E"][0], mat["rest"][0][0], mat["frict"][0][0]))
    if case["kind"] == "ensemble":
        e = ensemble.Ensemble(c)
        e.setup()
        return dict(case=case, keep=e, system=e.sys, out=_pinned(len(e.case["atoms"]["tag"])))
    n = len(c["atoms"]["tag"])
    g = api.DemSystem({k: v for k, v in c.items() if k != "atoms"})
    state = dict(case=case, system=g, out=_pinned(n))
    if case["whole"]:
        host = {k: torch.from_numpy(np.ascontiguousarray(v)).pin_memory().numpy() for k, v in c["atoms"].items()}
        state["atoms"] = host
    else:
        g.upload(c["atoms"])
        g.setup()
    return state


def run(state):
    case = state["case"]
    if case["kind"] == "adjoint":
        seg = max(1, int(round(case["steps"] ** 0.5)))
        loss, grad = state["engine"].gradient(*state["at"], nsteps=case["steps"], segment=seg, loss=state["spec"])
        return dict(loss=loss, E=grad["E"], restitution=grad["restitution"], friction=grad["friction"],
                    radius=grad["radius"], **state["engine"].final_state())
    g = state["system"]
    if case["whole"]:
        g.upload(state["atoms"])
        g.setup()
    g.step(case["steps"])
    return g.atoms(state["out"])


# touching contacts and list entries per sphere
_DENSITY = dict(pour=(0.5, 2.9), column=(0.4, 2.9), hooke=(0.45, 3.0), bed=(2.6, 5.8), hopper=(0.4, 2.7),
                mixer=(0.2, 2.9), fibres=(0.9, 3.7), ensemble=(0.1, 2.9), adjoint=(0.1, 2.9))


def work(case):
    """Per step and sphere: x, v and omega read and written (144 B), radius, mass and inertia factors (24 B); per
    list entry its two atoms (8 B); per touching contact its history read and written and its constants (72 B; a bond
    adds its 28 values).  FP64 operations: 34 per sphere, 204 per touching contact, about 900 per bond.  The gradient
    goes over each step three times (forward, replay, reverse); the download writes 144 B per sphere."""
    touch, entries = _DENSITY[case["kind"]]
    per = 168.0 + 8.0 * entries + 72.0 * touch
    flops = 34.0 + 204.0 * touch
    if case["kind"] == "fibres":
        per += 0.9 * 448.0
        flops += 0.9 * 900.0
    n, passes = float(case["n"]), 3.0 if case["kind"] == "adjoint" else 1.0
    return {"bytes": n * (per * case["steps"] * passes + 144.0), "flops": n * flops * case["steps"] * passes}


# ----------------------------------------------------------------------------
# the same systems in plain torch, FP64: primitive planes only
# ----------------------------------------------------------------------------

def exact(case, seed):
    """Mesh walls (closest features of neighbouring triangles with their history slots), bonds and gradients have no
    value here short of writing the whole framework once more: None."""
    if case["kind"] not in ("pour", "column", "hooke", "bed", "ensemble") or case["n"] * case["steps"] > 50_000_000:
        return None
    c = _system(case, seed)
    if case["kind"] == "ensemble":
        c = ensemble.pack(c)[0]
    p = _Plain(c)
    p.build(p.every())
    p.forces(False)
    for _ in range(case["steps"]):
        p.step()
    return p.atoms()


class _Plain:
    """Velocity Verlet of spheres with the Hertz or Hooke law, tangential history and CDT rolling friction in a box
    periodic in x and y above a floor plane; atoms keep their input order, `order` is the cell-sorted one."""

    def __init__(self, c):
        d = self.dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
        t = lambda a: torch.as_tensor(np.array(a, dtype=np.float64), device=d)  # noqa: E731
        a = c["atoms"]
        self.c, self.n = c, len(a["tag"])
        self.tag, self.type = (torch.as_tensor(np.array(a[k]), dtype=torch.int64, device=d) for k in ("tag", "type"))
        self.x, self.v, self.w, self.r, self.m = (t(a[k]) for k in ("x", "v", "omega", "radius", "rmass"))
        self.tab = {k: t(np.asarray(c[k]).reshape(c["ntypes"] + 1, c["ntypes"] + 1))
                    for k in ("Yeff", "Geff", "betaeff", "coeffRestLog", "coeffFrict", "coeffRollFrict")}
        self.lo, self.prd = t(c["boxlo"]), t(c["boxhi"]) - t(c["boxlo"])
        self.per = torch.as_tensor(np.array(c["periodic"]), device=d) != 0
        self.g, self.dt, self.skin = t(c["gravity"]), c["dt"], c["skin"]
        cut = 2.0 * float(self.r.max()) + self.skin
        self.nc = [max(1, int(math.floor(float(q) / (cut * (1.0 + 1e-9))))) for q in self.prd]
        self.sys = self.type - 1 if c.get("ensemble") else torch.zeros_like(self.type)
        self.nsys = int(c.get("ensemble") or 1)
        if c.get("ensemble"):
            axis, pos, roll = c["planes_per_type"][0]
            self.planes = [(axis, t(pos)[self.type], self.type, roll)]
        else:
            self.planes = [(axis, torch.full((self.n,), pos, dtype=torch.float64, device=d),
                            torch.full_like(self.type, wt), roll) for axis, pos, wt, roll in c["planes"]]
        self.wall_hist = [torch.zeros_like(self.x) for _ in self.planes]
        self.order = torch.arange(self.n, device=d)
        self.hold = self.x.clone()
        self.i = self.j = torch.zeros(0, dtype=torch.int64, device=d)
        self.hist = torch.zeros((0, 3), dtype=torch.float64, device=d)

    def every(self):
        return torch.ones(self.nsys, dtype=torch.bool, device=self.dev)

    def image(self, dx):
        return torch.where(self.per, dx - self.prd * torch.round(dx / self.prd), dx)

    def build(self, which):
        """Neighbour lists, cell order and history carry-over of the systems in the mask `which`."""
        mine = which[self.sys]
        x = self.x
        y = torch.where(x < self.lo, x + self.prd, x)
        y = torch.where(y >= self.lo + self.prd, y - self.prd, y)
        self.x = torch.where(mine[:, None] & self.per, y, x)
        self.hold = torch.where(mine[:, None], self.x, self.hold)
        cell = [((self.x[:, k] - self.lo[k]) * (1.0 / (self.prd[k] / self.nc[k]))).long().clamp(0, self.nc[k] - 1)
                for k in range(3)]
        ncell = self.nc[0] * self.nc[1] * self.nc[2]
        key = cell[0] + self.nc[0] * (cell[1] + self.nc[1] * cell[2]) + ncell * self.sys
        # systems that do not rebuild keep their order: their cells count as one
        key = torch.where(mine, key, ncell * self.sys)
        self.order = self.order[torch.argsort(key[self.order], stable=True)]
        count = torch.bincount(key, minlength=ncell * self.nsys)
        start = torch.cumsum(count, 0) - count
        found_i, found_j = [], []
        me = torch.nonzero(mine).flatten()
        for code in range(27):
            off = (code % 3 - 1, code // 3 % 3 - 1, code // 9 - 1)
            at, ok = [], torch.ones_like(me, dtype=torch.bool)
            for k in range(3):
                q = cell[k][me] + off[k]
                if bool(self.per[k]):
                    q = q % self.nc[k]
                ok &= (q >= 0) & (q < self.nc[k])
                at.append(q.clamp(0, self.nc[k] - 1))
            other = at[0] + self.nc[0] * (at[1] + self.nc[1] * at[2]) + ncell * self.sys[me]
            cnt = torch.where(ok, count[other], 0)
            for s in range(int(cnt.max())):
                i = me[cnt > s]
                j = self.order[start[other[cnt > s]] + s]
                dx = self.image(self.x[i] - self.x[j])
                near = (j > i) & ((dx * dx).sum(1) < (self.r[i] + self.r[j] + self.skin) ** 2)
                found_i.append(i[near])
                found_j.append(j[near])
        i, j = torch.cat(found_i), torch.cat(found_j)
        hist = torch.zeros((len(i), 3), dtype=torch.float64, device=self.dev)
        if len(self.i):
            old = self.i * self.n + self.j
            sort = torch.argsort(old)
            pos = torch.searchsorted(old[sort], i * self.n + j).clamp(max=len(old) - 1)
            dx = self.image(self.x[i] - self.x[j])
            keep = (old[sort][pos] == i * self.n + j) & ((dx * dx).sum(1) < (self.r[i] + self.r[j]) ** 2)
            hist[keep] = self.hist[sort[pos[keep]]]
        stay = ~mine[self.i]
        self.i, self.j = torch.cat([self.i[stay], i]), torch.cat([self.j[stay], j])
        self.hist = torch.cat([self.hist[stay], hist])

    def law(self, ti, tj, overlap, en, dist, vr, ri, rj, wi, wj, meff, reff, shear, update, rolling):
        """Force on i and torques on i and j of contacts whose centres lie `dist` apart along en (j to i); rj None: a
        wall.  Updates `shear` in place."""
        T = {k: v[ti, tj] for k, v in self.tab.items()}
        vn = (vr * en).sum(1, keepdim=True)
        cri = ri - 0.5 * overlap
        crj = torch.zeros_like(cri) if rj is None else rj - 0.5 * overlap
        wr = (cri / dist)[:, None] * wi + (crj / dist)[:, None] * wj
        vt = vr - vn * en + torch.linalg.cross(en * dist[:, None], wr)
        if self.c["normal_model"] == 0:
            root = torch.sqrt(reff * overlap)
            kn, kt = 4.0 / 3.0 * T["Yeff"] * root, 8.0 * T["Geff"] * root
            damp = -2.0 * math.sqrt(5.0 / 6.0) * T["betaeff"]
            gn, gt = damp * torch.sqrt(2.0 * T["Yeff"] * root * meff), damp * torch.sqrt(kt * meff)
        else:
            root, Y = torch.sqrt(reff), T["Yeff"]
            kn = kt = 16.0 / 15.0 * root * Y * (15.0 * meff * self.c["charVel"] ** 2 / (16.0 * root * Y)) ** 0.2
            ln2 = T["coeffRestLog"] ** 2
            gn = gt = torch.sqrt(4.0 * meff * kn * ln2 / (ln2 + math.pi ** 2))
        fn = kn * overlap - gn * vn[:, 0]
        s = shear.clone()
        if update:
            s = s + vt * self.dt
            s = s - (s * en).sum(1, keepdim=True) * en
        spring = kt * torch.sqrt((s * s).sum(1))
        cap = T["coeffFrict"] * fn.abs()
        slide = (spring > cap)[:, None]
        s = torch.where(slide, s * (cap / torch.where(spring > 0, spring, 1.0))[:, None], s)
        ft = -kt[:, None] * s - torch.where(slide, 0.0, gt[:, None] * vt)
        if update:
            shear.copy_(s)
        tor = torch.linalg.cross(en, ft)
        roll = torch.zeros_like(tor)
        if rolling:
            wrel = wr if rj is None else wi - wj
            size = torch.sqrt((wrel * wrel).sum(1))
            fac = torch.where(size > 0, T["coeffRollFrict"] * kn * overlap * reff / torch.where(size > 0, size, 1.0), 0.0)
            roll = fac[:, None] * wrel
            roll = roll - (roll * en).sum(1, keepdim=True) * en
        return fn[:, None] * en + ft, -cri[:, None] * tor - roll, -crj[:, None] * tor + roll

    def forces(self, update):
        f, q = self.m[:, None] * self.g, torch.zeros_like(self.x)
        dx = self.image(self.x[self.i] - self.x[self.j])
        rsq, rs = (dx * dx).sum(1), self.r[self.i] + self.r[self.j]
        on = torch.nonzero(rsq < rs * rs).flatten()
        i, j, r = self.i[on], self.j[on], torch.sqrt(rsq[on])
        shear = self.hist[on]
        ri, rj, mi, mj = self.r[i], self.r[j], self.m[i], self.m[j]
        F, Ti, Tj = self.law(self.type[i], self.type[j], rs[on] - r, dx[on] / r[:, None], r, self.v[i] - self.v[j], ri, rj,
                             self.w[i], self.w[j], mi * mj / (mi + mj), ri * rj / (ri + rj), shear, update,
                             self.c["rolling_model"])
        self.hist[on] = shear
        f.index_add_(0, i, F).index_add_(0, j, -F)
        q.index_add_(0, i, Ti).index_add_(0, j, Tj)
        for (axis, pos, wt, rolling), hist in zip(self.planes, self.wall_hist):
            gap = self.x[:, axis] - pos
            near = gap.abs() <= self.r
            on = torch.nonzero(near).flatten()
            hist[~near] = 0.0
            en = torch.zeros((len(on), 3), dtype=torch.float64, device=self.dev)
            en[:, axis] = torch.sign(gap[on])
            shear = hist[on]
            ri, r = self.r[on], gap[on].abs()
            F, Ti, _ = self.law(self.type[on], wt[on], ri - r, en, r, self.v[on], ri, None, self.w[on],
                                torch.zeros_like(en), self.m[on], ri, shear, update, rolling)
            hist[on] = shear
            f.index_add_(0, on, F)
            q.index_add_(0, on, Ti)
        self.f, self.q = f, q

    def kick(self):
        h = 0.5 * self.dt
        self.v = self.v + h * self.f / self.m[:, None]
        self.w = self.w + h * self.q / (0.4 * self.m * self.r * self.r)[:, None]

    def step(self):
        self.kick()
        self.x = self.x + self.dt * self.v
        d = self.x - self.hold
        moved = torch.zeros(self.nsys, dtype=torch.bool, device=self.dev)
        moved[self.sys[(d * d).sum(1) > 0.25 * self.skin * self.skin]] = True
        if bool(moved.any()):
            self.build(moved)
        self.forces(True)
        self.kick()

    def atoms(self):
        o = self.order
        of = lambda v: v[o].cpu().numpy()  # noqa: E731
        return dict(tag=of(self.tag.int()), type=of(self.type.int()), x=of(self.x), v=of(self.v), omega=of(self.w),
                    f=of(self.f), torque=of(self.q), radius=of(self.r), rmass=of(self.m))
