"""The calls whose time matters to a user of this package, over the range in which they are made.

Four kinds of work, each through its public entry point:

  snapshot    force_snapshot_noalloc: the forces of one replica on buffers that the caller owns
              (a host program with its own allocator);
  interval    REMDGPU.ExecuteSteps + all_averages: one REMD interval of a T x P grid of replicas of
              one system (or of several systems at once: `batch`), the call a REMD driver makes
              over and over.  FP32 force arithmetic, the default, or FP64, the plain form that
              validation and drift runs use;
  checkpoint  an interval at whose end the driver writes its checkpoints: the state of every
              replica comes back to the host (ConvertVariablesToHost);
  relax       REMDGPU.equilibrate: MD steps launched one by one, then the velocity rescale, as every
              run starts.

Sizes follow the package's own systems (remd_b200.systems): 64 .. 4096 molecules of TIP3P, TIP4P or
TIP5P in bulk, in a nanotube or in a slit, cutoffs 8.5 .. 12 A, 1 .. 256 replicas.  Intervals are 10
or more MD steps.

What run() hands on has the precision that the handle computes forces in: an FP32 handle's averages
and states, which leave a program as text of seven digits, as float32; an FP64 handle's, and the
caller's own force buffers, as they are.
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

from remd_b200 import engine as E
from remd_b200 import systems as S
from remd_b200.inputs import ELE, UNIT_COULOMB, UNIT_TIME, ReplicaState, SystemSpec, load_model, moltype_path

BULK, TUBE, SLIT = 0, 1, 2
NFWALL = 1000


def listed():
    return [
        # one small confined replica: launches and latency are all there is
        dict(name="snapshot tube 128", kind="snapshot", model="tip4p", confined=TUBE, nmol=128, wall=6.5, rc=8.5,
             rs=7.5),
        # the largest replica the caller-buffer call takes in earnest, on an odd size
        dict(name="snapshot bulk 1999", kind="snapshot", model="tip5p", confined=BULK, nmol=1999, wall=0.0, rc=12.0,
             rs=10.0),
        # a quick look at one replica of the smallest size
        dict(name="interval one tube 64", kind="interval", model="tip3p", confined=TUBE, nmol=64, wall=7.0, rc=8.5,
             rs=7.5, ntemp=1, npress=1, interval=10, precision="fp32"),
        # a nanotube study: TIP4P, N = 128, 4 T x 4 P
        dict(name="interval tube 128x16", kind="interval", model="tip4p", confined=TUBE, nmol=128, wall=6.0, rc=8.5,
             rs=7.5, ntemp=4, npress=4, interval=50, precision="fp32"),
        # a nano-slit study: TIP4P, N = 512, 16 T x 4 P
        dict(name="interval slit 512x64", kind="interval", model="tip4p", confined=SLIT, nmol=512, wall=10.0, rc=10.0,
             rs=9.0, ntemp=16, npress=4, interval=20, precision="fp32"),
        # bulk TIP5P with the longest cutoff, a moderate grid
        dict(name="interval bulk 1728x16", kind="interval", model="tip5p", confined=BULK, nmol=1728, wall=0.0, rc=12.0,
             rs=10.0, ntemp=8, npress=2, interval=10, precision="fp32"),
        # a long tube: few neighbours, many molecules, cell lists
        dict(name="interval tube 4096x8", kind="interval", model="tip4p", confined=TUBE, nmol=4096, wall=7.0, rc=10.0,
             rs=9.0, ntemp=4, npress=2, interval=10, precision="fp32"),
        # the throughput workload: eight uneven systems, 256 replicas, in one handle
        dict(name="batch of eight systems", kind="batch", batch=4, interval=10, precision="fp32"),
        # the same work in the plain form, as validation runs use it: a small confined system ...
        dict(name="fp64 slit 200x4", kind="interval", model="tip4p", confined=SLIT, nmol=200, wall=10.0, rc=9.0, rs=8.0,
             ntemp=2, npress=2, interval=20, precision="fp64"),
        # ... and a bulk one of ordinary size
        dict(name="fp64 bulk 729x8", kind="interval", model="tip3p", confined=BULK, nmol=729, wall=0.0, rc=10.0, rs=9.0,
             ntemp=4, npress=2, interval=10, precision="fp64"),
        # an interval that ends in a checkpoint of every replica
        dict(name="checkpoint slit 300x8", kind="checkpoint", model="tip3p", confined=SLIT, nmol=300, wall=12.0, rc=9.5,
             rs=8.5, ntemp=4, npress=2, interval=10, precision="fp32"),
        # the start of a run: MD steps and the velocity rescale
        dict(name="relax bulk 512x8", kind="relax", model="tip4p", confined=BULK, nmol=512, wall=0.0, rc=10.0, rs=9.0,
             ntemp=8, npress=1, interval=10, precision="fp32"),
    ]


def _geometry(rng, nmol, confined, rc):
    """(confined, wall, rc) of a liquid-density system that fits the minimum image, as
    systems.feasible_geometry makes it (tubes of 6 .. 8 A, slits of 7 .. 14 A)."""
    tube, slit = rng.uniform(6.0, 8.0), rng.uniform(7.0, 14.0)
    wall = {BULK: 0.0, TUBE: tube, SLIT: slit}[confined]
    if S.feasible_periodic_length(confined, nmol, wall) < 2.0 * rc + 2.0:
        rc = (S.feasible_periodic_length(confined, nmol, wall) - 2.0) / 2.0
        if rc < 8.5:
            confined, wall, rc = TUBE, tube, 8.5
    return confined, wall, rc


def draw(rng):
    kind = rng.choice(["snapshot", "snapshot", "interval", "interval", "interval", "interval", "fp64", "checkpoint",
                       "relax", "batch"])
    if kind == "batch":
        return dict(kind="batch", batch=rng.randrange(1000, 1000000), interval=rng.randint(8, 10), precision="fp32")
    model = rng.choice(["tip3p", "tip4p", "tip5p"])
    biggest = {"snapshot": 2048, "interval": 4096, "fp64": 900, "checkpoint": 2048, "relax": 2048}[kind]
    nmol = int(round(math.exp(rng.uniform(math.log(64), math.log(biggest)))))
    confined, wall, rc = _geometry(rng, nmol, rng.choice([BULK, TUBE, SLIT]), rng.uniform(8.5, 12.0))
    rs = rc - rng.choice([1.0, 2.0])
    case = dict(kind="interval" if kind == "fp64" else kind, model=model, confined=confined, nmol=nmol,
                wall=round(wall, 3), rc=round(rc, 3), rs=round(rs, 3))
    if kind == "snapshot":
        return case
    most = {"interval": 60000, "fp64": 6000, "checkpoint": 8000, "relax": 16000}[kind] // nmol
    nrep = int(round(math.exp(rng.uniform(0.0, math.log(max(1, min(64, most)))))))
    npress = rng.choice([n for n in (1, 2, 4) if n <= nrep])
    case.update(ntemp=max(1, nrep // npress), npress=npress, interval=rng.randint(10, 20 if nmol < 1000 else 10),
                precision="fp64" if kind == "fp64" else "fp32")
    return case


# ---------------------------------------------------------------- inputs
@functools.lru_cache(maxsize=64)
def _start(model, confined, nmol, wall, rc):
    """The lattice start of a system: box fractions, orientations, box (without the seed's motion)."""
    rng = np.random.default_rng([nmol, confined, int(1000 * wall), int(1000 * rc)])
    mt = load_model(model)
    pos, L = S.lattice(confined, nmol, wall, rc, rng)
    return pos / L, S.orientations(pos, L, mt.r, mt.charge, rng, tries=12), L


def _ensemble(name, model, confined, nmol, wall, rc, rs, ntemp, npress, interval, seed, thermal=True):
    """A T x P grid of replicas: the lattice start, each replica's molecules moved and turned a little
    and given velocities of its temperature, all from the seed."""
    mt = load_model(model)
    r0, q0, L = _start(model, confined, nmol, wall, rc)
    pconstant = {BULK: 1, TUBE: 2, SLIT: 3}[confined]
    Q, W = max(nmol / 128.0, 0.25), S.barostat_mass(pconstant, L, wall, confined)
    spec = SystemSpec(nmol=nmol, moltype=mt, tconstant=1, pconstant=pconstant, confined=confined, dt=2.0, rcut=rc,
                      rswitch=rs, nfwall=NFWALL if confined else 0, wall_length=wall, sgm_wall=S.WALL_SGM,
                      eps_wall=S.WALL_EPS, rho_wall=S.WALL_RHO, tstat_mass=Q, bstat_mass=W, interval=interval,
                      moltype_file=moltype_path(model))
    T, P = S.conditions_geometrical(ntemp, npress, 240.0, 360.0, 0.1e6, 200e6)
    ens = S.Ensemble(name, spec, ntemp, npress, T, P)
    m, inertia = mt.reduced_mass(), mt.reduced_inertia()
    for k in range(ntemp * npress):
        rng = np.random.default_rng([seed, nmol, confined, k])
        q = q0 + 0.02 * rng.normal(size=q0.shape)
        st = ReplicaState(r=(r0 + rng.normal(size=r0.shape) * (0.03 / L)) % 1.0, v=np.zeros((nmol, 3)),
                          q=q / np.linalg.norm(q, axis=1, keepdims=True), p=np.zeros((nmol, 4)), m=np.full(nmol, m),
                          I=np.tile(inertia, (nmol, 1)), Q=Q, W=W, L=L.copy(), T=T[k], P=P[k])
        if thermal:
            S.thermalize(st, confined, rng)
        ens.states.append(st)
    return ens


def _batch(number):
    """Eight uneven systems, 256 replicas: sizes, models, confinement and cutoffs drawn from the number
    as systems.config4 draws them (124 .. 736 molecules for number 4)."""
    rng = np.random.default_rng(number)
    grids = [S.CONFIG4_GRIDS[i] for i in rng.permutation(len(S.CONFIG4_GRIDS))]
    for nt, npr in grids:
        nmol = int(round(math.exp(rng.uniform(math.log(64), math.log(2048 if number == 4 else 900)))))
        model = ["tip3p", "tip4p", "tip5p"][rng.integers(3)]
        confined = int(rng.integers(3))
        tube, slit = float(rng.uniform(6.0, 8.0)), float(rng.uniform(7.0, 14.0))
        rc, drs = float(rng.uniform(8.5, 12.0)), float(rng.choice([1.0, 2.0]))
        confined, wall, rc = S.feasible_geometry(rng, confined, nmol, tube, slit, rc)
        yield model, confined, nmol, wall, rc, rc - drs, nt, npr


def _ensembles(case, seed):
    if case["kind"] == "batch":
        return [_ensemble("batch.%d" % k, *s, case["interval"], seed + k) for k, s in enumerate(_batch(case["batch"]))]
    return [_ensemble(case["kind"], *(case[k] for k in ("model", "confined", "nmol", "wall", "rc", "rs")),
                      case.get("ntemp", 1), case.get("npress", 1), case.get("interval", 10), seed,
                      thermal=case["kind"] != "snapshot")]


class _Snapshot:
    """The caller's buffers of one replica."""

    def __init__(self, ens):
        self.spec, st = ens.spec, ens.states[0]
        n, dev = self.spec.nmol, dict(dtype=torch.float64, device="cuda")
        self.L = st.L
        self.r, self.q = torch.tensor(st.r, **dev), torch.tensor(st.q, **dev)
        self.wall = None
        if self.spec.confined:
            s = self.spec
            self.wall = torch.tensor(E.wall_table(s.confined, s.nfwall, s.wall_length, s.sgm_wall, s.eps_wall,
                                                  s.rho_wall), **dev)
        self.f, self.n = torch.empty((n, 3), **dev), torch.empty((n, 4), **dev)
        self.out = torch.empty(8, **dev)


class _Run:
    """A handle and the conditions its driver passes."""

    def __init__(self, case, ensembles):
        self.kind, self.precision, self.steps = case["kind"], case["precision"], case["interval"]
        self.eng = E.REMDGPU(ensembles, precision=case["precision"])
        self.T = np.concatenate([e.T for e in ensembles])
        self.P = np.concatenate([e.P for e in ensembles])


def prepare(case, seed):
    ensembles = _ensembles(case, seed)
    return _Snapshot(ensembles[0]) if case["kind"] == "snapshot" else _Run(case, ensembles)


def run(state):
    if isinstance(state, _Snapshot):
        s = state
        E.force_snapshot_noalloc(s.spec, s.r.data_ptr(), s.q.data_ptr(), s.L,
                                 s.wall.data_ptr() if s.wall is not None else 0, s.f.data_ptr(), s.n.data_ptr(),
                                 s.out.data_ptr(), torch.cuda.current_stream().cuda_stream)
        return {"force": s.f, "torque": s.n, "sums": s.out.float()}   # FP32 pair sums
    kept = np.float64 if state.precision == "fp64" else np.float32
    if state.kind == "relax":
        state.eng.equilibrate(rounds=1, steps=state.steps)
    else:
        state.eng.ExecuteSteps(state.T, state.P)
    out = {"averages": state.eng.all_averages().astype(kept)}
    if state.kind == "checkpoint" or state.precision == "fp64":
        views = [state.eng.ConvertVariablesToHost(k) for k in range(state.eng.nrep)]
        for name in ("r", "v", "q", "p"):
            out[name] = np.stack([g[name] for g in views]).astype(kept)
    return out


# ---------------------------------------------------------------- work
def _pairs(model, confined, nmol, wall, rc):
    """Unordered molecule pairs within rc at the start's density."""
    if confined == BULK:
        near = 0.0334 * 4.0 / 3.0 * math.pi * rc ** 3
    elif confined == TUBE:
        near = 2.0 * rc * nmol / S.feasible_periodic_length(TUBE, nmol, wall)
    else:
        near = math.pi * rc * rc * nmol / S.feasible_periodic_length(SLIT, nmol, wall) ** 2
    return 0.5 * nmol * min(nmol - 1, near)


def work(case):
    """Snapshot: positions and orientations in, forces and torques out.  Otherwise the molecule state in
    and out once a pass, and per MD step 326 flops a molecule pair (TIP3P, TIP4P) or 515 (TIP5P)."""
    if case["kind"] == "batch":
        systems = list(_batch(case["batch"]))
    else:
        systems = [tuple(case[k] for k in ("model", "confined", "nmol", "wall", "rc", "rs")) +
                   (case.get("ntemp", 1), case.get("npress", 1))]
    nbytes = flops = 0.0
    for model, confined, nmol, wall, rc, _, nt, npr in systems:
        reps = nt * npr
        flops += reps * _pairs(model, confined, nmol, wall, rc) * (515 if model == "tip5p" else 326)
        nbytes += reps * (nmol * 8 * (14 if case["kind"] == "snapshot" else 28) + 8 * 19)
    return {"bytes": nbytes, "flops": flops * case.get("interval", 1)}


# ---------------------------------------------------------------- the same in 64 bits
def exact(case, seed):
    ensembles = _ensembles(case, seed)
    if case["kind"] == "snapshot":
        sim = _Exact(ensembles[0])
        sim.forces()
        sums = torch.cat([sim.lj, sim.clmb, sim.wall, sim.vir[0], sim.npairs.double(), sim.npairs.double() * 0.0])
        return {"force": sim.f[0], "torque": sim.n[0], "sums": sums}
    sims = [_Exact(e) for e in ensembles]
    for sim in sims:
        sim.start()
        sim.interval(case["interval"])
        if case["kind"] == "relax":
            sim.rescale()
    out = {"averages": torch.cat([s.averages() for s in sims])}
    if case["kind"] == "checkpoint" or case["precision"] == "fp64":
        out.update(r=sims[0].r, v=sims[0].v, q=sims[0].q, p=sims[0].p)
    return out


def _wall_table(spec):
    """{force, energy} at nfwall radii (tube) or half-spacings (slit), lengths in A, energies in kJ/mol."""
    n, R, sigma, eps = spec.nfwall, spec.wall_length, spec.sgm_wall, spec.eps_wall
    dr = R / n
    if spec.confined == TUBE:
        s6 = float(np.float32(float(np.float32(sigma)) ** 6))
        phi = math.pi - np.arange(10000) * (math.pi / 10000)
        u = np.empty(n)
        for i in range(n):
            r = i * dr
            x = 1.0 / np.sqrt((R * R + r * r - 2.0 * R * r * np.cos(phi)).astype(np.float32)).astype(np.float64)
            u[i] = np.sum(63.0 / 32.0 * s6 * x ** 11 - 3.0 * x ** 5)
        u *= math.pi * spec.rho_wall * eps * s6 * R * (math.pi / 10000)
        f = np.zeros(n)
        f[1:-1] = -(u[2:] - u[:-2]) / (2.0 * dr * np.arange(1, n - 1) * dr)
        f[0] = f[1]
        f[-1] = (f[-2] - f[-3]) * 2.0 + f[-3]
    else:
        i = np.arange(n) * dr * 0.5
        d, e = 1.0 / (0.5 * R + i), 1.0 / (0.5 * R - i)
        f = (9.0 * eps * d ** 9 - 3.0 * sigma * d ** 3) * d - (9.0 * eps * e ** 9 - 3.0 * sigma * e ** 3) * e
        u = eps * d ** 9 - sigma * d ** 3 + eps * e ** 9 - sigma * e ** 3
    return np.stack([f, u], 1)


def _basis(a, k):
    """P_k of a quaternion array."""
    a0, a1, a2, a3 = a.unbind(-1)
    return torch.stack({1: (-a1, a0, a3, -a2), 2: (-a2, -a3, a0, a1), 3: (-a3, a2, -a1, a0)}[k], -1)


class _Exact:
    """The replicas of one ensemble in 64 bits: all pairs, plain torch."""

    def __init__(self, ens):
        self.spec = spec = ens.spec
        mt = spec.moltype
        dev = "cuda" if torch.cuda.is_available() else "cpu"
        put = lambda a: torch.tensor(np.array(a), dtype=torch.float64, device=dev)  # noqa: E731
        self.put = put
        for name in ("r", "v", "q", "p", "L", "Pv"):
            setattr(self, name, put([getattr(s, name) for s in ens.states]))
        for name in ("s", "Ps", "T", "P"):
            setattr(self, name, put([getattr(s, name) for s in ens.states]))
        self.Q, self.W, self.m = ens.states[0].Q, ens.states[0].W, float(ens.states[0].m[0])
        self.I, self.body = put(ens.states[0].I[0]), put(mt.r)
        self.R, self.N = len(ens.states), spec.nmol
        self.dt = spec.dt * 1e-15 / UNIT_TIME
        charge = mt.charge * (ELE / UNIT_COULOMB)
        self.sites = [(k, l, float(charge[k] * charge[l])) for k in range(mt.nsite) for l in range(mt.nsite)
                      if charge[k] * charge[l] != 0.0 or k == l == 0]
        self.sigma2, self.eps = float(mt.sigma[0]) ** 2, float(mt.eps[0])
        if spec.confined:
            self.table = put(_wall_table(spec))
        self.gkT = 6.0 * self.N * self.T

    def turn(self):
        """Rotation matrices (body to space) of the quaternions."""
        a, b, c, d = self.q.unbind(-1)
        rows = ((a * a + b * b - c * c - d * d, 2 * (b * c - a * d), 2 * (b * d + a * c)),
                (2 * (b * c + a * d), a * a - b * b + c * c - d * d, 2 * (c * d - a * b)),
                (2 * (b * d - a * c), 2 * (c * d + a * b), a * a - b * b - c * c + d * d))
        return torch.stack([torch.stack(x, -1) for x in rows], -2)

    def neighbours(self):
        """Pairs i < j within the cutoff as flat indexes into replicas x molecules."""
        found = []
        upper = torch.ones((self.N, self.N), dtype=torch.bool, device=self.r.device).triu(1)
        for k in range(self.R):
            d2 = torch.zeros((self.N, self.N), dtype=torch.float64, device=self.r.device)
            for x in range(3):
                a = self.r[k, :, x]
                d = a[:, None] - a[None, :]
                d2 += ((d - d.round()) * self.L[k, x]) ** 2
            i, j = torch.nonzero((d2 <= self.spec.rcut ** 2) & upper, as_tuple=True)
            found.append((i + k * self.N, j + k * self.N))
        return torch.cat([i for i, _ in found]), torch.cat([j for _, j in found])

    def forces(self):
        """Forces, body torques, energies and virial: switched Lennard-Jones between the oxygens and
        Coulomb between the charged sites, the switch acting on the centres' distance; the wall."""
        R, N, spec = self.R, self.N, self.spec
        rot = self.turn()
        off = torch.einsum("rnxy,ky->rnkx", rot, self.body)
        fs, fc = torch.zeros_like(off).view(R * N, -1, 3), torch.zeros((R * N, 3), dtype=off.dtype, device=off.device)
        lj, clmb = (torch.zeros(R, dtype=off.dtype, device=off.device) for _ in range(2))
        vir = torch.zeros((R, 3), dtype=off.dtype, device=off.device)
        flat, pos, every_i, every_j = off.reshape(R * N, -1, 3), self.r.reshape(R * N, 3), *self.neighbours()
        rc, rs = spec.rcut, spec.rswitch
        self.npairs = torch.bincount(every_i // N, minlength=R)
        for part in range(0, len(every_i), 2000000):
            i, j = every_i[part:part + 2000000], every_j[part:part + 2000000]
            rep = i // N
            L = self.L[rep]
            d = pos[i] - pos[j]
            d = (d - d.round()) * L
            dist = d.norm(dim=1)
            a, b = dist - rc, dist - rs
            far = (dist > rs).double()
            c = 1.0 / (rs - rc) ** 5
            sw = 1.0 - far + far * c * a ** 3 * (10.0 * b * b - 5.0 * a * b + a * a)
            dsw = far * 30.0 * c * a * a * b * b
            total, el, ec = torch.zeros_like(d), torch.zeros_like(dist), torch.zeros_like(dist)
            for k, l, qq in self.sites:
                x = d + flat[i, k] - flat[j, l]
                x = x - L * (x / L).round()
                inv2 = 1.0 / (x * x).sum(1)
                inv = inv2.sqrt()
                t = qq * inv * inv2
                ec += qq * inv
                if k == l == 0:
                    s6 = (self.sigma2 * inv2) ** 3
                    el += 4.0 * self.eps * s6 * (s6 - 1.0)
                    t = t + 48.0 * self.eps * s6 * (s6 - 0.5) * inv2
                t = x * (t * sw)[:, None]
                fs[:, k].index_add_(0, i, t)
                fs[:, l].index_add_(0, j, t, alpha=-1.0)
                total += t
            t = d * (-dsw / dist * (el + ec))[:, None]
            fc.index_add_(0, i, t)
            fc.index_add_(0, j, t, alpha=-1.0)
            vir.index_add_(0, rep, (total + t) * d)
            lj.index_add_(0, rep, sw * el)
            clmb.index_add_(0, rep, sw * ec)
        fs, fc = fs.view(R, N, -1, 3), fc.view(R, N, 3)
        self.wall = torch.zeros_like(lj)
        if spec.confined:
            x = (self.r - 0.5) * self.L[:, None] + off[:, :, 0]
            x = x[..., :2] if spec.confined == TUBE else x[..., 2:]
            rad = x.norm(dim=-1)
            dr = spec.wall_length / spec.nfwall * (1.0 if spec.confined == TUBE else 0.5)
            at = (rad / dr).clamp(max=spec.nfwall - 2).long()
            slope = (self.table[at + 1] - self.table[at]) / dr
            f, u = (slope * (rad - dr * at.double())[..., None] + self.table[at]).unbind(-1)
            if spec.confined == TUBE:
                fs[:, :, 0, :2] += f[..., None] * x
            else:
                fs[:, :, 0, 2] += f * torch.where(x[..., 0] < 0, -1.0, 1.0)
            self.wall = u.sum(1)
        self.f = fc + fs.sum(2)
        fb = torch.einsum("rnyx,rnky->rnkx", rot, fs)
        b = self.body.expand_as(fb)
        self.n = torch.cat([(b * fb).sum((2, 3))[..., None], torch.linalg.cross(b, fb).sum(2)], -1)
        self.lj, self.clmb, self.vir, self.pot = lj, clmb, vir, lj + clmb + self.wall

    def volume(self):
        if self.spec.confined == TUBE:
            return math.pi * (self.spec.wall_length - 1.7) ** 2 * self.L[:, 2]
        return self.L[:, 0] * self.L[:, 1] * (self.spec.wall_length if self.spec.confined == SLIT else self.L[:, 2])

    # Nose-Poincare thermostat, Andersen barostat (pconstant 1 in bulk, 2 in a tube, 3 in a slit)
    def thermostat(self):
        c = 1.0 + self.Ps / (2.0 * self.Q) * 0.5 * self.dt
        self.s, self.Ps = self.s * c * c, self.Ps / c

    def kick(self):
        h = 0.5 * self.dt
        self.v = self.v + self.f * (self.L * self.s[:, None])[:, None] * h / self.m
        q, n = self.q, self.n
        sn = q * n[..., :1] + sum(_basis(q, k) * n[..., k:k + 1] for k in (1, 2, 3))
        self.p = self.p + sn * (2.0 * self.s * h)[:, None, None]
        self.Ps = self.Ps - self.pot * h - self.P * self.volume() * h
        L, V, s = self.L, self.vir, self.s
        if self.spec.confined == BULK:
            self.Pv[:, 0] += (V.sum(1) / (3.0 * L.prod(1)) - self.P) * s * h
        elif self.spec.confined == TUBE:
            self.Pv[:, 2] += s * (V[:, 2] / L[:, 2] - self.P * math.pi * (self.spec.wall_length - 1.7) ** 2) * h
        else:
            w = self.spec.wall_length
            self.Pv[:, 0] += s * (V[:, 0] / L[:, 0] - self.P * L[:, 1] * w) * h
            self.Pv[:, 1] += s * (V[:, 1] / L[:, 1] - self.P * L[:, 0] * w) * h

    def box(self):
        h, Pv = 0.5 * self.dt, self.Pv
        if self.spec.confined == BULK:
            self.Ps = self.Ps - Pv[:, 0] ** 2 / self.W * h
            V = (self.volume() + Pv[:, 0] * self.s / self.W * h).float()   # the method's box length is a float
            self.L = (V.double() ** float(np.float32(1.0 / 3.0))).float().double()[:, None].repeat(1, 3)
        elif self.spec.confined == TUBE:
            self.Ps = self.Ps - 0.5 * Pv[:, 2] ** 2 / self.W * h
            self.L[:, 2] += self.s * Pv[:, 2] / self.W * h
        else:
            self.Ps = self.Ps - (Pv[:, 0] ** 2 + Pv[:, 1] ** 2) * 0.5 / self.W * h
            self.L[:, :2] += (self.s[:, None] * Pv[:, :2]) * (0.5 / self.W) * self.dt

    def spin(self, axis, h):
        """Free rotation about a body axis; its kinetic sum."""
        Pq, Pp, inertia = _basis(self.q, axis), _basis(self.p, axis), self.I[axis - 1]
        xi = (self.p * Pq).sum(-1) * (0.25 / self.s)[:, None] / inertia
        c, s = torch.cos(xi * h)[..., None], torch.sin(xi * h)[..., None]
        self.q, self.p = self.q * c + Pq * s, self.p * c + Pp * s
        return (xi * xi).sum(1) * inertia

    def step(self, first):
        h = 0.5 * self.dt
        if not first:
            self.kick()
            self.thermostat()
        self.thermostat()
        self.kick()
        self.box()
        sums = 0.5 * self.spin(3, h) + 0.5 * self.spin(2, h)
        r = self.r + self.v * (self.dt / (self.L ** 2 * self.s[:, None]))[:, None]
        self.r = r - r.floor()
        sums = sums + self.spin(1, self.dt) + 0.5 * self.spin(2, h) + 0.5 * self.spin(3, h)
        kin = (2.0 * self.m * self.v ** 2).sum(1) / (self.L * self.s[:, None]) ** 2
        if self.spec.confined == BULK:
            self.Pv[:, 0] += self.s * kin.sum(1) / (self.volume() * 3.0) * h
        elif self.spec.confined == TUBE:
            self.Pv[:, 2] += self.s * kin[:, 2] / self.L[:, 2] * h
        else:
            self.Pv[:, :2] += self.s[:, None] * kin[:, :2] / self.L[:, :2] * h
        self.Ps = self.Ps + (0.25 * kin.sum(1) + 2.0 * sums - (1.0 + self.s.log()) * self.gkT + self.H0) * self.dt
        self.box()
        self.forces()

    def start(self):
        self.forces()
        self.H0 = torch.zeros_like(self.s)
        self.H0 = self.averages()[:, 11]

    def interval(self, steps):
        for k in range(steps):
            self.step(k == 0)
        self.kick()
        self.thermostat()

    def kinetic(self):
        tra = (self.v ** 2).sum(1) * self.m * 0.5 / (self.L * self.s[:, None]) ** 2
        xi = torch.stack([(self.p * _basis(self.q, k)).sum(-1) for k in (1, 2, 3)], -1)
        xi = xi * (0.25 / self.s)[:, None, None] / self.I
        return tra, (2.0 * self.I * xi * xi).sum((1, 2))

    def still(self):
        """The mean momentum (in a tube along the axis, with the spin about it) taken out."""
        mean = self.v.mean(1)
        free = {BULK: (1.0, 1.0, 1.0), TUBE: (0.0, 0.0, 1.0), SLIT: (1.0, 1.0, 0.0)}[self.spec.confined]
        self.v = self.v - (mean * self.put(free))[:, None]
        if self.spec.confined == TUBE:
            self.unspin()

    def unspin(self):
        x = (self.r - 0.5) * self.L[:, None]
        scale = (self.L * self.s[:, None])[:, None]
        u = self.v / scale
        lz = (x[..., 0] * u[..., 1] - x[..., 1] * u[..., 0]).mean(1)[:, None]
        r2 = x[..., 0] ** 2 + x[..., 1] ** 2
        w = torch.where(r2 > 1.0, lz / r2, torch.zeros_like(r2))
        turn = torch.stack([w * x[..., 1], -w * x[..., 0], torch.zeros_like(w)], -1)
        self.v = self.v + turn * scale

    def rescale(self):
        """Kinetic energies set to 3/2 N T each, momentum out, s = 1, barostat at rest; H0 anew."""
        want = 1.5 * self.N * self.T
        self.v, self.p = self.v / self.s[:, None, None], self.p / self.s[:, None, None]
        self.s = torch.ones_like(self.s)
        self.v = self.v * (want / self.kinetic()[0].sum(1)).sqrt()[:, None, None]
        self.still()
        if self.spec.confined == TUBE:
            self.unspin()
        self.Ps, self.Pv = torch.zeros_like(self.Ps), torch.zeros_like(self.Pv)
        self.p = self.p * (want / self.kinetic()[1]).sqrt()[:, None, None]
        self.H0 = self.H0 * 0.0
        self.H0 = self.averages()[:, 11]

    def averages(self):
        """The 19 averages of each replica, in the package's order."""
        tra, rot = self.kinetic()
        V, kin = self.volume(), tra.sum(1) + rot
        used = {BULK: self.Pv, TUBE: self.Pv[:, 2:], SLIT: self.Pv[:, :2]}[self.spec.confined]
        tot = (self.pot + kin + 0.5 * self.Ps ** 2 / self.Q + self.gkT * self.s.log() +
               0.5 * (used ** 2).sum(1) / self.W + self.P * V)
        press = (2.0 * tra + self.vir) / V[:, None]
        return torch.stack([self.lj, self.clmb, self.wall, V, tra.sum(1), rot, kin / (3.0 * self.N), press.sum(1) / 3.0,
                            press[:, 0], press[:, 1], press[:, 2], tot, tot - self.H0, self.s, self.Ps, self.Pv[:, 0],
                            self.Pv[:, 1], self.Pv[:, 2], torch.zeros_like(V)], 1)
