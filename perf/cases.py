"""Performance cases: the work that users of this package have it do, through its
public entry points (:class:`mjolnir_b200.engine.Engine` and the C ABI).

A case is a plain dict.  ``run(prepare(case, seed))`` is one pass of it,
``work(case)`` the bytes and operations that the pass cannot do without,
``tolerance(case)`` how far another correct implementation may be off, and
``exact(case, seed)`` the pass's outputs from a plain torch restatement of the
same molecular dynamics in 64 bits (which uses none of this package's code
beyond the description of the system).

Kinds of pass:
  step     `steps` integrator steps of resident systems, then the state is read
  upload   new positions and velocities of every system are uploaded, `steps`
           steps run, positions and velocities are downloaded
  observe  `frames` times: `steps` steps, the energies, positions (a simulation
           with its observers)
  forces   new coordinates, then every term's forces and the energies (a host
           program that integrates by itself)
  noalloc  ExcludedVolume forces and energy of the caller's own device arrays
"""
import ctypes
import math

import numpy as np
import torch

from mjolnir_b200 import _capi
from mjolnir_b200 import systems as S
from mjolnir_b200.engine import Engine

TERMS = ("bond", "angle", "dihedral", "exv", "dh", "lj")
MELT_DENSITY = 10000 / (4 / 3 * math.pi * 300.0 ** 3)      # beads per cubic angstrom in the melts

# launch shapes that the autotuner picks for the two large workloads, as a
# program keeps them (they change no result in the mixed form)
BATCH_TUNED = {"exv": dict(schedule=3, tpp=2, unroll=1, lanes=8, half=True),
               "dh": dict(schedule=4, tpp=2, unroll=1, lanes=16, half=False)}
FLUID_TUNED = {"exv": dict(schedule=2, tpp=2, unroll=1, half=False),
               "dh": dict(schedule=5, tpp=8, unroll=1, half=False)}


def _case(name=None, **kw):
    c = dict(kind="step", system="melt", precision="mixed", steps=100, integrator="BAOAB", margin_exv=0.5,
             margin_dh=0.5, tuned=False, mixed_sizes=False, **({"name": name} if name else {}))
    c.update(kw)
    return c


def listed():
    return [
        # the smallest job of a server's stream: one short chain, where launches count
        _case("chain_200", system="melt", chains=1, beads=200),
        # the 4,096-particle Lennard-Jones fluid alone on the GPU, both forms
        _case("lj_4096_mixed", system="lj", n=4096, margin_lj=0.2, steps=50),
        _case("lj_4096_fp64", system="lj", n=4096, margin_lj=0.2, steps=50, precision="fp64"),
        # a 10,000-bead polymer melt alone: the plain FP64 path
        _case("melt_10000_fp64", system="melt", chains=50, beads=200, precision="fp64"),
        # a simulation with its observers: energies and positions every 10 steps; ragged size
        _case("observe_melt_4151", kind="observe", system="melt", chains=7, beads=593, steps=10, frames=10),
        # another integrator and periodic boundaries, particles of uneven size
        _case("gjf_melt_2997", system="melt", chains=27, beads=111, periodic=True, integrator="G-JFLangevin",
              mixed_sizes=True),
        # a server's arena: 40 jobs of uneven size, half of them periodic, untuned
        _case("serve_40", system="batch", nsys=40, nmin=200, nmax=12000, half_periodic=True),
        # the benchmark: 256 melts, tuned shapes, state uploaded and downloaded every 100 steps
        _case("batch_256", kind="upload", system="batch", nsys=256, nmin=500, nmax=20000, margin_exv=0.25,
              margin_dh=0.1, tuned=True),
        # the 1,048,576-bead periodic fluid as one system, tuned shapes
        _case("fluid_1m_mixed", system="fluid", n=1 << 20, margin_exv=0.3, margin_dh=0.1, steps=20, tuned=True),
        # a quarter of it in the plain FP64 form with untuned shapes
        _case("fluid_262k_fp64", system="fluid", n=1 << 18, margin_exv=0.3, margin_dh=0.1, steps=20,
              precision="fp64"),
        # forces and energies of every term at new coordinates, FP64
        _case("forces_32768_fp64", kind="forces", system="fluid", n=32768, margin_exv=0.3, margin_dh=0.1,
              precision="fp64"),
        # the allocation-free ExcludedVolume entry point on device arrays, periodic, odd size
        _case("noalloc_20001", kind="noalloc", system="beads", n=20001, periodic=True, precision="fp64"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    precision = rng.choice(["mixed", "fp64"])
    margins = dict(margin_exv=round(rng.uniform(0.2, 0.6), 2), margin_dh=round(rng.uniform(0.1, 0.5), 2))
    what = rng.choice(["melt", "melt", "lj", "lj", "fluid", "batch", "forces", "observe", "noalloc"])
    integrator = rng.choice(["BAOAB", "BAOAB", "VelocityVerlet", "G-JFLangevin", "UnderdampedLangevin"])
    if what == "lj":
        return _case(system="lj", n=rng.randint(7, 32) ** 3, margin_lj=round(rng.uniform(0.1, 0.5), 2),
                     precision=precision, integrator=rng.choice(["BAOAB", "VelocityVerlet"]),
                     mixed_sizes=rng.random() < 0.5, steps=rng.randint(10, 50))
    if what in ("melt", "observe"):
        n = _log_int(rng, 150, 30000)
        chains = max(1, int(round(n / rng.uniform(60, 400))))
        c = _case(system="melt", chains=chains, beads=max(4, n // chains), precision=precision,
                  periodic=rng.random() < 0.5, mixed_sizes=rng.random() < 0.5, steps=rng.randint(20, 120), **margins)
        if what == "observe":
            c.update(kind="observe", steps=rng.randint(3, 20), frames=5)
        else:
            c.update(integrator=integrator)
        return c
    if what == "fluid":
        return _case(system="fluid", n=_log_int(rng, 3000, 300000), precision=precision, steps=rng.randint(5, 20),
                     mixed_sizes=rng.random() < 0.5, **margins)
    if what == "batch":
        return _case(kind=rng.choice(["step", "upload"]), system="batch", nsys=rng.randint(2, 96),
                     nmin=200, nmax=_log_int(rng, 1000, 12000), half_periodic=rng.random() < 0.5,
                     precision=precision, steps=rng.randint(20, 100), **margins)
    if what == "forces":
        return _case(kind="forces", system=rng.choice(["fluid", "melt_cube"]), n=_log_int(rng, 1000, 120000),
                     precision=precision, mixed_sizes=rng.random() < 0.5, **margins)
    return _case(kind="noalloc", system="beads", n=_log_int(rng, 500, 65536), periodic=rng.random() < 0.7,
                 precision="fp64", mixed_sizes=rng.random() < 0.5)


# ------------------------------------------------------------------ systems

def _uneven(d, seed):
    """Radii, charges and Lennard-Jones parameters of uneven size (never larger than the even ones)."""
    rng = np.random.default_rng([int(seed), 77])
    for t in (d.exv, d.dh):
        if t is not None:
            t.param0 = t.param0 * rng.uniform(0.75, 1.0, len(t.idx))
    if d.lj is not None:
        d.lj.param0 = d.lj.param0 * rng.uniform(0.9, 1.0, len(d.lj.idx))
        d.lj.param1 = d.lj.param1 * rng.uniform(0.5, 1.0, len(d.lj.idx))
    return d


def _in_cube(d):
    """The melt in a periodic cube around its sphere."""
    r = float(np.abs(d.pos).max()) + 2.0
    d.boundary, d.lower, d.upper = "PeriodicCuboid", (-r, -r, -r), (r, r, r)
    return d


def _shake(d, seed, sigma):
    d.pos = d.pos + np.random.default_rng([int(seed), 5]).normal(0.0, sigma, d.pos.shape)
    return d


def _batch(case, seed):
    """Independent melts as systems.polymer_batch draws them (sizes log-uniform, temperature and ionic
    strength per system), the sizes fixed by the case, every second one in a periodic cube if asked."""
    sizes = np.exp(np.random.default_rng([case["nsys"], case["nmax"]]).uniform(
        math.log(case["nmin"]), math.log(case["nmax"]), case["nsys"]))
    rng = np.random.default_rng([seed, 9])
    out = []
    for k, size in enumerate(sizes):
        chains = max(1, int(round(size / 200)))
        beads = max(4, int(round(size / chains)))
        d = S.polymer_melt(nchains=chains, nbeads=beads, radius=300.0 * (chains * beads / 10000.0) ** (1 / 3),
                           temperature=float(rng.uniform(280.0, 360.0)),
                           ionic_strength=float(rng.uniform(0.05, 0.3)), seed=(seed % 100003) * 1009 + k)
        out.append(_in_cube(d) if case.get("half_periodic") and k % 2 else d)
    return out


def _descs(case, seed):
    """The systems of a case, made from the seed alone."""
    seed = int(seed) % (1 << 31)
    sysk = case["system"]
    if sysk == "lj":
        out = [S.lj_fluid(n=case["n"], density=0.8, margin=case["margin_lj"], seed=seed)]
    elif sysk in ("melt", "melt_cube"):
        chains, beads = (case["chains"], case["beads"]) if sysk == "melt" else (max(1, case["n"] // 200), 200)
        radius = (chains * beads / MELT_DENSITY / (4 / 3 * math.pi)) ** (1 / 3)
        out = [S.polymer_melt(nchains=chains, nbeads=beads, radius=max(radius, 40.0), seed=seed)]
        if case.get("periodic") or sysk == "melt_cube":
            out = [_in_cube(d) for d in out]
    elif sysk == "batch":
        out = _batch(case, seed)
    else:
        out = [S.bead_fluid(n=case["n"], density=0.003, seed=seed)]
    for d in out:
        if case["mixed_sizes"]:
            _uneven(d, seed)
        if d.exv is not None:
            d.exv.margin, d.dh.margin = case["margin_exv"], case["margin_dh"]
        d.integrator = case["integrator"]
    return out


class _State:
    pass


def _pinned(n):
    return torch.empty((n, 3), dtype=torch.float64, pin_memory=True)


def prepare(case, seed):
    st = _State()
    st.case = case
    if case["kind"] == "noalloc":
        d = _descs(case, seed)[0]
        st.lib = _capi.lib()
        st.n = d.n
        st.pos = torch.from_numpy(d.pos).cuda()
        st.radius = torch.from_numpy(np.ascontiguousarray(d.exv.param0)).cuda()
        st.force = torch.empty_like(st.pos)
        st.energy = torch.empty(1, dtype=torch.float64, device="cuda")
        st.lower, st.upper = np.array(d.lower), np.array(d.upper)
        st.boundary = _capi.PERIODIC_CUBOID if case["periodic"] else _capi.UNLIMITED
        return st
    descs = _descs(case, seed)
    e = st.engine = Engine(case["precision"])
    shapes = (BATCH_TUNED if case["system"] == "batch" else FLUID_TUNED) if case["tuned"] else {}
    for t, c in shapes.items():             # what may be set before the lists are built
        e.set_half_lists(t, c["half"])
        e.set_pair_schedule(t, c["schedule"])
        e.set_pair_unroll(t, c["unroll"])
        if "lanes" in c:
            e.set_build_lanes(t, c["lanes"])
    st.sids = [e.add_system(d) for d in descs]
    e.commit()
    for t, c in shapes.items():
        e.set_threads_per_particle(t, c["tpp"])
    n = sum(d.n for d in descs)
    st.big = case["kind"] == "upload" or len(descs) > 1 or n > 50000
    if st.big:
        st.pos_out, st.vel_out = _pinned(n), _pinned(n)
    if case["kind"] == "upload":
        st.pos_in, st.vel_in = _pinned(n), _pinned(n)
        e.get_state_all(st.pos_in.numpy(), st.vel_in.numpy())
    if case["kind"] == "forces":
        st.new_pos = _new_pos(descs[0], seed)
        st.present = [t for t in TERMS if _has(descs[0], t)]
    return st


def _has(d, term):
    return getattr(d, {"bond": "bonds", "angle": "angles", "dihedral": "dihedrals"}.get(term, term)) is not None


def _new_pos(d, seed):
    """Coordinates a few steps away from those committed, inside the box."""
    p = _shake(d.copy(), seed, 0.05).pos
    if d.periodic:
        lo, up = np.array(d.lower), np.array(d.upper)
        p = np.where(p < lo, p + (up - lo), np.where(p >= up, p - (up - lo), p))
    return p


def _energies(e, sid):
    got = e.energies(sid)
    return np.array([got[t] for t in TERMS])


def run(st):
    case = st.case
    kind = case["kind"]
    if kind == "noalloc":
        f64 = ctypes.POINTER(ctypes.c_double)
        code = st.lib.mjg_exv_force_noalloc(
            st.n, st.boundary, _capi.f64(st.lower), _capi.f64(st.upper), ctypes.cast(st.pos.data_ptr(), f64),
            ctypes.cast(st.radius.data_ptr(), f64), 0.2, 2.0, ctypes.cast(st.force.data_ptr(), f64),
            ctypes.cast(st.energy.data_ptr(), f64), ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
        if code != _capi.OK:
            raise RuntimeError(f"mjg_exv_force_noalloc: {code}")
        return {"force": st.force, "energy": st.energy}
    e = st.engine
    if kind == "observe":
        frames = []
        for _ in range(case["frames"]):
            e.step(case["steps"])
            frames.append({"energies": _energies(e, st.sids[0]), "pos": e.positions(st.sids[0])})
        return frames
    if kind == "forces":
        sid = st.sids[0]
        e.set_state(sid, pos=st.new_pos)
        out = {}
        for t in st.present:
            f, en = e.term_force(sid, t)
            out[t] = {"force": f, "energy": en}
        return out
    if kind == "upload":
        e.set_state_all(st.pos_in.numpy(), st.vel_in.numpy())
    e.step(case["steps"])
    if st.big:
        e.get_state_all(st.pos_out.numpy(), st.vel_out.numpy())
        return {"pos": st.pos_out, "vel": st.vel_out}
    pos, vel, force = e.state(st.sids[0])
    return {"pos": pos, "vel": vel, "force": force}


# --------------------------------------------------------------------- work

def _beads(case):
    """(beads, bonded beads, charged beads) of a case, expected."""
    k = case["system"]
    if k == "lj":
        return case["n"], 0, 0
    if k == "batch":
        lo, hi = case["nmin"], case["nmax"]
        n = case["nsys"] * ((hi - lo) / math.log(hi / lo) if hi > lo else lo)
        return n, n, 0.2 * n
    if k in ("melt", "melt_cube"):
        n = case["chains"] * case["beads"] if k == "melt" else max(1, case["n"] // 200) * 200
        return n, n, 0.2 * n
    return case["n"], 0, 0.3 * case["n"]


def work(case):
    n, bonded, charged = _beads(case)
    sphere = 4 / 3 * math.pi
    if case["system"] == "lj":
        pair_flops = n * 0.5 * sphere * 2.5 ** 3 * 0.8 * 45
    else:
        rho = 0.003 if case["system"] in ("fluid", "beads") else MELT_DENSITY
        rc = 42.3 if case["system"] == "fluid" else 52.0
        pair_flops = n * 0.5 * sphere * 8.0 ** 3 * rho * 45
        if case["system"] != "beads":
            pair_flops += charged * 0.5 * sphere * rc ** 3 * rho * (charged / n) * 60
    evaluation = pair_flops + bonded * (30 + 90 + 180)
    state = 96.0 * n                       # position and velocity, read and written, 64 bits
    if case["kind"] == "noalloc":
        return {"bytes": 56.0 * n + 8, "flops": evaluation}
    if case["kind"] == "forces":
        terms = (2 if case["system"] == "fluid" else 5)
        return {"bytes": (24.0 + 24.0 * terms) * n, "flops": 2 * evaluation}
    steps = case["steps"] * case.get("frames", 1)
    out = 96.0 * n if case["kind"] == "upload" else 48.0 * n * case.get("frames", 1)
    return {"bytes": state * steps + out, "flops": (evaluation + 150.0 * n) * steps}


def tolerance(case):
    # Measured against exact(): FP64 states 1e-16 to 6e-13 after 100 steps (one force evaluation 8e-16); mixed
    # forces 4e-7, states 3e-7 or less, energies 8e-8.  In the Lennard-Jones liquid trajectories part by about a
    # factor of ten every hundred steps: 7e-7 to 2.5e-6 at step 100, the second pass of 50 steps.
    if case["precision"] == "fp64":
        return {"rel": 3e-12, "max": 1e-9}
    return {"rel": 1e-5, "max": 2e-3} if case["system"] == "lj" else {"rel": 2e-6, "max": 1e-3}


# -------------------------------------------------------------------- exact
# The same molecular dynamics in plain torch, 64 bits.  All systems of a case
# are advanced together; a pair list (every pair within cutoff + skin, found
# along sorted z) is made again when a particle has moved half the skin.

_KB = 1.38064852e-23 * (1.0 / 4.184 / 1000.0) * 6.022140857e23


def _dev():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _pairs_within(pos, box, r):
    """(i, j), i < j, of all pairs of one system with distance below r."""
    dev = pos.device
    n = pos.shape[0]
    z, order = torch.sort(pos[:, 2])
    p = pos[order]
    found = []
    block = 512
    shifts = [0.0] if box is None else [0.0, -float(box[2]), float(box[2])]
    for b in range(0, n, block):
        q = p[b:b + block]
        lo, hi = float(z[b]) - r, float(z[min(b + block, n) - 1]) + r
        if box is not None and hi - lo >= float(box[2]):
            ranges = [(0, n)]
        else:
            ranges = []
            for s in shifts:
                edge = torch.searchsorted(z, torch.tensor([lo + s, hi + s], dtype=z.dtype, device=dev)).tolist()
                if edge[1] > edge[0]:
                    ranges.append(tuple(edge))
        for x, y in ranges:
            for c in range(x, y, 65536):
                cc = p[c:min(c + 65536, y)]
                d2 = torch.zeros((q.shape[0], cc.shape[0]), dtype=torch.float32, device=dev)
                for ax in range(3):
                    d = (cc[None, :, ax] - q[:, None, ax]).float()
                    if box is not None:
                        d = d - float(box[ax]) * torch.round(d / float(box[ax]))
                    d2 += d * d
                a, k = torch.nonzero(d2 < r * r, as_tuple=True)
                a, k = order[b + a], order[c + k]
                m = a < k
                found.append(torch.stack([a[m], k[m]]))
    return torch.cat(found, dim=1) if found else torch.zeros((2, 0), dtype=torch.long, device=dev)


def _mulhilo(a, x):
    p = a * x                                # modulo 2^64
    return (p >> 32) & 0xffffffff, p & 0xffffffff


def _gauss(seed, index, step):
    """Three normal deviates a particle: Philox4x32-10 and Box-Muller, key = seed, counter = (particle, step)."""
    c = [index & 0xffffffff, index >> 32, torch.full_like(index, step & 0xffffffff), torch.full_like(index, step >> 32)]
    k0, k1 = seed & 0xffffffff, (seed >> 32) & 0xffffffff
    for r in range(10):
        if r:
            k0, k1 = (k0 + 0x9E3779B9) & 0xffffffff, (k1 + 0xBB67AE85) & 0xffffffff
        h0, l0 = _mulhilo(0xD2511F53, c[0])
        h1, l1 = _mulhilo(0xCD9E8D57, c[2])
        c = [h1 ^ c[1] ^ k0, l1, h0 ^ c[3] ^ k1, l0]
    u = [x.double() for x in c]
    t = 2.0 ** -32
    r0, r1 = torch.sqrt(-2 * torch.log((u[0] + 0.5) * t)), torch.sqrt(-2 * torch.log((u[2] + 0.5) * t))
    a0, a1 = 2 * math.pi * (u[1] * t), 2 * math.pi * (u[3] * t)
    return torch.stack([r0 * torch.cos(a0), r0 * torch.sin(a0), r1 * torch.cos(a1)], dim=1)


def _debye(T, I):
    """Debye length and Coulomb constant 1 / (4 pi eps) in water, kcal/mol and angstrom."""
    e0 = 8.854187817e-12 / 1.6021766208e-19 / 1.6021766208e-19
    e0 = e0 * (1000.0 / (1.0 / 4.184)) / 6.022140857e23 / 1e10
    ek = (249.4 - 0.788 * T + 7.2e-4 * T * T) * (1 - 2.551e-1 * I + 5.151e-2 * I * I - 6.889e-3 * I ** 3)
    length = math.sqrt(e0 * ek * _KB * T / (2 * 6.022140857e23 * (I / (1e-3 * 1e30))))
    return length, 1.0 / (4 * math.pi * e0 * ek)


class _Exact:
    """Systems side by side in flat arrays."""

    def __init__(self, descs):
        dev = _dev()
        t = lambda x, k=torch.float64: torch.as_tensor(np.ascontiguousarray(x), dtype=k).to(dev)   # noqa: E731
        self.descs, self.off = descs, np.concatenate([[0], np.cumsum([d.n for d in descs])])
        n = int(self.off[-1])
        self.n = n
        self.pos = t(np.concatenate([d.pos for d in descs]))
        self.vel = t(np.concatenate([d.vel for d in descs]))
        self.mass = t(np.concatenate([d.mass for d in descs]))[:, None]
        self.gamma = t(np.concatenate([d.gamma for d in descs]))[:, None]
        self.T = t(np.concatenate([np.full(d.n, d.temperature) for d in descs]))[:, None]
        inf = float("inf")
        self.low = t(np.concatenate([np.tile(d.lower if d.periodic else (-inf,) * 3, (d.n, 1)) for d in descs]))
        self.up = t(np.concatenate([np.tile(d.upper if d.periodic else (inf,) * 3, (d.n, 1)) for d in descs]))
        self.box = torch.where(torch.isinf(self.up), torch.zeros_like(self.up), self.up - self.low)
        self.periodic = any(d.periodic for d in descs)
        self.sys = torch.cat([torch.full((d.n,), k, dtype=torch.long) for k, d in enumerate(descs)]).to(dev)
        self.local = torch.cat([torch.arange(d.n) for d in descs]).to(dev)
        self.dt, self.kind = descs[0].dt, descs[0].integrator
        self.bonded = {}
        for name, key, ar in (("bond", "bonds", 2), ("angle", "angles", 3), ("dihedral", "dihedrals", 4)):
            got = [(o, getattr(d, key)) for o, d in zip(self.off, descs) if getattr(d, key) is not None]
            if got:
                cols = len(got[0][1])
                self.bonded[name] = [t(np.concatenate([o + g[0] for o, g in got]), torch.long)] + \
                    [t(np.concatenate([g[k] for _, g in got]).astype(float)) for k in range(1, cols)]
        self.lists, self.list_pos, self.skin = {}, None, 3.0 if descs[0].lj is None else 0.6
        self.wrap()

    def cutoff(self, d, name):
        if name == "exv":
            return float(d.exv.param0.max()) * 2 * d.exv.cutoff
        if name == "lj":
            return float(d.lj.param0.max()) * d.lj.cutoff
        return _debye(d.temperature, d.ionic_strength)[0] * d.dh.cutoff

    def wrap(self):
        self.pos = torch.where(self.pos < self.low, self.pos + self.box,
                               torch.where(self.pos >= self.up, self.pos - self.box, self.pos))

    def direction(self, i, j):
        d = self.pos[j] - self.pos[i]
        if not self.periodic:
            return d
        b = self.box[i]
        return torch.where(d < -b / 2, d + b, torch.where(d >= b / 2, d - b, d))

    def refresh(self):
        if self.list_pos is not None:
            d = (self.pos - self.list_pos).abs()
            if self.periodic:
                d = torch.minimum(d, (self.box - d).abs().where(self.box > 0, d))
            if float(d.square().sum(1).max()) < (0.5 * self.skin) ** 2:
                return
        self.list_pos = self.pos.clone()
        self.lists = {}
        dev = self.pos.device
        for k, d in enumerate(self.descs):
            o = int(self.off[k])
            box = [u - w for u, w in zip(d.upper, d.lower)] if d.periodic else None
            for name in ("exv", "dh", "lj"):
                t = getattr(d, name)
                if t is None:
                    continue
                idx = torch.as_tensor(t.idx, device=dev)
                pair = idx[_pairs_within(self.pos[o + idx], box, self.cutoff(d, name) + self.skin)]
                if d.bonds is not None and d.ignore_bond_within:        # chains of consecutive beads
                    chain = torch.zeros(d.n, dtype=torch.long, device=dev)
                    starts = np.setdiff1d(np.arange(d.n), np.asarray(d.bonds[0])[:, 1])
                    chain[torch.as_tensor(starts, device=dev)] = 1
                    chain = torch.cumsum(chain, 0)
                    near = (chain[pair[0]] == chain[pair[1]]) & ((pair[0] - pair[1]).abs() <= d.ignore_bond_within)
                    pair = pair[:, ~near]
                p0 = torch.zeros(d.n, dtype=torch.float64, device=dev)
                p0[idx] = torch.as_tensor(t.param0, device=dev)
                p1 = torch.zeros_like(p0)
                if t.param1 is not None:
                    p1[idx] = torch.as_tensor(t.param1, device=dev)
                a, b = pair
                if name == "exv":
                    par = [p0[a] + p0[b], torch.full_like(p0[a], t.epsilon), torch.full_like(p0[a], t.cutoff)]
                elif name == "lj":
                    par = [(p0[a] + p0[b]) / 2, torch.sqrt(p1[a] * p1[b]), torch.full_like(p0[a], t.cutoff)]
                else:
                    ln, c4 = _debye(d.temperature, d.ionic_strength)
                    par = [p0[a] * p0[b] * c4, torch.full_like(p0[a], ln), torch.full_like(p0[a], t.cutoff)]
                self.lists.setdefault(name, []).append((o + a, o + b, *par))
        self.lists = {k: [torch.cat(x) for x in zip(*v)] for k, v in self.lists.items()}

    def pair_term(self, name):
        f = torch.zeros_like(self.pos)
        i, j, s, e, cut = self.lists[name]
        total = 0.0
        for b in range(0, len(i), 1 << 24):
            k = slice(b, b + (1 << 24))
            d = self.direction(i[k], j[k])
            r2 = d.square().sum(1)
            if name == "dh":
                r, ln = r2.sqrt(), e[k]
                inside = r < cut[k] * ln
                ex = torch.exp(-r / ln)
                c = -s[k] * (ln + r) / (ln * r2 * r) * ex
                en = s[k] * (ex / r - torch.exp(-cut[k]) / (cut[k] * ln))
            else:
                inside = r2 <= (s[k] * cut[k]).square()
                q = (s[k].square() / r2) ** 3
                if name == "exv":
                    c, en = -12 * e[k] * q * q / r2, e[k] * (q * q - cut[k] ** -12)
                else:
                    c = 24 * e[k] * (q - 2 * q * q) / r2
                    en = 4 * e[k] * (q * q - q - (cut[k] ** -12 - cut[k] ** -6))
            g = d * torch.where(inside, c, torch.zeros_like(c))[:, None]
            f.index_add_(0, i[k], g)
            f.index_add_(0, j[k], -g)
            total += float(torch.where(inside, en, torch.zeros_like(en)).sum())
        return f, total

    def local_term(self, name):
        f = torch.zeros_like(self.pos)
        idx, k, *par = self.bonded[name]
        if name == "bond":
            d = self.direction(idx[:, 0], idx[:, 1])
            r = d.norm(dim=1)
            g = d * (-2 * k * (r - par[0]) / r)[:, None]
            f.index_add_(0, idx[:, 0], -g)
            f.index_add_(0, idx[:, 1], g)
            return f, float((k * (r - par[0]).square()).sum())
        if name == "angle":
            a, c = self.direction(idx[:, 1], idx[:, 0]), self.direction(idx[:, 1], idx[:, 2])
            la, lc = a.norm(dim=1, keepdim=True), c.norm(dim=1, keepdim=True)
            ea, ec = a / la, c / lc
            cos = (ea * ec).sum(1).clamp(-1, 1)
            th = torch.acos(cos)
            m = (-2 * k * (th - par[0]) / torch.sin(th).clamp(min=1e-8))[:, None]
            fa, fc = m / la * (cos[:, None] * ea - ec), m / lc * (cos[:, None] * ec - ea)
            for q, g in ((0, fa), (1, -fa - fc), (2, fc)):
                f.index_add_(0, idx[:, q], g)
            return f, float((k * (th - par[0]).square()).sum())
        mult, v0 = par
        ij, kj = self.direction(idx[:, 1], idx[:, 0]), self.direction(idx[:, 1], idx[:, 2])
        kl = -self.direction(idx[:, 2], idx[:, 3])
        m, n = torch.linalg.cross(ij, kj), torch.linalg.cross(kj, kl)
        r = kj.norm(dim=1, keepdim=True)
        phi = torch.atan2((ij * n).sum(1) * r[:, 0], (m * n).sum(1))
        co = (k * mult * torch.sin(mult * (phi - v0)))[:, None]
        fi = co * r / m.square().sum(1, keepdim=True) * m
        fl = -co * r / n.square().sum(1, keepdim=True) * n
        x, y = (ij * kj).sum(1, keepdim=True) / r.square(), (kl * kj).sum(1, keepdim=True) / r.square()
        for q, g in ((0, fi), (1, (x - 1) * fi - y * fl), (2, (y - 1) * fl - x * fi), (3, fl)):
            f.index_add_(0, idx[:, q], g)
        return f, float((k * (1 + torch.cos(mult * (phi - v0)))).sum())

    def term(self, name):
        return self.local_term(name) if name in self.bonded else self.pair_term(name)

    def terms(self):
        self.refresh()
        return [t for t in TERMS if t in self.bonded or t in self.lists]

    def forces(self):
        return sum(self.term(t)[0] for t in self.terms())

    def noise(self, step):
        out = torch.empty_like(self.pos)
        for k, d in enumerate(self.descs):
            s = slice(int(self.off[k]), int(self.off[k + 1]))
            out[s] = _gauss(int(d.seed) & ((1 << 64) - 1), self.local[s], step)
        return out

    def run(self, steps, first=0):
        dt, half, m, g = self.dt, self.dt / 2, self.mass, self.gamma
        kT = _KB * self.T
        f = self.forces()
        if self.kind == "UnderdampedLangevin" and first == 0:
            self.acc = f / m + self.noise(0) * torch.sqrt(2 * kT / dt) * torch.sqrt(g / m)
        for t in range(first, first + steps):
            if self.kind == "VelocityVerlet":
                self.vel = self.vel + half / m * f
                self.pos = self.pos + dt * self.vel
            elif self.kind == "BAOAB":
                self.vel = self.vel + half / m * f
                d = half * self.vel
                ex = torch.exp(-g * dt)
                self.vel = self.vel * ex + torch.sqrt(kT * (1 - torch.exp(-2 * g * dt)) / m) * self.noise(t)
                self.pos = self.pos + (d + half * self.vel)
            elif self.kind == "G-JFLangevin":
                b = 1 / (1 + g * dt / (2 * m))
                a = 1 - g * b * dt / m
                beta = torch.sqrt(2 * g * kT * dt) * self.noise(t)
                d = b * dt * (self.vel + (dt * f + beta) / (2 * m))
                self.vel = a * (self.vel + half / m * f) + b / m * beta
                self.pos = self.pos + d
            else:
                o = 1 - g * half
                self.pos = self.pos + dt * o * self.vel + dt * dt / 2 * self.acc
                self.vel = self.vel * (o * (o * o + g * half)) + half * o * self.acc
            self.wrap()
            f = self.forces()
            if self.kind == "UnderdampedLangevin":
                self.acc = f / m + self.noise(t + 1) * torch.sqrt(2 * kT / dt) * torch.sqrt(g / m)
                self.vel = self.vel + half * (1 - g * half) * self.acc
            else:
                self.vel = self.vel + half / m * f
        return f


def exact(case, seed):
    descs = _descs(case, seed)
    kind = case["kind"]
    if kind == "noalloc" and not case["periodic"]:
        descs[0].boundary = "Unlimited"
    if kind == "forces":
        descs[0].pos = _new_pos(descs[0], seed)
    if kind in ("noalloc", "forces"):
        x = _Exact(descs)
        out = {t: dict(zip(("force", "energy"), x.term(t))) for t in x.terms() if kind == "forces" or t == "exv"}
        if kind == "noalloc":
            f, en = out["exv"]["force"], out["exv"]["energy"]
            return {"force": f, "energy": torch.tensor([en], dtype=torch.float64)}
        return out
    x = _Exact(descs)
    if kind == "observe":
        frames = []
        for k in range(case["frames"]):
            x.run(case["steps"], first=k * case["steps"])
            en = {t: x.term(t)[1] for t in x.terms()}
            frames.append({"energies": np.array([en.get(t, 0.0) for t in TERMS]), "pos": x.pos.clone()})
        return frames
    f = x.run(case["steps"])
    big = kind == "upload" or len(descs) > 1 or descs[0].n > 50000
    return {"pos": x.pos, "vel": x.vel} if big else {"pos": x.pos, "vel": x.vel, "force": f}
