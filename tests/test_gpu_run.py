"""The multi-step kernel of small arenas against the step's own launches
(graphs off): the same bits in the mixed form, the order of the FP64 sums apart
in the plain form.  Sizes at the edges of its split: less than a warp, one
cluster, a ragged last warp, several particles per thread, several systems."""
import numpy as np
import pytest

from mjolnir_b200 import systems as S
from mjolnir_b200.engine import Engine

pytestmark = pytest.mark.gpu


def cube(d):
    r = float(np.abs(d.pos).max()) + 2.0
    d.boundary, d.lower, d.upper = "PeriodicCuboid", (-r, -r, -r), (r, r, r)
    return d


def systems(name):
    if name == "beads_5":                       # no list has a partner for long
        return [S.polymer_melt(nchains=1, nbeads=5, radius=30.0, seed=3, charged_fraction=0.9)]
    if name == "chain_33":
        return [S.polymer_melt(nchains=1, nbeads=33, radius=40.0, seed=4, margin=0.1)]
    if name == "melt_cube":
        return [cube(S.polymer_melt(nchains=9, nbeads=111, radius=55.0, seed=5, margin=0.15))]
    if name == "lj":
        return [S.lj_fluid(n=4096, margin=0.1, seed=6)]
    if name == "fluid_40001":                   # several pair items per warp, cells of many members
        return [S.bead_fluid(n=40001, density=0.003, seed=7, margin=0.1, dt=0.6)]
    out = [S.polymer_melt(nchains=4, nbeads=50, radius=50.0, seed=31, margin=0.1), S.lj_fluid(n=343, seed=32, margin=0.05),
           S.bead_fluid(n=1500, density=0.003, seed=33, dt=0.6, margin=0.1),
           cube(S.polymer_melt(nchains=3, nbeads=41, radius=40.0, seed=34, margin=0.1))]
    if name == "integrators":
        for d, kind in zip(out, ("UnderdampedLangevin", "VelocityVerlet", "G-JFLangevin", "g-BAOABLangevin")):
            d.integrator = kind
        return out
    return [d for k in range(16) for d in (S.polymer_melt(nchains=1, nbeads=20 + 7 * k, radius=40.0, seed=50 + k, margin=0.1),
                                           out[k % 4])]     # 32 systems


def run(name, precision, graphs, half=False, frozen=False, steps=(1, 37, 62)):
    descs = systems(name)
    e = Engine(precision, graphs=graphs)
    ids = [e.add_system(d) for d in descs]
    if half:
        for t in ("exv", "dh", "lj"):
            e.set_half_lists(t, True)
    e.commit()
    if frozen:
        e.freeze(ids[1])
    n0 = e.launch_count()
    for k in steps:
        e.step(k)
    launches = e.launch_count() - n0
    out = []
    for sid, d in zip(ids, descs):
        terms = [t for t in ("exv", "dh", "lj") if getattr(d, t) is not None]
        out.append((e.state(sid), e.step_count(sid), [e.rebuild_count(sid, t) for t in terms],
                    [e.neighbors(sid, t) for t in terms]))
    e.close()
    return out, launches


@pytest.mark.parametrize("name", ["beads_5", "chain_33", "melt_cube", "lj", "fluid_40001", "integrators", "many"])
@pytest.mark.parametrize("precision", ["mixed", "fp64"])
def test_steps_of_one_launch_equal_the_launched_steps(name, precision):
    got, few = run(name, precision, True)
    want, many = run(name, precision, False)
    assert few < many / 20
    for g, w in zip(got, want):
        assert g[1] == w[1] and g[2] == w[2]
        assert all(np.array_equal(x, y) for x, y in zip(g[3], w[3]))
        for x, y in zip(g[0], w[0]):
            if precision == "mixed":
                assert np.array_equal(x, y)
            else:
                # the sums of a step differ by rounding (1e-16 of the terms); 100 steps of these systems
                # amplify that by less than a factor of 1e4 (the liquid's e-fold is about 40 steps)
                assert np.abs(x - y).max() <= 1e-10 * max(1.0, np.abs(y).max())
    assert any(any(c > 0 for c in g[2]) for g in got) or name == "beads_5"


@pytest.mark.parametrize("half,frozen", [(True, False), (False, True), (True, True)])
def test_half_lists_and_frozen_systems(half, frozen):
    got, _ = run("many", "mixed", True, half, frozen)
    want, _ = run("many", "mixed", False, False, frozen)
    for g, w in zip(got, want):
        assert g[1] == w[1] and g[2] == w[2]
        for x, y in zip(g[0], w[0]):
            assert np.array_equal(x, y)


@pytest.mark.parametrize("graphs", [True, False])
def test_fp64_runs_repeat(graphs):
    """FP64 sums that no launch leaves to the order of arrival repeat bit for bit: three pair terms on one
    particle, and pair terms beside at most two bonds."""
    three = S.bead_fluid(n=1500, density=0.003, seed=33, dt=0.6, margin=0.1)
    lj = S.lj_fluid(n=343, seed=32, margin=0.05)
    three.lj = lj.lj
    three.lj.idx = np.arange(three.n)
    three.lj.param0, three.lj.param1 = np.full(three.n, 4.0), np.full(three.n, 0.3)
    bonded = S.polymer_melt(nchains=9, nbeads=111, radius=55.0, seed=5, margin=0.15)
    bonded.angles = bonded.dihedrals = None
    outs = []
    for _ in range(3):
        e = Engine("fp64", graphs=graphs)
        ids = [e.add_system(d) for d in (three, bonded)]
        e.commit()
        e.step(300)
        outs.append([x for sid in ids for x in e.state(sid)])
        e.close()
    for o in outs[1:]:
        assert all(np.array_equal(x, y) for x, y in zip(o, outs[0]))


@pytest.mark.parametrize("name,per_launch", [("chain_33", 1024), ("integrators", 1024), ("fluid_40001", 209)])
def test_chunks_of_several_launches(name, per_launch):
    """A chunk longer than a launch: the closing half of the step before opens the next launch, and the step
    counters, margins and displacements carry over."""
    steps = (per_launch, per_launch + 1, 2 * per_launch + 17)
    got, few = run(name, "mixed", True, steps=steps)
    want, _ = run(name, "mixed", False, steps=steps)
    assert few == 1 + 2 + 3
    for g, w in zip(got, want):
        assert g[1] == w[1] and g[2] == w[2]
        assert all(np.array_equal(x, y) for x, y in zip((*g[0], *g[3]), (*w[0], *w[3])))


def test_overflow_in_a_later_launch_rolls_the_chunk_back():
    """A list that outgrows its capacity only in the second launch of a chunk or later: the copy that the first
    launch took is restored, with the accelerations of UnderdampedLangevin and the coefficients of G-JF."""
    descs = [S.lj_fluid(n=1000, density=0.3, margin=0.05, seed=44 + k) for k in range(3)]      # condenses
    for d, kind in zip(descs, ("UnderdampedLangevin", "G-JFLangevin", "BAOAB")):
        d.integrator = kind

    def states(steps, cap=None):
        e = Engine("mixed")
        ids = [e.add_system(d) for d in descs]
        e.commit()
        if cap:
            e.debug_set_list_capacity("lj", cap)
        n0 = e.launch_count()
        e.step(steps)
        launches = e.launch_count() - n0
        out = [x for sid in ids for x in e.state(sid)]
        e.close()
        return out, launches

    # the smallest capacity that the first launch's lists keep within
    cap = next(c for c in range(24, 129) if states(1024, c)[1] == 1)
    want, plain = states(5000)
    got, redone = states(5000, cap)
    assert plain == 5 and redone > 5
    assert all(np.array_equal(x, y) for x, y in zip(got, want))


@pytest.mark.parametrize("graphs", [True, 2, False])
def test_capacity_of_contiguous_lists(graphs):
    """Lists stored particle by particle keep their distance when the capacity is lowered below their length, and
    take a capacity that is no multiple of a copy's 16 bytes: the lists stay readable, and the overflow is met."""
    d = S.lj_fluid(n=1000, density=0.8, margin=0.1, seed=44)
    want = None
    for schedule, caps in ((0, ()), (5, (8,)), (5, (333, 9))):
        e = Engine("mixed", graphs=graphs)
        sid = e.add_system(d)
        e.commit()
        e.set_pair_schedule("lj", schedule)
        pairs = e.neighbors(sid, "lj")
        for cap in caps:
            e.debug_set_list_capacity("lj", cap)
            assert np.array_equal(e.neighbors(sid, "lj"), pairs)
        got = [x for k in (1, 300) for x in (e.step(k), *e.state(sid))[1:]]
        e.close()
        want = want or got
        assert all(np.array_equal(x, y) for x, y in zip(got, want))
