"""The three ways mjg_step runs an arena: many steps in one launch, captured
graphs (with conditional rebuild nodes where few systems carry a term, plain
rebuild launches otherwise) and separate launches.  Bit for bit the same in the
mixed form, at every launch shape that each of them honours."""
import numpy as np
import pytest

from mjolnir_b200 import systems as S
from mjolnir_b200.engine import Engine

pytestmark = pytest.mark.gpu

DESCS = {
    # few systems: every term's rebuild sits behind a graph conditional
    "few": lambda: [S.polymer_melt(nchains=4, nbeads=60, radius=45.0, seed=41, margin=0.1),
                    S.bead_fluid(n=3000, density=0.003, seed=42, dt=0.6, margin=0.1), S.lj_fluid(n=512, seed=43, margin=0.05)],
    # more than four systems with each of two terms, one of them frozen
    "several": lambda: [S.polymer_melt(nchains=2, nbeads=30 + k, radius=40.0, seed=60 + k, margin=0.1) for k in range(9)],
    # more systems than the multi-step kernel takes
    "many": lambda: [S.polymer_melt(nchains=1, nbeads=10 + k, radius=30.0, seed=100 + k, margin=0.1) for k in range(65)],
}


def run(name, precision="mixed", graphs=True, shape=None, half=False, steps=(1, 2, 3, 4, 5, 6, 40, 31)):
    e = Engine(precision, graphs=graphs)
    ids = [e.add_system(d) for d in DESCS[name]()]
    e.commit()
    if shape:
        for term in ("exv", "dh", "lj") if name == "few" else ("exv", "dh"):
            if half:
                e.set_half_lists(term, True)
            e.set_pair_schedule(term, shape[0])
            e.set_threads_per_particle(term, shape[1])
            e.set_pair_unroll(term, shape[2])
    path = e.step_path()
    for j, k in enumerate(steps):
        if name == "several" and j == 5:
            e.freeze(ids[3])
        e.step(k)
    out = [x for sid in ids for x in (*e.state(sid), np.array([e.step_count(sid)] + [
        e.rebuild_count(sid, t) for t in ("exv", "dh")] if name != "few" else [e.step_count(sid)]))]
    e.close()
    return out, path


@pytest.mark.parametrize("name", ["few", "several", "many"])
def test_paths_agree(name):
    want, path = run(name, graphs=False)
    assert path == 0
    for graphs, expect in ((True, 1 if name == "many" else 2), (2, 1)):
        got, path = run(name, graphs=graphs)
        assert path == expect
        assert all(np.array_equal(x, y) for x, y in zip(got, want))


SHAPES = [(0, 1, 1), (0, 4, 4), (0, 32, 2), (2, 4, 1), (3, 8, 1), (1, 16, 2), (4, 4, 2), (4, 32, 1), (5, 8, 4), (5, 32, 1)]


@pytest.mark.parametrize("graphs", [False, 2, True])
@pytest.mark.parametrize("half", [False, True])
def test_launch_shapes_on_every_path(graphs, half):
    """Every schedule through the launches that honour it (graphs off, captured graphs), and the threads per
    particle and list layouts through the multi-step kernel."""
    want, _ = run("few", graphs=False)
    for shape in SHAPES:
        got, _ = run("few", graphs=graphs, shape=shape, half=half)
        assert all(np.array_equal(x, y) for x, y in zip(got, want)), shape


@pytest.mark.parametrize("graphs", [False, 2, True])
def test_launch_shapes_fp64(graphs):
    want, _ = run("few", "fp64", graphs=False)
    for shape in [s for s in SHAPES if s[0] != 1]:
        got, _ = run("few", "fp64", graphs=graphs, shape=shape)
        for x, y in zip(got, want):
            # rounding of the sums' order, as in the parity test of the launch shapes (velocities and forces react
            # more strongly than positions: the steepest pair potential's relative slope is some 1e2)
            assert np.abs(x - y).max() <= 1e-7 * max(1.0, np.abs(y).max()), shape


def test_the_line_between_the_paths():
    """At the largest arena that steps in one launch, and one particle above it: the mixed form's first steps
    there still run in one launch, and again after a commit; then the graphs are captured."""
    for precision, n, path in (("mixed", 90000, 2), ("mixed", 90001, 1), ("mixed", 131073, 1), ("fp64", 90001, 2)):
        d = S.bead_fluid(n=n, density=0.003, seed=8, dt=0.6, margin=0.05)
        outs = []
        for graphs in (True, False):
            e = Engine(precision, graphs=graphs)
            sid = e.add_system(d)
            e.commit()
            single = []
            for k in (15, 100, 142, 5, 0, 20):
                if k == 0:
                    e.commit()
                    continue
                n0 = e.launch_count()
                e.step(k)
                single.append(e.launch_count() - n0 <= 2)       # at most two launches of the multi-step kernel
            if graphs:
                assert e.step_path() == path
                early = path == 2 or n <= 131072
                assert single == [early, early, path == 2, path == 2, early]
            assert e.rebuild_count(sid, "exv") > 0
            outs.append(e.state(sid))
            e.close()
        for x, y in zip(*outs):
            assert np.array_equal(x, y) if precision == "mixed" else np.abs(x - y).max() <= 1e-7 * np.abs(y).max()
