"""What stops the multi-step kernel.  A wait between its blocks that runs out of
time (a limit of one clock cycle, which nearly every wait exceeds): the chunk is
rolled back and steps by launches, with the same bits, and nothing of the
interrupted steps reaches later ones; without rollback the context refuses to
step until the next commit.  A launch that the runtime refuses: the arena steps
by captured graphs."""
import numpy as np
import pytest

from mjolnir_b200 import _capi as A
from mjolnir_b200 import systems as S
from mjolnir_b200.engine import Engine

pytestmark = pytest.mark.gpu


def systems(name):
    lj = S.lj_fluid(n=4096, margin=0.1, seed=6)          # more blocks than one cluster
    if name == "lj":
        return [lj]
    out = [lj, S.polymer_melt(nchains=4, nbeads=50, radius=50.0, seed=31, margin=0.1),
           S.bead_fluid(n=9000, density=0.003, seed=33, dt=0.6, margin=0.1)]
    for d, kind in zip(out, ("UnderdampedLangevin", "G-JFLangevin", "BAOAB")):
        d.integrator = kind
    return out


def engine(name, **kw):
    e = Engine("mixed", **kw)
    ids = [e.add_system(d) for d in systems(name)]
    e.commit()
    return e, ids


def states(e, ids):
    return [x for sid in ids for x in (*e.state(sid), np.array([e.step_count(sid)]))]


@pytest.mark.parametrize("name", ["lj", "integrators"])
def test_chunk_is_rolled_back_and_launched(name):
    ref, rid = engine(name, graphs=False)
    e, ids = engine(name)
    for k, limit in ((20, 0), (2500, 1), (30, 1), (40, 0)):   # 2,500 steps: several launches in a chunk
        ref.step(k)
        e.debug_set_wait_limit(limit)
        e.step(k)
        for x, y in zip(states(e, ids), states(ref, rid)):
            assert np.array_equal(x, y), (k, limit)
    e.debug_set_wait_limit(1)
    e.step(5)
    e.rebuild()                                               # counters of a rebuild start clean
    ref.step(5)
    ref.rebuild()
    for sid, r in zip(ids, rid):
        for t in ("exv", "dh", "lj"):
            try:
                want = ref.neighbors(r, t)
            except A.MjgError:
                continue
            assert np.array_equal(e.neighbors(sid, t), want)
    e.close()
    ref.close()


def test_without_rollback_steps_are_refused_until_commit():
    e, ids = engine("lj", rollback=False)
    e.step(10)
    e.debug_set_wait_limit(1)
    with pytest.raises(A.MjgError) as err:
        e.step(50)
    assert err.value.code == A.ECUDA
    e.debug_set_wait_limit(0)
    with pytest.raises(A.MjgError) as err:
        e.step(1)
    assert err.value.code == A.ESTATE
    d = systems("lj")[0]
    e.set_state(ids[0], d.pos, d.vel)
    e.commit()
    e.step(25)
    ref, rid = engine("lj")
    ref.step(10)
    ref.set_state(rid[0], d.pos, d.vel)
    ref.commit()
    ref.step(25)
    for x, y in zip(states(e, ids), states(ref, rid)):
        assert np.array_equal(x, y)
    e.close()
    ref.close()


@pytest.mark.parametrize("rollback", [True, False])
def test_refused_launch_steps_by_graphs(rollback):
    """More blocks than any GPU holds at once: the runtime returns an error and launches nothing."""
    ref, rid = engine("integrators", graphs=False)
    e, ids = engine("integrators", rollback=rollback)
    for k, blocks in ((5, 0), (40, 1 << 20), (30, 1 << 20), (40, 0), (20, 3), (20, 11)):   # 3: one small cluster
        e.debug_set_run_blocks(blocks)
        n0 = e.launch_count()
        e.step(k)
        assert (e.launch_count() - n0 == 1) == (blocks < 100)
        ref.step(k)
        for x, y in zip(states(e, ids), states(ref, rid)):
            assert np.array_equal(x, y), (k, blocks)
    e.debug_set_run_blocks(1 << 20)
    e.step(1)
    e.debug_set_run_blocks(0)
    e.close()
    ref.close()
