"""The step's bonded forces, computed from joined records, against the separate
bond, angle and dihedral forces: the same integers in the mixed form, rounding
apart in FP64.  Topologies: chains (every term joins), terms given backwards or
twice, impropers and long-range bonds that join nothing or leave a window."""
import numpy as np
import pytest

from mjolnir_b200 import systems as S
from mjolnir_b200.engine import Engine

pytestmark = pytest.mark.gpu


def system(kind, n):
    rng = np.random.default_rng([n, len(kind)])
    d = S.polymer_melt(nchains=1, nbeads=n, radius=max(40.0, 3.0 * n ** 0.5), seed=n)
    d.exv = d.dh = None
    if kind == "chain":
        return d
    b, a, q = d.bonds[0].copy(), d.angles[0].copy(), d.dihedrals[0].copy()
    if kind == "backwards":                              # every second term starts at its other end
        b[::2], a[::2], q[::2] = b[::2, ::-1], a[::2, ::-1], q[::2, ::-1]
        b, a = np.concatenate([b, b[: n // 3]]), np.concatenate([a, a[: n // 4]])
    else:                                                # impropers, bonds and angles anywhere
        q = np.stack([rng.permutation(n)[:4] for _ in range(n)])
        a = np.stack([rng.permutation(n)[:3] for _ in range(n)])
        b = np.stack([rng.permutation(n)[:2] for _ in range(n)])
    d.bonds = (b, rng.uniform(1, 100, len(b)), rng.uniform(3, 5, len(b)))
    d.angles = (a, rng.uniform(1, 10, len(a)), rng.uniform(1.5, 2.5, len(a)))
    d.dihedrals = (q, rng.uniform(0.1, 1, len(q)), rng.integers(-3, 4, len(q)).astype(np.int32),
                   rng.uniform(-3, 3, len(q)))
    return d


@pytest.mark.parametrize("kind", ["chain", "backwards", "anywhere"])
@pytest.mark.parametrize("n", [5, 255, 256, 257, 700])
@pytest.mark.parametrize("precision", ["mixed", "fp64"])
def test_records_equal_separate_terms(kind, n, precision):
    d = system(kind, n)
    e = Engine(precision)
    sid = e.add_system(d)
    e.commit()
    total = e.state(sid)[2]
    parts = [e.term_force(sid, t)[0] for t in ("bond", "angle", "dihedral")]
    e.close()
    want = parts[0] + parts[1] + parts[2]
    if precision == "mixed":
        # multiples of 2^-28 below 2^22: their FP64 sums are exact
        assert np.array_equal(total, want)
    else:
        # sums of at most some ten terms per particle in another order
        assert np.abs(total - want).max() <= 1e-13 * sum(np.abs(p).max() for p in parts) * 10


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
def test_bond_of_exactly_half_a_box(precision):
    """Two beads exactly half a periodic box apart: the minimum image takes
    -half a box for the bond's displacement (core/BoundaryCondition.hpp:81-91),
    and the step's bonded forces have that direction."""
    d = S.polymer_melt(nchains=1, nbeads=6, radius=40.0, seed=1)
    d.exv = d.dh = None
    d.boundary, d.lower, d.upper = "PeriodicCuboid", (-8.0, -8.0, -8.0), (8.0, 8.0, 8.0)
    d.pos = np.array([[-4.0, 0, 0], [4, 0, 0], [4, -4, 1], [4, 4, 1], [2, 1, 4], [1, 3, -4]], dtype=float)
    d.bonds = (np.array([[0, 1], [2, 3], [4, 5]]), np.full(3, 10.0), np.full(3, 3.8))
    d.angles = (np.array([[0, 1, 2], [2, 3, 4]]), np.full(2, 2.0), np.full(2, 1.9))      # these join two of the bonds
    d.dihedrals = None
    e = Engine(precision)
    sid = e.add_system(d)
    e.commit()
    total = e.state(sid)[2]
    bond, angle = (e.term_force(sid, t)[0] for t in ("bond", "angle"))
    e.close()
    assert bond[0, 0] < 0 < bond[1, 0]        # pulled together through the boundary: r1 - r0 is -8 there
    assert np.abs(total - bond - angle).max() <= (0.0 if precision == "mixed" else 1e-12)
