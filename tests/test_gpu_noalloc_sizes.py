"""The allocation-free ExcludedVolume entry point at the edges of its launches
(one particle, a ragged group, block and scan boundaries, the largest size; one
cell per axis more or less than a scan block) against the context path."""
import numpy as np
import pytest

from conftest import rel_rms
from mjolnir_b200 import systems as S
from test_zz_no_alloc import context_exv, noalloc_exv

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 31, 33, 257, 3001, 16385, 65536])
@pytest.mark.parametrize("boundary", ["PeriodicCuboid", "Unlimited"])
def test_sizes(n, boundary):
    d = S.bead_fluid(n=max(n, 8), density=0.003, seed=70 + n % 7, dt=0.3)
    d.dh = None
    if n < 8:
        d.pos, d.vel, d.mass, d.gamma = d.pos[:n], d.vel[:n], d.mass[:n], d.gamma[:n]
        d.exv.idx, d.exv.param0 = d.exv.idx[:n], d.exv.param0[:n]
    d.exv.param0 = d.exv.param0 * np.random.default_rng(n).uniform(0.7, 1.0, n)
    d.boundary = boundary
    d.single_molecule = False
    f_ref, e_ref = context_exv(d)
    f, e = noalloc_exv(d)
    # FP64 sums of a few terms each in another order: 1e-12 as in the parity tests
    assert np.isfinite(f).all()
    assert rel_rms(f, f_ref) <= 1e-12
    assert abs(e - e_ref) <= 1e-12 * max(abs(e_ref), 1e-12)
