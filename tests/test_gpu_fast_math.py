"""The mixed form's single-instruction reciprocal, reciprocal root and power of
two (mjolnir_b200/csrc/pair_eval.cuh) against CUDA's functions that they stand
for, over every FP32 mantissa, and what they do with coincident particles."""
import ctypes as C
import os
import subprocess

import pytest

from conftest import ROOT
from mjolnir_b200 import _capi as A
from mjolnir_b200 import build
from mjolnir_b200 import systems as S
from mjolnir_b200.engine import Engine

pytestmark = pytest.mark.gpu


class Result(C.Structure):
    _fields_ = [("differ", C.c_ulonglong), ("beyond", C.c_ulonglong), ("worst", C.c_double)]


@pytest.fixture(scope="module")
def scan(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("fast_math") / "fast_math.so")
    subprocess.run([build.nvcc(), *build.ARCH, *build.NVFLAGS, "-I", build.CSRC, "-shared", "-o", so,
                    os.path.join(ROOT, "tests", "fast_math.cu"), "-lcudart"], check=True)
    fn = C.CDLL(so).fast_math_scan

    def call(which, first_exp, exps):
        r = Result()
        assert fn(which, first_exp, exps, C.byref(r)) == 0
        return r
    return call


def test_reciprocal(scan):
    """Squared distances from 2^-60 to 2^60."""
    r = scan(0, -60, 120)
    assert r.differ == 0 and r.beyond == 0
    assert r.worst <= 2.0 ** -24               # half a unit in the last place


def test_reciprocal_root(scan):
    r = scan(1, -60, 120)
    assert r.differ == 0


def test_exponential(scan):
    """Distances from 2^-10 to 2^6 Debye lengths."""
    r = scan(2, -10, 16)
    assert r.differ == 0


@pytest.mark.parametrize("kind", ["exv", "dh", "lj"])
def test_coincident_particles_are_reported(kind):
    """A pair at distance zero has no finite force; the reciprocal's Newton step and the products that follow
    give NaN or infinity, and the range check must refuse both."""
    if kind == "lj":
        d = S.lj_fluid(n=512, seed=3)
    else:
        d = S.bead_fluid(n=1000, density=0.003, seed=3, dt=0.3)
        if kind == "exv":
            d.dh = None
        else:
            d.exv = None
    i, j = (d.dh.idx[:2] if kind == "dh" else (0, 1))
    d.pos = d.pos.copy()
    d.pos[j] = d.pos[i]
    for graphs in (True, False):
        e = Engine("mixed", graphs=graphs)
        e.add_system(d)
        with pytest.raises(A.MjgError) as err:
            e.commit()
            e.step(1)
        assert err.value.code in (A.EOVERFLOW, A.ENONFINITE)
        e.close()
