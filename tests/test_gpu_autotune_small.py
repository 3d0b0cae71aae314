"""The autotuner on an operator whose launches all take the four-threads-per-
site kernel (hop.cu hop_is_split): it has no shape to choose, and the table
that larger lattices of the same kind, Ls, precision and link form share stays
as it was; above that size it still fills the table."""
import numpy as np
import pytest

from cps_veloc_b200 import _abi as A
from cps_veloc_b200.dirac import DiracOpDwf, DiracOpWilson, Lattice, gen_gauge, gen_gaussian

pytestmark = pytest.mark.gpu


def _op(L, kind, seed):
    lat = Lattice(L, (1, 1, 1, -1))
    lat.import_gauge(gen_gauge(L, seed=seed))
    return lat, DiracOpWilson(lat, mass=0.1) if kind == "wilson" else DiracOpDwf(lat, mass=0.05, ls=8)


def _shapes(lat, D, prec):
    out = []
    for reals in {A.DOUBLE: (None,), A.SINGLE: (12, 18), A.HALF: (12, 18, 112, 118)}[prec]:
        if reals:
            lat.set_link_reals(prec, reals)
        out.append(D.hop_shape(prec))
    return out


@pytest.mark.parametrize("prec", [A.DOUBLE, A.SINGLE, A.HALF])
@pytest.mark.parametrize("kind,small", [("wilson", (4, 4, 4, 4)), ("dwf", (4, 4, 4, 4)), ("dwf", (4, 4, 8, 8))])
def test_small_operator_leaves_the_table(kind, small, prec):
    A.check(A.lib().cpsgpu_finalize())
    big_lat, big = _op((8, 8, 8, 16), kind, 991)
    big.set_hop_shape(prec, 64, 1)  # what a larger lattice runs, in its current link form
    want = _shapes(big_lat, big, prec)
    lat, D = _op(small, kind, 992)
    x = gen_gaussian(D.f_size, seed=993)
    before, _ = D.MatPcDagMatPc(x, A.DOUBLE)
    for nrhs in (1, 2):
        D.autotune(prec, nrhs=nrhs)
    assert _shapes(big_lat, big, prec) == want
    np.testing.assert_array_equal(D.MatPcDagMatPc(x, A.DOUBLE)[0], before)
    A.check(A.lib().cpsgpu_finalize())


def test_larger_operator_still_tunes():
    A.check(A.lib().cpsgpu_finalize())
    _, D = _op((8, 8, 8, 16), "dwf", 994)
    assert D.autotune(A.SINGLE) == 8  # four epilogues, two link forms
    A.check(A.lib().cpsgpu_finalize())
