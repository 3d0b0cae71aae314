"""The kernels take their blocks forwards and backwards in turn (Lattice::turn):
a result has the same bits whichever way the first of its kernels goes.  The
operators here launch an even number of turning kernels or an odd one with a
hop between, so that the repeats start both ways; lattices whose last block of
sites is partial, slabs of more than one block, and launch shapes with both
grid orders (the default small-launch hop does not turn, so a shape is set)."""
import numpy as np
import pytest

from cps_veloc_b200 import _abi as A
from cps_veloc_b200.dirac import DiracOpDwf, DiracOpMobius, DiracOpWilson, Lattice, gen_gauge, gen_gaussian

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", [A.DOUBLE, A.SINGLE, A.HALF])
@pytest.mark.parametrize("kind,L,ls", [("wilson", (6, 4, 6, 10), 1), ("dwf", (6, 4, 2, 6), 5), ("dwf", (4, 4, 6, 6), 8),
                                       ("mobius", (6, 4, 4, 6), 10), ("mobius", (4, 6, 2, 6), 12)])
def test_both_ways_same_bits(kind, L, ls, prec):
    A.check(A.lib().cpsgpu_finalize())  # no shape set by another test
    lat = Lattice(L, (1, -1, 1, -1))
    lat.import_gauge(gen_gauge(L, seed=981))
    D = {"wilson": lambda: DiracOpWilson(lat, mass=0.1), "dwf": lambda: DiracOpDwf(lat, mass=0.05, ls=ls),
         "mobius": lambda: DiracOpMobius(lat, mass=0.05, ls=ls, b=1.5, c=0.5)}[kind]()
    x = gen_gaussian(D.f_size, seed=982)
    for shape in ((32, 1, 1, 0), (32, 1, 1, 1)):
        D.set_hop_shape(prec, *shape)

        def one_hop():  # the next call starts the other way
            D.M5inv(x, 0, prec=prec) if kind == "mobius" else D.Dslash(x, 1, 0, prec)

        def once():
            one_hop()
            y, dot = D.MatPcDagMatPc(x, prec=prec)
            sol = np.zeros_like(x)
            r = D.InvCg(sol, x, stop_rsd=1e-6, max_num_iter=20, precision=prec)
            return y, dot, sol, r.iterations

        first, second = once(), once()
        one_hop()
        third = once()
        for other in (second, third):
            np.testing.assert_array_equal(first[0], other[0])
            np.testing.assert_array_equal(first[2], other[2])
            assert first[1] == other[1] and first[3] == other[3]
    A.check(A.lib().cpsgpu_finalize())
