"""The Ls x Ls mixing as a recurrence along s (mix_scan.cu and the hop's mixing
epilogue) against the oracle: every instantiated Ls and ones that are not,
checkerboards that are no multiple of a block, band (zmobius_dslash_4's b, c
mixing) and scan (M5^-1 and its products) matrices, and the operators whose
matrices do not have the form (|K| > 1, real b_s, c_s that differ between
slices, Ls = 2), which keep the dense kernels."""
import numpy as np
import pytest

from cps_veloc_b200 import _abi as A
from cps_veloc_b200.dirac import DiracOpMobius, Lattice, gen_gauge, gen_gaussian
from helpers import OracleOps, rel

pytestmark = pytest.mark.gpu

TOL = {A.DOUBLE: 1e-13, A.SINGLE: 2e-6, A.HALF: 5e-3}


def _op(oracle, L, ls, b=1.5, c=0.5, mass=0.05, seed=951):
    u = gen_gauge(L, seed=seed)
    lat = Lattice(L)
    lat.import_gauge(u)
    return DiracOpMobius(lat, mass=mass, ls=ls, b=b, c=c), OracleOps(oracle, L, u, ls=ls, b=b, c=c)


def _check(D, ops, mass, prec, pieces=True):
    x = gen_gaussian(D.f_size, seed=952)
    for dag in (0, 1):
        assert rel(D.M5inv(x, dag, prec=prec), ops.mobius_m5inv(x, mass, dag)) < TOL[prec]
        if pieces:
            assert rel(D.Dslash4(x, 0, dag, prec=prec), ops.mobius_dslash_4(x, mass, 0, dag)) < TOL[prec]
    y, dot = D.MatPcDagMatPc(x, prec=prec)
    yo, doto = ops.mobius_mdagm(x, mass)
    assert rel(y, yo) < TOL[prec] and dot == pytest.approx(doto, rel=TOL[prec])


@pytest.mark.parametrize("prec", [A.DOUBLE, A.SINGLE, A.HALF])
@pytest.mark.parametrize("L,ls", [((2, 2, 2, 2), 3), ((4, 2, 2, 2), 4), ((6, 2, 2, 2), 5), ((4, 4, 2, 2), 6),
                                  ((2, 2, 2, 6), 8), ((4, 6, 2, 2), 9), ((6, 6, 2, 2), 10), ((4, 4, 4, 4), 12),
                                  ((2, 6, 2, 6), 14), ((4, 2, 2, 10), 16), ((2, 2, 2, 4), 20), ((2, 2, 2, 2), 24),
                                  ((2, 2, 2, 2), 32), ((4, 4, 2, 4), 7), ((2, 2, 6, 2), 11), ((4, 2, 2, 6), 13), ((2, 4, 2, 2), 15)])
def test_recurrence(oracle, L, ls, prec):
    D, ops = _op(oracle, L, ls)
    _check(D, ops, 0.05, prec)


@pytest.mark.parametrize("prec", [A.DOUBLE, A.SINGLE, A.HALF])
@pytest.mark.parametrize("ls,b,c,mass", [(8, 0.1, 2.0, 0.05),  # K = 2.79
                                         (2, 1.5, 0.5, 0.05), (8, 1.0, 0.0, 0.0)])
def test_edges_of_the_form(oracle, ls, b, c, mass, prec):
    D, ops = _op(oracle, (4, 4, 2, 2), ls, b, c, mass)
    _check(D, ops, mass, prec, pieces=c != 0.0 or prec != A.HALF)


@pytest.mark.parametrize("prec", [A.DOUBLE, A.SINGLE, A.HALF])
def test_real_slices_that_differ_stay_dense(oracle, prec):
    D, ops = _op(oracle, (4, 4, 4, 4), 8)
    b = [1.0 + 0.1 * s for s in range(8)]
    c = [x - 1.0 for x in b]
    D.set_zmobius(b, c)
    ops.set_zmobius([complex(x) for x in b], [complex(x) for x in c])
    x = gen_gaussian(D.f_size, seed=953)
    for impl in (D.MIX_DEFAULT, D.MIX_SHARED):
        D.set_mix_impl(impl)
        for dag in (0, 1):
            assert rel(D.M5inv(x, dag, prec=prec), ops.mobius_m5inv(x, 0.05, dag)) < TOL[prec]


def test_several_right_hand_sides():
    """a batched solve: the recurrence over several right-hand sides, some of
    them finished (their blocks return) while others run"""
    L, ls = (4, 4, 4, 6), 12
    lat = Lattice(L)
    lat.import_gauge(gen_gauge(L, seed=954))
    D = DiracOpMobius(lat, mass=0.05, ls=ls)
    for prec in (A.DOUBLE, A.SINGLE, A.HALF):
        srcs = [gen_gaussian(D.f_size, seed=955 + k) for k in range(3)]
        srcs[1] = 1e-3 * D.MatPcDagMatPc(srcs[1])[0]
        sols = [np.zeros(D.f_size) for _ in srcs]
        for r in D.InvCgMulti(sols, srcs, stop_rsd=1e-10, precision=prec):
            assert r.status == A.CONVERGED and r.true_res <= 1e-10


@pytest.mark.parametrize("b,c,ls", [(1.45, 0.45, 12), (1.0, 0.4545, 8), (1.5, 0.5, 10), (2.5, 1.5, 16), (4.0, 3.0, 6),
                                    (4.5, 3.5, 10)])
def test_precision_of_the_form(oracle, b, c, ls):
    """K from -2e-5 over 0.02 to 0.57 and, dense, 0.62: no term of the recurrence may be larger than the matrix (c / |K|
    is up to 2e4 here).  MatPcDagMatPc is four mixings and four hops; a mixing's error is below 7e-8 in FP32 and 2e-16 in FP64 (the
    roundings of its coefficients and three operations), a hop's below 1.2e-7 and 2.5e-16 (the 2-norm of 8 sums of
    products of unit roundoff 6e-8 and 1.1e-16), and the oracle's as FP64's: 8e-7 and 4e-15 in all."""
    D, ops = _op(oracle, (4, 4, 4, 4), ls, b, c)
    x = gen_gaussian(D.f_size, seed=961)
    yo, _ = ops.mobius_mdagm(x, 0.05)
    assert rel(D.MatPcDagMatPc(x, prec=A.SINGLE)[0], yo) < 8e-7
    assert rel(D.MatPcDagMatPc(x, prec=A.DOUBLE)[0], yo) < 4e-15


@pytest.mark.parametrize("prec", [A.DOUBLE, A.SINGLE, A.HALF])
def test_named_kernels_are_dense(oracle, prec):
    """cpsgpu_set_mix_impl 2 and 3 run the dense kernels on matrices that have the recurrence's form, in the standalone
    mixings and the hop's epilogue: their bits are each other's and not the default's, and the default is no further
    from the oracle (the roundings of one side may exceed the other's by chance: 1.3)"""
    D, ops = _op(oracle, (4, 4, 4, 4), 12, 1.45, 0.45)
    x = gen_gaussian(D.f_size, seed=962)

    def fields():
        return [D.M5inv(x, 0, prec=prec), D.M5inv(x, 1, prec=prec), D.Dslash4(x, 0, 1, prec=prec), D.MatPcDagMatPc(x, prec=prec)[0]]

    default = fields()
    D.set_mix_impl(D.MIX_SHARED)
    shared = fields()
    D.set_mix_impl(D.MIX_REG)
    ref = [ops.mobius_m5inv(x, 0.05, 0), ops.mobius_m5inv(x, 0.05, 1), ops.mobius_dslash_4(x, 0.05, 0, 1),
           ops.mobius_mdagm(x, 0.05)[0]]
    for a, b, c, r in zip(fields(), shared, default, ref):
        np.testing.assert_array_equal(a, b)
        assert rel(c, r) <= 1.3 * rel(b, r)
    assert any((b != c).any() for b, c in zip(shared, default))
    D.set_mix_impl(D.MIX_DEFAULT)
    for a, c in zip(fields(), default):
        np.testing.assert_array_equal(a, c)
