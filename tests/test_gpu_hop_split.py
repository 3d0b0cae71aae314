"""The small launches' hop (four threads per site, hop.cuh hop_split_kernel)
against the one-thread hop it stands in for: the same bits for every field,
for Wilson and DWF (odd and even Ls), every precision and link form, both
checkerboards and daggers, partial site blocks and several right-hand sides;
and the solves around it.  A shape set by the caller keeps the one-thread
hop, so setting one gives the other side of the comparison."""
import numpy as np
import pytest

from cps_veloc_b200 import _abi as A
from cps_veloc_b200.dirac import DiracOpDwf, DiracOpWilson, Lattice, gen_gauge, gen_gaussian, solve_batch
from helpers import OracleOps, rel

pytestmark = pytest.mark.gpu

REALS = {A.DOUBLE: (None,), A.SINGLE: (12, 18), A.HALF: (12, 18, 112, 118)}


def _op(kind, L, ls):
    A.check(A.lib().cpsgpu_finalize())  # no shape set by another test
    u = gen_gauge(L, seed=971)
    lat = Lattice(L, (1, -1, 1, -1))
    lat.import_gauge(u)
    return u, lat, DiracOpWilson(lat, mass=0.1) if kind == "wilson" else DiracOpDwf(lat, mass=0.05, ls=ls)


def _fields(D, x, prec):
    out = [D.Dslash(x, cb, dag, prec) for cb in (0, 1) for dag in (0, 1)]
    y, dot = D.MatPcDagMatPc(x, prec)
    return out + [D.MatPc(x, prec), D.MatPcDag(x, prec), y], dot


@pytest.mark.parametrize("prec", [A.DOUBLE, A.SINGLE, A.HALF])
@pytest.mark.parametrize("kind,L,ls", [("wilson", (2, 2, 2, 2), 1), ("wilson", (6, 4, 2, 6), 1),
                                       ("wilson", (8, 8, 8, 8), 1), ("dwf", (2, 2, 2, 4), 2), ("dwf", (4, 2, 6, 2), 5),
                                       ("dwf", (4, 4, 4, 4), 8), ("dwf", (6, 6, 4, 4), 7)])
def test_same_bits_as_one_thread(oracle, kind, L, ls, prec):
    u, lat, D = _op(kind, L, ls)
    x = gen_gaussian(D.f_size, seed=972)
    for reals in REALS[prec]:
        if reals:
            lat.set_link_reals(prec, reals)
        A.check(A.lib().cpsgpu_finalize())
        split, dot = _fields(D, x, prec)
        D.set_hop_shape(prec, 32, 1)
        one, dot1 = _fields(D, x, prec)
        for a, b in zip(split, one):
            np.testing.assert_array_equal(a, b)
        assert dot == pytest.approx(dot1, rel=1e-12 if prec == A.DOUBLE else 1e-6)
    ops = OracleOps(oracle, L, u, ls=ls, bc=(1, -1, 1, -1))
    ref = ops.wilson_dslash(x, 1, 0) if kind == "wilson" else ops.dwf_dslash(x, 0.05, 1, 0)
    assert rel(split[2], ref) < {A.DOUBLE: 1e-13, A.SINGLE: 2e-6, A.HALF: 5e-3}[prec]
    A.check(A.lib().cpsgpu_finalize())


@pytest.mark.parametrize("prec", [A.DOUBLE, A.SINGLE, A.HALF])
@pytest.mark.parametrize("shift", [0.0, 0.3])
def test_solves(prec, shift):
    """CG (its residual and solution epilogues, with a shift too) and a batch
    whose sources finish at different iterations"""
    _, _, D = _op("dwf", (4, 4, 4, 4), 6)
    srcs = [gen_gaussian(D.f_size, seed=973 + k) for k in range(3)]
    srcs[1] = D.MatPcDagMatPc(srcs[1])[0]
    x = np.zeros(D.f_size)
    r = D.InvCg(x, srcs[0], stop_rsd=1e-10, shift=shift, precision=prec)
    assert r.status == A.CONVERGED and r.true_res <= 1e-10
    y, _ = D.MatPcDagMatPc(x)
    assert rel(y + shift * x, srcs[0]) <= 1.01e-10
    sols = [np.zeros(D.f_size) for _ in srcs]
    for b, s, q in zip(srcs, sols, D.InvCgMulti(sols, srcs, stop_rsd=1e-10, precision=prec)):
        assert q.status == A.CONVERGED and rel(D.MatPcDagMatPc(s)[0], b) <= 1.01e-10


@pytest.mark.parametrize("count", [2, 3])
def test_batch_counts_all_its_sites(count):
    """Independent solves in one launch: the rule goes by the sites of all of them.  Two FP64 systems of 4096 sites are
    few enough for four threads per site, three are not: those give the bits of the one-thread hop of the same shape
    (the four-threads kernel sums its dot products in another order)."""
    res = []
    for forced in (False, True):
        A.check(A.lib().cpsgpu_finalize())
        items = []
        for k in range(count):
            lat = Lattice((4, 4, 8, 8), (1, 1, 1, -1))
            lat.import_gauge(gen_gauge((4, 4, 8, 8), seed=976 + k))
            D = DiracOpDwf(lat, mass=0.05, ls=8)
            if forced:
                D.set_hop_shape(A.DOUBLE, *D.hop_shape(A.DOUBLE))
            items.append((D, np.zeros(D.f_size), gen_gaussian(D.f_size, seed=980 + k)))
        for r in solve_batch(items, stop_rsd=1e-10, precision=A.DOUBLE):
            assert r.status == A.CONVERGED and r.true_res <= 1e-10
        res.append([sol for _, sol, _ in items])
    assert all((a == b).all() for a, b in zip(*res)) == (count == 3)
    A.check(A.lib().cpsgpu_finalize())


@pytest.mark.parametrize("prec", [A.DOUBLE, A.SINGLE, A.HALF])
@pytest.mark.parametrize("ls", [2, 6, 10, 12, 14])
def test_default_shape_of_larger_launches(ls, prec):
    """above the rule's bound, with a partial last block of sites: the default shape's fields against one slice and 32
    sites per block"""
    L = {2: (10, 10, 10, 18), 6: (10, 6, 10, 14)}.get(ls, (10, 6, 6, 10))
    u, lat, D = _op("dwf", L, ls)
    x = gen_gaussian(D.f_size, seed=985)
    default, dot = _fields(D, x, prec)
    D.set_hop_shape(prec, 32, 1)
    one, dot1 = _fields(D, x, prec)
    for a, b in zip(default, one):
        np.testing.assert_array_equal(a, b)
    assert dot == pytest.approx(dot1, rel=1e-12)
    A.check(A.lib().cpsgpu_finalize())
