"""The multishift CG's captured graphs (multishift.cu) hold the addresses of
its fields, residuals and partials.  A call that makes any of those anew, or a
solve that moves a buffer of the lattice, has to leave no graph behind that
still points at the old ones: the precisions in turn on one operator, other
numbers of shifts and solution types between, larger solves on the lattice
between, and fields made and filled where freed ones were.  Each repeated call
gives the first one's bits."""
import ctypes as C

import numpy as np
import pytest

from cps_veloc_b200 import _abi as A
from cps_veloc_b200.dirac import DiracOpDwf, DiracOpMobius, DiracOpWilson, Lattice, gen_gauge, gen_gaussian

pytestmark = pytest.mark.gpu

L = (4, 4, 6, 4)


def _op(kind, lat):
    return {"wilson": lambda: DiracOpWilson(lat, mass=0.1), "dwf": lambda: DiracOpDwf(lat, mass=0.1, ls=6),
            "mobius": lambda: DiracOpMobius(lat, mass=0.1, ls=6, b=1.5, c=0.5)}[kind]()


def _call(D, chi, prec, n=5, type_=A.MS_MULTI):
    psi = [np.zeros(D.f_size) for _ in range(1 if type_ == A.MS_SINGLE else n)]
    rsd = np.full(n, 1e-9)
    it = D.MInvCG(psi, chi, float(chi @ chi), list(np.logspace(-2, 1, n)), rsd, type=type_, alpha=[1.0 / (1 + k) for k in range(n)],
                  precision=prec)
    return [it, rsd.copy(), *psi]


class _Occupied:
    """FP64 fields of ones, in the memory that the call before gave back"""

    def __init__(self, D, count):
        self.h = []
        one = np.ones(D.f_size)
        for _ in range(count):
            f = C.c_void_p()
            A.check(A.lib().cpsgpu_field_create(D._h, A.DOUBLE, 1, C.byref(f)))
            A.check(A.lib().cpsgpu_field_upload(f, A.dptr(one)))
            self.h.append(f)
        self.n, self.one = D.f_size, one

    def close(self):
        out = np.empty(self.n)
        for f in self.h:
            A.check(A.lib().cpsgpu_field_download(f, A.dptr(out)))
            np.testing.assert_array_equal(out, self.one)  # no solve wrote here
            A.lib().cpsgpu_field_destroy(f)


@pytest.mark.parametrize("kind", ["wilson", "dwf", "mobius"])
def test_calls_in_turn_on_one_operator(kind):
    lat = Lattice(L, (1, 1, 1, -1))
    lat.import_gauge(gen_gauge(L, seed=931))
    D = _op(kind, lat)
    chi = gen_gaussian(D.f_size, seed=932)
    kinds = [(A.DOUBLE, 5, A.MS_MULTI), (A.SINGLE, 5, A.MS_MULTI), (A.DOUBLE, 9, A.MS_SINGLE), (A.DOUBLE, 5, A.MS_MULTI),
             (A.SINGLE, 3, A.MS_MULTI), (A.DOUBLE, 2, A.MS_MULTI)]
    first = [_call(_op(kind, lat), chi, *k) for k in kinds]  # each on an operator of its own
    for _ in range(2):
        for k, want in zip(kinds, first):
            busy = _Occupied(D, 5)
            got = _call(D, chi, *k)
            busy.close()
            for a, b in zip(got, want):
                np.testing.assert_array_equal(a, b)


def test_larger_solves_on_the_lattice_between():
    lat = Lattice(L, (1, 1, 1, -1))
    lat.import_gauge(gen_gauge(L, seed=933))
    D = _op("dwf", lat)
    chi = gen_gaussian(D.f_size, seed=934)
    want = _call(D, chi, A.DOUBLE)
    for n in (4, 16, 48):
        srcs = [gen_gaussian(D.f_size, seed=935 + k) for k in range(n)]
        D.InvCgMulti([np.zeros(D.f_size) for _ in srcs], srcs, stop_rsd=1e-4, precision=A.DOUBLE)
        busy = _Occupied(D, 4)
        got = _call(D, chi, A.DOUBLE)
        busy.close()
        for a, b in zip(got, want):
            np.testing.assert_array_equal(a, b)


def test_operators_of_one_lattice_share_the_ring():
    """Operators of different Ls (the ring grows and moves), in turn, each call with the bits of its first; a second
    operator takes no ring of its own, and the ring goes with the last of them."""
    import torch

    lat = Lattice((8, 8, 8, 16), (1, 1, 1, -1))
    lat.import_gauge(gen_gauge((8, 8, 8, 16), seed=938))

    def free():
        return torch.cuda.mem_get_info()[0]

    chis = {ls: gen_gaussian(24 * lat.vol // 2 * ls, seed=939 + ls) for ls in (8, 12, 4)}
    ops = {ls: DiracOpDwf(lat, mass=0.1, ls=ls) for ls in chis}
    first = {ls: _call(D, chis[ls], A.DOUBLE) for ls, D in ops.items()}
    for ls in (4, 12, 8, 12, 4):
        for a, b in zip(_call(ops[ls], chis[ls], A.DOUBLE), first[ls]):
            np.testing.assert_array_equal(a, b)
    for D in ops.values():
        D.close()
    ring = 7 * 192 * lat.vol // 2 * 12
    start = free()
    A1, B1 = DiracOpDwf(lat, mass=0.1, ls=12), DiracOpDwf(lat, mass=0.2, ls=12)
    _call(A1, chis[12], A.DOUBLE)
    one = start - free()
    _call(B1, chis[12], A.DOUBLE)
    two = start - free() - one
    assert one - two > 0.9 * ring  # 66 MB
    A1.close()
    B1.close()
    assert start - free() < 0.1 * ring
