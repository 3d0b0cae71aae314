"""The multishift CG's deferred updates (shifts s > 0 applied once per chunk of
8 iterations, multishift.cu ms_flush_kernel) against the oracle: runs capped
at the chunk's edges, shifts that converge inside a chunk, every solution
type, one and two shifts (the per-iteration updates) beside many."""
import numpy as np
import pytest

from cps_veloc_b200 import _abi as A
from cps_veloc_b200.dirac import DiracOpDwf, DiracOpWilson, Lattice, gen_gauge, gen_gaussian
from helpers import OracleOps, rel

pytestmark = pytest.mark.gpu

L = (4, 2, 6, 2)  # 48 sites: the last block of the elementwise passes is partial


def _op(oracle, kind):
    u = gen_gauge(L, seed=911)
    lat = Lattice(L)
    lat.import_gauge(u)
    if kind == "wilson":
        D = DiracOpWilson(lat, mass=1 / (2 * 0.12) - 4)
        return D, OracleOps(oracle, L, u, ls=1), dict(kappa=D.kappa)
    return DiracOpDwf(lat, mass=0.1, ls=5), OracleOps(oracle, L, u, ls=5), dict(mass=0.1)


@pytest.mark.parametrize("cap", [1, 2, 7, 8, 9, 16, 17])
@pytest.mark.parametrize("kind,n,type_", [("wilson", 1, 1), ("wilson", 2, 1), ("wilson", 3, 1), ("dwf", 9, 1),
                                          ("wilson", 9, 0), ("dwf", 4, 0), ("dwf", 3, 2)])
def test_capped_runs(oracle, kind, n, type_, cap):
    """The iterates themselves at 1e-10: a capped run of k <= 17 iterations
    differs from the oracle by the FP64 roundings of its sums (1e-16 each)
    times the growth of the CG recurrence, below 1e-12 here."""
    D, ops, kw = _op(oracle, kind)
    chi = gen_gaussian(ops.n, seed=912)
    shifts = list(np.logspace(-2, 1, n)) if n > 1 else [0.05]
    alpha = [(-1.0) ** k / (1 + k) for k in range(n)]
    start = [gen_gaussian(ops.n, seed=920 + k) if type_ != 1 else np.zeros(ops.n) for k in range(1 if type_ == 0 else n)]
    psi_o, ko, _ = ops.minvcg(kind, chi, shifts, [1e-13] * n, type=type_, alpha=alpha, max_num_iter=cap, psi0=start, **kw)
    psi = [x.copy() for x in start]
    k = D.MInvCG(psi, chi, float(chi @ chi), shifts, np.full(n, 1e-13), type=type_, alpha=alpha, max_num_iter=cap)
    assert k == ko
    for a, b in zip(psi, psi_o):
        assert rel(a, b) < 1e-10


def test_shifts_that_stop_inside_a_chunk(oracle):
    """Widely spread shifts and stopping residuals: each shift stops at an
    iteration of its own and is left alone from then on."""
    D, ops, kw = _op(oracle, "dwf")
    chi = gen_gaussian(ops.n, seed=913)
    shifts = list(np.logspace(-3, 2, 11))
    rsd = [10.0 ** -(4 + k % 7) for k in range(11)]
    psi_o, ko, rso = ops.minvcg("dwf", chi, shifts, rsd, type=1, **kw)
    psi = [np.zeros(ops.n) for _ in shifts]
    rs = np.array(rsd)
    k = D.MInvCG(psi, chi, float(chi @ chi), shifts, rs, type=A.MS_MULTI)
    assert abs(k - ko) <= 1
    for s in range(11):
        # the same iterate up to rounding, or one iteration apart where the residual sits at its bound
        assert rel(psi[s], psi_o[s]) < 10 * rsd[s]
        assert rs[s] == pytest.approx(rso[s], rel=1e-2)


@pytest.mark.parametrize("n", [2, 3, 8])
def test_fp32_recurrences_then_refinement(oracle, n):
    D, ops, kw = _op(oracle, "dwf")
    chi = gen_gaussian(ops.n, seed=914)
    shifts = list(np.logspace(-2, 1, n))
    psi = [np.zeros(ops.n) for _ in shifts]
    D.MInvCG(psi, chi, float(chi @ chi), shifts, np.full(n, 1e-10), type=A.MS_MULTI, precision=A.SINGLE)
    for s, sh in enumerate(shifts):
        y, _ = ops.dwf_mdagm(psi[s], 0.1)
        assert rel(y + sh * psi[s], chi) <= 1.01e-10
