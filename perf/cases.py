"""Performance cases of the fermion-solve path: what is timed, on which inputs, and what the answers should be.

Every case is one call that a CPS measurement or an HMC/RHMC run makes through the public interface
(cps_veloc_b200.dirac, cps_veloc_b200.dd and the C ABI under them), on seeded SU(3) links U = exp(i 0.3 H) and
Gaussian sources, periodic in space and antiperiodic in time.  The operators run with the launch shapes a program
gets without asking for any (the CPS-side shim does not call the autotuner; the autotuner's table is shared by the
whole process, so one tuned case would change the others).

    mdagm       DiracOp::MatPcDagMatPc on host vectors: one operator application, as CPS calls it per iteration
    cg          DiracOp::InvCg to a relative residual, zero guess: on host vectors, or on fields kept on the device
                with the solution read back
    multi       InvCg of several right-hand sides of one operator (the spin-colour components of a propagator)
    multishift  DiracOp::MInvCG: the rational approximations of RHMC; every solution (the force) or their weighted
                sum (heat bath, action)
    batch       independent solves of different masses in one call (mass scans, small volumes)
    force       RHMC_EvolveMomFforce: the fermion force of the poles added to the momenta

exact() restates the operators in complex128 torch from their definitions (wilson_dslash.C:64-515,
dwf_dslash_4.C:68-154, dwf_dslash_5_plus_omp.C:115-271, zmobius_m-sym2.h, f_dwf_base_force.C:41-300).
"""
import ctypes
import math

import numpy as np
import torch

from cps_veloc_b200 import _abi as A
from cps_veloc_b200 import dd
from cps_veloc_b200.dirac import DiracOpDwf, DiracOpMobius, DiracOpWilson, Lattice, solve_batch

M5 = 1.8
MOB_B, MOB_C = 1.5, 0.5
PREC = {"double": A.DOUBLE, "single": A.SINGLE, "half": A.HALF}
# iterations per decade of the residual of these systems (measured: DWF m_f 0.01, Mobius m_f 0.005, Wilson kappa 0.125)
ITERS = {"wilson": 6.6, "dwf": 19.6, "mobius": 51.0}
MASS = {"wilson": 1 / (2 * 0.125) - 4, "dwf": 0.01, "mobius": 0.005}


def _case(name, op, kind, lattice, ls=1, prec="double", stop=0.0, **more):
    x, y, z, t = lattice
    return {"name": name, "op": op, "kind": kind, "x": x, "y": y, "z": z, "t": t, "ls": ls, "prec": prec, "stop": stop,
            **more}


def listed():
    return [
        # the smallest calls, where launches and latency are all there is: the operator on one small vector, and the
        # reference's own test system (f_wilson_inv: 4^3x8-sized, stop 1e-8)
        _case("mdagm_dwf_8x8_ls8", "mdagm", "dwf", (8, 8, 8, 8), 8),
        _case("cg_wilson_4x8_double", "cg", "wilson", (4, 4, 4, 8), 1, "double", 1e-8, device=False),
        # many small systems at once
        _case("batch_dwf_8x16_ls8", "batch", "dwf", (8, 8, 8, 16), 8, "single", 1e-10, count=8),
        # a propagator's 12 spin-colour sources on a small volume
        _case("multi12_dwf_8x16_ls8", "multi", "dwf", (8, 8, 8, 16), 8, "single", 1e-8, count=12),
        # ragged extents: no power of two, blocks of sites that do not divide the checkerboard
        _case("cg_mobius_ragged_single", "cg", "mobius", (10, 6, 14, 18), 10, "single", 1e-8, device=False),
        _case("cg_dwf_ragged_half", "cg", "dwf", (12, 14, 20, 22), 12, "half", 1e-10, device=True),
        # the benchmark's system in the default precision (what the shim solves with) and with the FP32 inner solve
        _case("cg_dwf_16x32_ls16_double", "cg", "dwf", (16, 16, 16, 32), 16, "double", 1e-10, device=True),
        _case("cg_dwf_16x32_ls16_single", "cg", "dwf", (16, 16, 16, 32), 16, "single", 1e-10, device=True),
        # the largest: the Mobius system with the FP16 inner solve, to the relaxed residual of all-mode averaging
        _case("cg_mobius_24x64_ls12_half", "cg", "mobius", (24, 24, 24, 64), 12, "half", 1e-5, device=True),
        # RHMC: the force's separate solutions, and the action's weighted sum
        _case("multishift_dwf_12x24_ls8", "multishift", "dwf", (12, 12, 12, 24), 8, "double", 1e-8, count=10, summed=False),
        _case("multishift_wilson_24x48", "multishift", "wilson", (24, 24, 24, 48), 1, "double", 1e-10, count=16,
              summed=True),
        # and the force of its poles
        _case("force_dwf_16x16_ls8", "force", "dwf", (16, 16, 16, 16), 8, "double", 0.0, count=4),
    ]


def draw(rng):
    """Another call of the same kinds: volumes over their logarithm from 4^3x4 up, any even extents, odd Ls among the
    fifth extents, every precision an entry point takes."""
    largest = max(_cost(c) for c in listed())
    while True:
        op = rng.choice(["mdagm", "cg", "cg", "cg", "multi", "multishift", "batch", "force"])
        kind = rng.choice(["wilson", "dwf", "mobius"])
        if op in ("multi", "batch", "force") and kind == "mobius":
            kind = "dwf"
        if op == "batch":
            kind = "dwf"
        top = {"mdagm": 24, "cg": 24, "multi": 12, "multishift": 20, "batch": 8, "force": 16}[op]
        ext = [2 * max(2, round(math.exp(rng.uniform(math.log(4), math.log(top))) / 2)) for _ in range(3)]
        ext.append(2 * max(2, round(math.exp(rng.uniform(math.log(4), math.log(2 * top))) / 2)))
        ls = 1 if kind == "wilson" else rng.choice([4, 6, 7, 8, 10, 12, 16]) if kind == "dwf" else rng.choice([6, 8, 9, 10, 12, 16])
        prec = rng.choice(["double", "single", "half"]) if op in ("mdagm", "cg") else \
            "single" if op in ("multi", "batch") else "double"
        c = _case("", op, kind, ext, ls, prec, rng.choice([1e-5, 1e-8, 1e-10]) if op not in ("mdagm", "force") else 0.0)
        if op == "cg":
            c["device"] = rng.random() < 0.5
        if op == "multi":
            c["count"] = rng.choice([2, 3, 8, 12])
        if op == "batch":
            c["count"] = rng.choice([2, 3, 5, 8])
        if op == "multishift":
            c["count"], c["summed"] = rng.choice([4, 7, 10, 16]), rng.random() < 0.5
        if op == "force":
            c["count"] = rng.choice([1, 2, 5])
        del c["name"]
        if _cost(c) <= largest:
            return c


# ---------------------------------------------------------------- sizes
def _lattice(case):
    return tuple(case[k] for k in "xyzt")


def _sites(case):
    """5D sites of one preconditioned vector"""
    return case["x"] * case["y"] * case["z"] * case["t"] // 2 * case["ls"]


def _iters(case):
    return max(1.0, ITERS[case["kind"]] * -math.log10(case["stop"])) if case["stop"] else 1.0


def _shifts(n):
    return np.logspace(-4, 1, n)


def _applications(case):
    """MatPcDagMatPc applications of one pass, on one vector each"""
    n = {"mdagm": 1, "force": 1}.get(case["op"]) or _iters(case)
    return n * (case.get("count", 1) if case["op"] in ("multi", "batch", "force") else 1)


def _cost(case):
    n = case.get("count", 1) if case["op"] == "multishift" else 0
    return _sites(case) * (_applications(case) * 9 + n * _iters(case)) + 1


def work(case):
    """Bytes: the vectors that go in and out once at FP64, and for each iteration of a solve what one CG step has to
    read and write in its working precision: the operator's input and output, the residual, the direction and the
    solution read and written once, and the links twice (MatPc and its adjoint).  Flops: 1320 per site and hop (the
    reference's count, wilson_dslash.C:515), 4 hops per MatPcDagMatPc, and the Ls x Ls mixings of Mobius."""
    sites, v4, ls = _sites(case), case["x"] * case["y"] * case["z"] * case["t"], case["ls"]
    real = {"double": 8.0, "single": 4.0, "half": 52 / 24}[case["prec"]]
    link = {"double": 96.0, "single": 48.0, "half": 24.0}[case["prec"]]
    vec, links = 24 * real * sites, 4 * v4 * link
    n = case.get("count", 1)
    hop = 4 * 1320.0 * sites * (1 if case["kind"] != "mobius" else 1 + 4 * 24 * ls / (4 * 1320.0) * 2)
    op = case["op"]
    if op == "mdagm":
        return {"bytes": 2 * 192.0 * sites + links, "flops": hop}
    if op == "force":
        return {"bytes": n * 192.0 * sites + 3 * 4 * v4 * 144.0, "flops": n * (hop + 4 * 2.0 * sites * 2 * 2 * 72)}
    it = _iters(case)
    if op == "multishift":
        # per shift: its direction and its share of the solution
        outs = 1 if case["summed"] else n
        return {"bytes": it * (vec * (4 + 2 * (n - 1) + 2 * outs) + 2 * links) + 192.0 * sites * (1 + outs),
                "flops": it * (hop + n * 24 * 5.0 * sites)}
    systems = n if op in ("multi", "batch") else 1
    fields = 1 if op == "multi" else systems
    return {"bytes": it * (systems * 6 * vec + fields * 2 * links) + systems * 2 * 192.0 * sites,
            "flops": it * systems * (hop + 24 * 10.0 * sites)}


# ---------------------------------------------------------------- inputs
def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _links(case, seed):
    """[parity][cb site][mu][row][col] complex128: exp(i 0.3 H), row 2 = conj(row 0 x row 1)"""
    g = torch.Generator(device=_device())
    g.manual_seed(1000003 * seed + 17)
    n = case["x"] * case["y"] * case["z"] * case["t"] * 4
    a = torch.randn(n, 3, 3, 2, generator=g, device=_device(), dtype=torch.float64)
    a = torch.view_as_complex(a)
    h = (a + a.conj().transpose(1, 2)) / 2
    h = h - torch.eye(3, device=h.device) * (h.diagonal(dim1=1, dim2=2).sum(1) / 3)[:, None, None]
    x = 0.075j * h  # exp(x)^4
    e = torch.eye(3, device=h.device, dtype=x.dtype).expand(n, 3, 3)
    t = e
    for k in range(1, 13):
        t = _mm(t, x) / k
        e = e + t
    e = _mm(e, e)
    e = _mm(e, e)
    r0 = e[:, 0] / e[:, 0].abs().square().sum(1).sqrt()[:, None]
    r1 = e[:, 1] - r0 * (r0.conj() * e[:, 1]).sum(1)[:, None]
    r1 = r1 / r1.abs().square().sum(1).sqrt()[:, None]
    return torch.stack([r0, r1, torch.linalg.cross(r0, r1).conj()], 1).reshape(2, n // 8, 4, 3, 3)


def _mm(a, b):
    return (a[:, :, :, None] * b[:, None, :, :]).sum(2)


def _wilson_order(u):
    """the host array import_gauge takes: [parity][cb site][mu][col][row][re, im]"""
    return torch.view_as_real(u.transpose(3, 4).contiguous()).reshape(-1).cpu().numpy()


def _vectors(case, seed, count):
    """count Gaussian vectors in CPS order (one preconditioned checkerboard), float64 on the device"""
    g = torch.Generator(device=_device())
    g.manual_seed(1000003 * seed + 29)
    return torch.randn(count, 24 * _sites(case), generator=g, device=_device(), dtype=torch.float64)


def _masses(case):
    n = case["count"]
    return [0.01 * 10 ** (k / max(1, n - 1)) for k in range(n)]


def _operator(case, lat, mass=None):
    m = MASS[case["kind"]] if mass is None else mass
    if case["kind"] == "wilson":
        return DiracOpWilson(lat, mass=m)
    if case["kind"] == "dwf":
        return DiracOpDwf(lat, mass=m, ls=case["ls"], m5=M5)
    return DiracOpMobius(lat, mass=m, ls=case["ls"], m5=M5, b=MOB_B, c=MOB_C)


def _poles(case):
    return np.array([0.2 + 0.3 * k for k in range(case["count"])])


DT = 0.01


def _pinned(n):
    """a float64 host vector in page-locked memory, as a program that reads solutions back keeps"""
    return torch.empty(n, dtype=torch.float64, pin_memory=True).numpy()


def prepare(case, seed):
    op = case["op"]
    lat = Lattice(_lattice(case), bc=(1, 1, 1, -1))
    lat.import_gauge(_wilson_order(_links(case, seed)))
    st = {"case": case, "lat": lat}
    n = 24 * _sites(case)
    if op == "batch":
        st["ops"] = [_operator(case, lat, m) for m in _masses(case)]
        st["src"] = list(_vectors(case, seed, case["count"]).cpu().numpy())
        st["sol"] = [np.zeros(n) for _ in st["src"]]
        return st
    D = st["D"] = _operator(case, lat)
    if op == "mdagm":
        st["in"] = _vectors(case, seed, 1)[0].cpu().numpy()
    elif op == "cg":
        src = _vectors(case, seed, 1)[0].cpu().numpy()
        if case["device"]:
            st["src"], st["sol"] = dd.DeviceField(D), dd.DeviceField(D)
            st["src"].upload(src)
            st["host"] = _pinned(n)
        else:
            st["src"], st["sol"] = src, np.zeros(n)
    elif op == "multi":
        st["src"] = list(_vectors(case, seed, case["count"]).cpu().numpy())
        st["sol"] = [np.zeros(n) for _ in st["src"]]
    elif op == "multishift":
        st["src"] = _vectors(case, seed, 1)[0].cpu().numpy()
        st["norm"] = float(st["src"] @ st["src"])
        st["sol"] = [np.zeros(n) for _ in range(1 if case["summed"] else case["count"])]
    elif op == "force":
        # solutions of the poles and momenta as the integrator holds them
        st["sol"] = list(_vectors(case, seed, case["count"]).cpu().numpy())
        st["mom"] = _momenta(case, seed)
    return st


def _momenta(case, seed):
    """traceless antihermitian momenta, CANONICAL [site][mu][row][col][re, im]"""
    g = torch.Generator(device=_device())
    g.manual_seed(1000003 * seed + 31)
    n = case["x"] * case["y"] * case["z"] * case["t"] * 4
    a = torch.view_as_complex(torch.randn(n, 3, 3, 2, generator=g, device=_device(), dtype=torch.float64))
    return torch.view_as_real(_antiherm(a)).reshape(-1).cpu().numpy()


def _antiherm(f):
    a = (f - f.conj().transpose(-1, -2)) / 2
    tr = a.diagonal(dim1=-1, dim2=-2).sum(-1) / 3
    return a - torch.eye(3, device=a.device) * tr[..., None, None]


# ---------------------------------------------------------------- one pass
def run(st):
    case = st["case"]
    op, stop = case["op"], case["stop"]
    if op == "mdagm":
        out, dot = st["D"].MatPcDagMatPc(st["in"], PREC[case["prec"]])
        return {"out": out, "dot": dot}
    if op == "cg":
        D = st["D"]
        if not case["device"]:
            st["sol"].fill(0.0)
            D.InvCg(st["sol"], st["src"], stop_rsd=stop, precision=PREC[case["prec"]])
            return st["sol"]
        lib, sol, src, host = A.lib(), st["sol"], st["src"], st["host"]
        A.check(lib.cpsgpu_field_axpby(sol._h, -1.0, src._h, src._h))  # zero guess
        arg, res = A.CgArg(), A.CgResult()
        lib.cpsgpu_cg_arg_default(ctypes.byref(arg))
        arg.stop_rsd, arg.precision = stop, PREC[case["prec"]]
        A.check(lib.cpsgpu_invcg_field(D._h, sol._h, src._h, ctypes.byref(arg), ctypes.byref(res)))
        A.check(lib.cpsgpu_field_download(sol._h, A.dptr(host)))
        return host
    if op == "multi":
        for s in st["sol"]:
            s.fill(0.0)
        st["D"].InvCgMulti(st["sol"], st["src"], stop_rsd=stop, precision=PREC[case["prec"]])
        return st["sol"]
    if op == "batch":
        for s in st["sol"]:
            s.fill(0.0)
        solve_batch(list(zip(st["ops"], st["sol"], st["src"])), stop_rsd=stop, precision=PREC[case["prec"]])
        return st["sol"]
    if op == "multishift":
        sh = _shifts(case["count"])
        if case["summed"]:
            st["sol"][0].fill(0.0)
        st["D"].MInvCG(st["sol"], st["src"], st["norm"], sh, np.full(len(sh), stop),
                       type=A.MS_SINGLE if case["summed"] else A.MS_MULTI, alpha=_weights(case), precision=PREC[case["prec"]])
        return st["sol"]
    st["D"].RHMC_EvolveMomFforce(st["mom"], st["sol"], _poles(case), DT)
    return st["mom"]


def _weights(case):
    return 1.0 / (1.0 + np.arange(case["count"]))


# ---------------------------------------------------------------- what is compared
def tolerance(case):
    """One operator application: the storage's rounding (FP64 sums; FP32 storage and arithmetic; FP16 storage of every
    intermediate field).  A solve: any correct CG stops at a residual below stop, whose error in the solution is up to
    the condition of the system larger: against exact() 5 times stop (Wilson), 50 (DWF) and 25 (Mobius) are seen."""
    if case["op"] in ("mdagm", "force"):
        return {"rel": {"double": 2e-15, "single": 2e-6, "half": 4e-3}[case["prec"]]}
    return {"rel": {"wilson": 20, "dwf": 200, "mobius": 100}[case["kind"]] * case["stop"]}


# ---------------------------------------------------------------- 64-bit restatement
# gamma_mu row r: factor * component column (wilson_dslash.C:64-128); gamma_5 = diag(1, 1, -1, -1)
_G_COL = [[3, 2, 1, 0], [3, 2, 1, 0], [2, 3, 0, 1], [2, 3, 0, 1]]
_G_FAC = [[1j, 1j, -1j, -1j], [-1, 1, 1, -1], [1j, -1j, -1j, 1j], [1, 1, 1, 1]]


class _Exact:
    """The operators on [slice][cb site][spin][colour] complex128 fields."""

    def __init__(self, case, seed, mass=None):
        self.case, self.ls, self.kind = case, case["ls"], case["kind"]
        self.L = _lattice(case)
        self.mass = MASS[self.kind] if mass is None else mass
        self.u = _links(case, seed)
        self.fwd, self.bwd, self.lex = [], [], []
        lx, ly, lz, lt = self.L
        dev = self.u.device
        i = torch.arange(lx * ly * lz * lt // 2, device=dev)
        for p in (0, 1):
            r = i // (lx // 2)
            y, z, t = r % ly, (r // ly) % lz, r // (ly * lz)
            x = 2 * (i % (lx // 2)) + ((y + z + t + p) & 1)
            c = [x, y, z, t]
            self.lex.append(x + lx * (y + ly * (z + lz * t)))
            rows = []
            for step in (1, -1):
                row = []
                for mu in range(4):
                    d = list(c)
                    d[mu] = (c[mu] + step) % self.L[mu]
                    wrap = (c[mu] + step != d[mu]) & (mu == 3)
                    j = d[0] // 2 + (lx // 2) * (d[1] + ly * (d[2] + lz * d[3]))
                    row.append((j, torch.where(wrap, -1.0, 1.0).to(torch.float64)))
                rows.append(row)
            self.fwd.append(rows[0])
            self.bwd.append(rows[1])
        if self.kind == "wilson":
            self.kappa = 1 / (2 * (self.mass + 4))
        elif self.kind == "dwf":
            self.kappa = 1 / (2 * (5 - M5))
        else:
            kb, kc = 1 / (2 * (MOB_B * (4 - M5) + 1)), 1 / (2 * (MOB_C * (4 - M5) - 1))
            self.kappa = kb
            b = self._mix(MOB_B, MOB_C)
            m5inv = [torch.linalg.inv(m) for m in self._mix(1.0, kb / kc)]
            self.P = [x @ y for x, y in zip(b, m5inv)]

    def _mix(self, b, c):
        """b + c (hop from s-1 on the upper half, from s+1 on the lower, -m at the walls)"""
        n = self.ls
        up = b * torch.eye(n, dtype=torch.float64)
        for s in range(n):
            up[s, s - 1] += c if s else -self.mass * c
        dn = up.flip(0, 1)
        return [m.to(self.u.device) for m in (up, dn)]

    def hop4(self, v, pin, dag):
        """the 4D hop of slices v, input parity pin"""
        po, sd = 1 - pin, -1 if dag else 1
        out = torch.zeros_like(v)
        for mu in range(4):
            for table, k, forward in ((self.fwd, -sd, True), (self.bwd, sd, False)):
                j, sign = table[po][mu]
                w = v[:, j]
                c, f = _G_COL[mu], _G_FAC[mu]
                h = torch.stack([w[:, :, r] + k * f[r] * w[:, :, c[r]] for r in (0, 1)], 2) * sign[None, :, None, None]
                m = self.u[po, :, mu] if forward else self.u[pin, j, mu].conj().transpose(1, 2)
                g = sum(m[None, :, None, :, b] * h[:, :, :, b, None] for b in range(3))
                out[:, :, :2] += g
                for r in (2, 3):
                    out[:, :, r] += k * f[r] * g[:, :, c[r]]
        return out

    def dslash(self, v, cb, dag):
        if self.kind != "dwf":
            return self.hop4(v, cb, dag)
        out = torch.empty_like(v)
        for q in (0, 1):
            if v[q::2].shape[0]:
                out[q::2] = self.hop4(v[q::2].contiguous(), (q + cb) % 2, dag)
        w = torch.full((self.ls, 1, 1, 1), 2.0, dtype=torch.float64, device=v.device)
        wb, wa = w.clone(), w.clone()
        wb[0], wa[-1] = -2 * self.mass, -2 * self.mass
        lo, hi = (slice(2, 4), slice(0, 2)) if dag else (slice(0, 2), slice(2, 4))
        out[:, :, lo] += wb * v.roll(1, 0)[:, :, lo]
        out[:, :, hi] += wa * v.roll(-1, 0)[:, :, hi]
        return out

    def smix(self, mats, v):
        out = torch.empty_like(v)
        for half, m in enumerate(mats):
            sp = slice(2 * half, 2 * half + 2)
            out[:, :, sp] = (m.to(v.dtype) @ v[:, :, sp].reshape(self.ls, -1)).reshape(v[:, :, sp].shape)
        return out

    def matpc(self, v, dag=0):
        k2 = self.kappa ** 2
        if self.kind != "mobius":
            return v - k2 * self.dslash(self.dslash(v, 1, dag), 0, dag)
        if not dag:
            return v - k2 * self.hop4(self.smix(self.P, self.hop4(self.smix(self.P, v), 1, 0)), 0, 0)
        S = [m.T for m in self.P]
        return v - k2 * self.smix(S, self.hop4(self.smix(S, self.hop4(v, 1, 1)), 0, 1))

    def field(self, x):
        return torch.view_as_complex(x.reshape(self.ls, -1, 4, 3, 2).contiguous())

    def solve(self, b, shift=0.0, rsd=1e-13):
        x, r = torch.zeros_like(b), b.clone()
        p, rr = r.clone(), float(r.abs().square().sum())
        stop, seen = rr * rsd * rsd, 0
        while rr > stop and seen < 4000:
            m = self.matpc(p)
            q = self.matpc(m, 1) + shift * p
            a = rr / (float(m.abs().square().sum()) + shift * float(p.abs().square().sum()))
            x += a * p
            r -= a * q
            new = float(r.abs().square().sum())
            p = r + (new / rr) * p
            rr, seen = new, seen + 1
        return x

    def force(self, chi, mom, scale):
        """mom (CANONICAL, complex) += scale * traceless antihermitian part of U T"""
        psi = -self.kappa ** 2 * self.matpc(chi)
        v1 = [self.dslash(chi, 1, 0), chi]
        v2 = [self.dslash(psi, 1, 1), psi]  # [even half, odd half]

        def part(v, p):  # the half with 4D parity p in each slice
            s = torch.arange(self.ls, device=chi.device)
            return torch.where(((p + s) & 1 == 1)[:, None, None, None], v[1], v[0])

        def project(v, mu, k):
            return torch.stack([v[:, :, r] + k * _G_FAC[mu][r] * v[:, :, _G_COL[mu][r]] for r in (0, 1)], 2)

        for p in (0, 1):
            for mu in range(4):
                j, sign = self.fwd[p][mu]
                T = 0
                for k, a, w in ((-1, v1, v2), (1, v2, v1)):
                    ha, hw = project(part(a, 1 - p)[:, j], mu, k), project(part(w, p), mu, k)
                    T = T + sum((ha[s, :, r, :, None] * hw[s, :, r, None, :].conj()) for s in range(self.ls) for r in (0, 1))
                F = _antiherm(_mm(self.u[p, :, mu], T))
                mom[self.lex[p], mu] += scale * sign[:, None, None] * F


def _host(v):
    return torch.view_as_real(v.contiguous()).reshape(-1).cpu().numpy()


def exact(case, seed):
    op = case["op"]
    rounds = (case["count"] if op == "multishift" else 1) * _applications(case) * 1.4
    if _sites(case) * rounds > 5e8:
        return None
    if op == "mdagm":
        E = _Exact(case, seed)
        m = E.matpc(E.field(_vectors(case, seed, 1)[0]))
        return {"out": _host(E.matpc(m, 1)), "dot": float(m.abs().square().sum())}
    if op == "cg":
        E = _Exact(case, seed)
        return _host(E.solve(E.field(_vectors(case, seed, 1)[0])))
    if op == "multi":
        E = _Exact(case, seed)
        return [_host(E.solve(E.field(v))) for v in _vectors(case, seed, case["count"])]
    if op == "batch":
        out = []
        for m, v in zip(_masses(case), _vectors(case, seed, case["count"])):
            E = _Exact(case, seed, m)
            out.append(_host(E.solve(E.field(v))))
        return out
    if op == "multishift":
        E = _Exact(case, seed)
        b = E.field(_vectors(case, seed, 1)[0])
        x = [E.solve(b, float(s)) for s in _shifts(case["count"])]
        if case["summed"]:
            return [_host(sum(float(w) * v for w, v in zip(_weights(case), x)))]
        return [_host(v) for v in x]
    E = _Exact(case, seed)
    mom = torch.view_as_complex(torch.from_numpy(_momenta(case, seed)).to(E.u.device).reshape(-1, 4, 3, 3, 2))
    for v, a in zip(_vectors(case, seed, case["count"]), _poles(case)):
        E.force(E.field(v), mom, -2 * DT * float(a))
    return _host(mom)
