"""What this framework is timed on: the calls that a self-consistent-field
program makes of it, from one water molecule to (H2O)32 / cc-pVDZ.

Every case goes through the public Python entry points (``FockBuilder``,
``BatchBuilder``, ``FockJK``, ``rhf``) with the kernels a context picks by
itself.  Geometries, densities and energy weights come from the seed alone:
a new seed is another geometry (the same molecule sizes) and other densities.

The densities decay with the distance between their functions' atoms like
those of an insulator (diagonal occupations, random signs), so the screened
and mixed builds meet the spread of magnitudes they meet in an SCF.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from dalton_b200 import molecules, perfmodel
from dalton_b200.basis import build_basis
from dalton_b200.batch import BatchBuilder
from dalton_b200.fock import FockBuilder
from dalton_b200.grad import FockJK
from dalton_b200.scf import rhf

THRS = 1e-12

# Primitive shells up to which the plain torch evaluation at the end of this
# file stays under about 20 s.
EXACT_SHELLS = 76
EXACT_SHELLS_GRAD = 40


def listed():
    return [
        # The smallest call of an SCF: one molecule, one symmetric density,
        # matrices on the device.  Latency and launches.
        dict(name="fock_h2o_dz", kind="fock", mol="water", n=1, basis="cc-pVDZ"),
        # The same build as Dalton's HERFCK makes it: host matrices in and out.
        dict(name="host_h2o4_dz", kind="host", mol="water", n=4, basis="cc-pVDZ"),
        # One iteration of an incremental SCF: a density difference, Dalton's
        # density screen, quartets below the cutoff in FP32.
        dict(name="incr_h2o16_dz", kind="incr", mol="water", n=16, basis="cc-pVDZ", ifthrs=10, cutoff=1e-6),
        # The headline build: (H2O)32 / cc-pVDZ, all FP64.
        dict(name="fock_h2o32_dz", kind="fock", mol="water", n=32, basis="cc-pVDZ"),
        # A triple-zeta basis with f shells on an alkane.
        dict(name="fock_c5h12_tz", kind="fock", mol="alkane", n=5, basis="cc-pVTZ"),
        # Range-separated hybrid (the second, attenuated exchange pass) in
        # the segmented contracted 6-31G* basis.
        dict(name="rsh_h2o6_631gs", kind="rsh", mol="water", n=6, basis="6-31G*", mu=0.4),
        # Several densities at once, as a response solver hands them over:
        # general ones (two slots each), an antisymmetric one, J only, K only.
        dict(name="multi_h2o5_dz", kind="multi", mol="water", n=5, basis="cc-pVDZ"),
        # Many molecules of uneven size in one call (geometry sampling).
        dict(name="batch_h2o_631gs", kind="batch", mol="water", n=24, basis="6-31G*"),
        # The conventional form: Fock build from the integral store in HBM.
        dict(name="stored_h2o12_dz", kind="stored", mol="water", n=12, basis="cc-pVDZ"),
        # Forward and backward of the differentiable build: G, dL/dD, dL/dR.
        dict(name="autograd_h2o9_dz", kind="autograd", mol="water", n=9, basis="cc-pVDZ"),
        # One-electron integrals and one-electron gradient of a molecule.
        dict(name="oneel_h2o16_dz", kind="oneel", mol="water", n=16, basis="cc-pVDZ"),
        # A whole SCF: twelve iterations of the RHF driver.
        dict(name="scf_h2o3_dz", kind="scf", mol="water", n=3, basis="cc-pVDZ"),
    ]


def draw(rng):
    kind = rng.choice(["fock", "fock", "host", "incr", "rsh", "multi", "batch", "stored", "autograd", "oneel", "scf"])
    c = dict(kind=kind, mol=rng.choice(["water", "water", "alkane"]))
    if kind == "batch":
        c.update(mol="water", n=int(rng.randint(3, 24)), basis=rng.choice(["6-31G*", "STO-3G", "cc-pVDZ"]))
        return c
    c["basis"] = rng.choice(["cc-pVDZ", "cc-pVDZ", "6-31G*", "STO-3G", "cc-pVTZ", "aug-cc-pVDZ"])
    # atoms a size may reach, by kind and basis, so that no draw costs more
    # than the largest listed case
    top = {"fock": 20, "host": 16, "incr": 14, "rsh": 6, "multi": 5, "stored": 10, "autograd": 7, "oneel": 16,
           "scf": 3}[kind]
    if c["basis"] in ("cc-pVTZ", "aug-cc-pVDZ"):
        top = max(1, top // 4)
    if kind == "autograd" and c["basis"] == "cc-pVTZ":
        c["basis"] = "cc-pVDZ"  # the two-electron gradient covers s, p and d shells
    if c["mol"] == "alkane":
        top = max(2, top // 2)
        if c["basis"] == "aug-cc-pVDZ":
            c["basis"] = "cc-pVDZ"
        if kind == "scf":
            c["mol"] = "water"
    least = 2 if c["mol"] == "alkane" else 1
    c["n"] = int(round(math.exp(rng.uniform(math.log(least), math.log(top + 0.49)))))
    if kind == "rsh":
        c["mu"] = round(rng.uniform(0.2, 0.6), 2)
    if kind in ("fock", "host", "incr", "stored"):
        # exchange fraction of a hybrid functional, 1 for Hartree-Fock, 0 for none
        c["hfx"] = rng.choice([1.0, 1.0, 0.0, round(rng.uniform(0.05, 0.95), 2)])
    if kind == "incr":
        c["ifthrs"] = int(rng.randint(8, 12))
        c["cutoff"] = float(rng.choice([1e-7, 1e-6, 1e-5]))
    return c


# ------------------------------------------------------------------ inputs
def _molecule(case, seed):
    if case["mol"] == "water":
        n = case["n"]
        grid = (4, 4, 2) if n > 16 else None
        return molecules.water_cluster(n, grid, seed=seed)
    return molecules.alkane(case["n"], seed=seed)


def _density(bs, rng, sym=1, scale=1.0):
    """A density-like matrix: occupations on the diagonal, off-diagonal
    elements of random sign that decay with the atoms' distance; sym 1
    symmetric, 0 general, -1 antisymmetric."""
    n = bs.nbf
    xyz = bs.molecule.coords[bs.ao_atom()]
    r = np.linalg.norm(xyz[:, None, :] - xyz[None, :, :], axis=2)
    d = rng.normal(size=(n, n)) * 0.25 * np.exp(-0.6 * r)
    if sym == 1:
        d = 0.5 * (d + d.T) + np.diag(rng.uniform(0.2, 1.8, size=n))
    elif sym == -1:
        d = 0.5 * (d - d.T)
    return np.ascontiguousarray(d * scale)


MULTI_IFCTYP = [3, 13, 23, 1, 12]
MULTI_SYM = [0, 1, -1, 0, 1]


def _sizes(case):
    """Waters per molecule of a batch, the same for every seed."""
    rng = np.random.default_rng(case["n"])
    return [int(k) for k in rng.integers(1, 9, size=case["n"])]


def _cuda(a):
    return torch.tensor(a, dtype=torch.float64, device="cuda")


def _inputs(case, seed):
    """Basis sets and numpy inputs of a case, from the seed alone."""
    rng = np.random.default_rng(7919 * seed + 13)
    kind = case["kind"]
    if kind == "batch":
        mols = [molecules.water_cluster(k, seed=1000 * seed + i) for i, k in enumerate(_sizes(case))]
        bss = [build_basis(m, case["basis"]) for m in mols]
        return bss, [_density(b, rng) for b in bss]
    bs = build_basis(_molecule(case, seed), case["basis"])
    if kind == "incr":
        return bs, _density(bs, rng, scale=1e-2)
    if kind == "multi":
        return bs, np.stack([_density(bs, rng, sym=s) for s in MULTI_SYM])
    if kind == "autograd":
        return bs, (_density(bs, rng), _density(bs, rng))
    if kind == "oneel":
        return bs, (_density(bs, rng), _density(bs, rng))
    if kind == "scf":
        return bs, None
    return bs, _density(bs, rng)


def prepare(case, seed):
    kind = case["kind"]
    bs, x = _inputs(case, seed)
    st = dict(kind=kind, case=case)
    if kind == "batch":
        fbs = [FockBuilder(b) for b in bs]
        bb = BatchBuilder(fbs)
        dp = bb.pack([_cuda(d) for d in x])
        st.update(fbs=fbs, bb=bb, d=dp, f=torch.empty_like(dp))
        return st
    fb = FockBuilder(bs)
    st["fb"] = fb
    if kind in ("fock", "incr", "rsh", "multi", "stored"):
        st["d"] = _cuda(x)
        st["f"] = torch.empty_like(st["d"])
        if kind == "stored":
            fb.store_integrals(THRS)
    elif kind == "host":
        st["d"] = x
    elif kind == "autograd":
        st["d"], st["gbar"] = _cuda(x[0]), _cuda(x[1])
        st["xyz"] = _cuda(bs.molecule.coords)
    elif kind == "oneel":
        st["d"], st["w"] = x
    elif kind == "scf":
        st["bs"] = bs
    return st


def run(st):
    kind, hfx = st["kind"], st["case"].get("hfx", 1.0)
    if kind == "fock":
        return st["fb"].herfck_device(st["d"], fmat=st["f"], ifctyp=13, thrs=THRS, stats=False,
                                      hfxfac=hfx)
    if kind == "host":
        return st["fb"].herfck(st["d"], 13, thrs=THRS, hfxfac=hfx)
    if kind == "incr":
        return st["fb"].herfck_device(st["d"], fmat=st["f"], ifctyp=13, thrs=THRS, ifthrs=st["case"]["ifthrs"],
                                      mixed_cutoff=st["case"]["cutoff"], hfxfac=hfx, stats=False)
    if kind == "rsh":
        return st["fb"].herfck_device(st["d"], fmat=st["f"], ifctyp=13, hfxfac=0.2, hfxmu=st["case"]["mu"], hfxatt=0.6,
                                      thrs=THRS, stats=False)
    if kind == "multi":
        return st["fb"].herfck_device(st["d"], fmat=st["f"], ifctyp=MULTI_IFCTYP, thrs=THRS, stats=False)
    if kind == "batch":
        return st["bb"].herfck_batch(st["d"], st["f"], thrs=THRS, stats=False)
    if kind == "stored":
        return st["fb"].herfck_stored(st["d"], fmat=st["f"], ifctyp=13, thrs=THRS, hfxfac=hfx,
                                      stats=False)
    if kind == "autograd":
        d = st["d"].detach().requires_grad_(True)
        xyz = st["xyz"].detach().requires_grad_(True)
        g = FockJK.apply(d, xyz, st["fb"])
        gd, gr = torch.autograd.grad(g, (d, xyz), st["gbar"])
        return g.detach(), gd, gr
    if kind == "oneel":
        s, t, v = st["fb"].oneint()
        return s, t, v, st["fb"].grad1e(st["d"], st["w"])
    r = rhf(st["bs"], st["fb"], fixed_iterations=12)
    return r["energy"], r["dmat"], r["fock"]


# -------------------------------------------------------------------- work
def _shells(bs):
    """Primitive shells (l, exponent, coefficient size, centre) the build
    cannot do without: a general contraction's exponents once each."""
    out = []
    for i in range(bs.nblock):
        c = np.abs(bs.block_coefs(i)).max(axis=1)
        for a, ck in zip(bs.block_exps(i), c):
            out.append((int(bs.block_l[i]), float(a), float(ck), bs.molecule.coords[int(bs.block_atom[i])]))
    return out


def _quartet_flops(bs, flops_prim, flops_con):
    """Model FLOPs of one pass over the primitive shell quartets whose
    spherical-Gaussian Schwarz estimate reaches THRS."""
    sh = _shells(bs)
    l = np.array([s[0] for s in sh])
    a = np.array([s[1] for s in sh])
    c = np.array([s[2] for s in sh])
    x = np.array([s[3] for s in sh])
    i, j = np.tril_indices(len(sh))
    sw = l[j] > l[i]
    i, j = np.where(sw, j, i), np.where(sw, i, j)
    p = a[i] + a[j]
    r2 = ((x[i] - x[j]) ** 2).sum(axis=1)
    lsum = l[i] + l[j]
    # sqrt (ab|ab) of s functions, with the size of the polynomial factors
    q = c[i] * c[j] * np.exp(-a[i] * a[j] / p * r2) * math.sqrt(2.0 * math.pi ** 2.5) / p / (2.0 * p) ** 0.25
    q = q * (0.5 / p) ** (0.5 * lsum)
    cls = {}
    for la in range(4):
        for lb in range(la + 1):
            sel = (l[i] == la) & (l[j] == lb)
            if sel.any():
                cls[(la, lb)] = np.sort(q[sel])
    flops = 0.0
    keys = sorted(cls)
    for m, bra in enumerate(keys):
        for ket in keys[: m + 1]:
            qb, qk = cls[bra], cls[ket]
            n = len(qk) - np.searchsorted(qk, THRS / np.maximum(qb, 1e-300))
            cnt = float(n.sum())
            if bra == ket:
                cnt = 0.5 * (cnt + (qb * qb >= THRS).sum())
            flops += cnt * float(flops_prim(*bra, *ket) + flops_con(*bra, *ket))
    return flops


def _fock_flops(bs):
    return _quartet_flops(bs, perfmodel.flops_per_primitive, perfmodel.flops_per_contracted)


def _digest_flops(bs):
    return _quartet_flops(bs, lambda *c: 0.0, lambda *c: 12.0 * np.prod([perfmodel.nsph(l) for l in c]))


def _grad_flops(bs):
    return _quartet_flops(bs, perfmodel.grad_flops_per_primitive, perfmodel.grad_flops_per_contracted)


def work(case):
    kind = case["kind"]
    bs, _ = _inputs(case, 0)
    if kind == "batch":
        return {"bytes": sum(2 * 8 * b.nbf ** 2 for b in bs), "flops": sum(_fock_flops(b) for b in bs)}
    n2 = 8 * bs.nbf ** 2
    if kind == "rsh":
        return {"bytes": 2 * n2, "flops": 2 * _fock_flops(bs)}
    if kind == "multi":
        nd = len(MULTI_IFCTYP)
        return {"bytes": 2 * nd * n2, "flops": _fock_flops(bs) + (nd - 1) * _digest_flops(bs)}
    if kind == "stored":
        f = _digest_flops(bs)
        return {"bytes": 2 * n2 + f / 12.0 * 8.0, "flops": f}
    if kind == "autograd":
        return {"bytes": 4 * n2, "flops": 2 * _fock_flops(bs) + _grad_flops(bs)}
    if kind == "oneel":
        # per pair of primitive functions and nucleus about 60 operations
        nf = sum((s[0] + 1) * (s[0] + 2) // 2 for s in _shells(bs))
        return {"bytes": 5 * n2, "flops": 0.5 * nf * nf * bs.molecule.natom * 60.0 * 3.0}
    if kind == "scf":
        return {"bytes": 12 * 2 * n2, "flops": 12 * (_fock_flops(bs) + 30.0 * bs.nbf ** 3)}
    return {"bytes": 2 * n2, "flops": _fock_flops(bs)}


def tolerance(case):
    """About four times the largest error against `exact`, or against the
    unscreened FP64 build, that the sizes of `draw` showed."""
    kind = case["kind"]
    if kind == "incr":
        # the density screen skips whole blocks below 10^-ifthrs, and FP32
        # integrals stand below the cutoff: 5e-7, 3e-8, 5e-9, -, 5e-11 seen
        # at ifthrs 8, 9, 10, 11, 12
        return {"rel": 2e-6 * 10.0 ** (8 - case["ifthrs"])}
    if kind == "scf":
        return {"rel": 1e-9}   # the density after twelve iterations: 6e-11 seen
    if kind == "autograd":
        return {"rel": 8e-12}  # the gradient: 2e-12 seen
    if kind == "oneel":
        return {"rel": 1e-13}  # the gradient: 2e-14 seen
    return {"rel": 2e-12}      # quartets below the Schwarz threshold: 4e-13 seen


# ------------------------------------------------- exact: plain torch, FP64
# The integrals from their definition in Hermite Gaussians (McMurchie and
# Davidson, J. Comput. Phys. 26, 218 (1978)), every primitive quartet, no
# screening, dense tensors.
def _dev():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _carts(l):
    return [(i, j, l - i - j) for i in range(l, -1, -1) for j in range(l - i, -1, -1)]


def _tuv(L):
    return [(t, u, v) for t in range(L + 1) for u in range(L + 1 - t) for v in range(L + 1 - t - u)]


def _solid(l):
    """Real solid harmonics m = -l..l over x^i y^j z^k, in the normalisation
    in which the coefficients carry the norm of x^l without (2l-1)!!."""
    s = math.sqrt
    if l == 2:
        rows = [{(1, 1, 0): 1.0}, {(0, 1, 1): 1.0},
                {(0, 0, 2): 1 / s(3), (2, 0, 0): -0.5 / s(3), (0, 2, 0): -0.5 / s(3)},
                {(1, 0, 1): 1.0}, {(2, 0, 0): 0.5, (0, 2, 0): -0.5}]
    elif l == 3:
        a, b, c = s(5 / 8) / s(15), s(3 / 8) / s(15), 1 / s(15)
        rows = [{(2, 1, 0): 3 * a, (0, 3, 0): -a}, {(1, 1, 1): 1.0},
                {(0, 1, 2): 4 * b, (2, 1, 0): -b, (0, 3, 0): -b},
                {(0, 0, 3): c, (2, 0, 1): -1.5 * c, (0, 2, 1): -1.5 * c},
                {(1, 0, 2): 4 * b, (3, 0, 0): -b, (1, 2, 0): -b},
                {(2, 0, 1): 0.5, (0, 2, 1): -0.5}, {(3, 0, 0): a, (1, 2, 0): -3 * a}]
    else:
        return np.eye((l + 1) * (l + 2) // 2)
    car = _carts(l)
    m = np.zeros((2 * l + 1, len(car)))
    for r, row in enumerate(rows):
        for k, v in row.items():
            m[r, car.index(k)] = v
    return m


def _boys(M, T):
    """F_0..F_M: the ascending series of F_M and downward recursion for
    T < 36, erf and upward recursion above."""
    small = T < 36.0
    Ts = torch.where(small, T, torch.ones_like(T))
    term = torch.full_like(Ts, 1.0 / (2 * M + 1))
    tot = term
    for k in range(1, 170):
        term = term * (2.0 * Ts / (2 * M + 2 * k + 1))
        tot = tot + term
    e = torch.exp(-Ts)
    lo = [e * tot]
    for m in range(M - 1, -1, -1):
        lo.append((2.0 * Ts * lo[-1] + e) / (2 * m + 1))
    lo = lo[::-1]
    Tb = torch.where(small, torch.full_like(T, 40.0), T)
    eb = torch.exp(-Tb)
    hi = [0.5 * torch.sqrt(math.pi / Tb) * torch.erf(torch.sqrt(Tb))]
    for m in range(M):
        hi.append(((2 * m + 1) * hi[-1] - eb) / (2.0 * Tb))
    return [torch.where(small, a, b) for a, b in zip(lo, hi)]


def _hermite_r(L, fac, alpha, x, y, z):
    """{(t,u,v): R_tuv} for t+u+v <= L, scaled by fac."""
    F = _boys(L, alpha * (x * x + y * y + z * z))
    r = {}
    for n in range(L, -1, -1):
        nr = {(0, 0, 0): fac * F[n] * (-2.0 * alpha) ** n}
        for s in range(1, L - n + 1):
            for t, u, v in _tuv(s):
                if t + u + v != s:
                    continue
                if t:
                    val = x * r[(t - 1, u, v)] + ((t - 1) * r[(t - 2, u, v)] if t > 1 else 0.0)
                elif u:
                    val = y * r[(t, u - 1, v)] + ((u - 1) * r[(t, u - 2, v)] if u > 1 else 0.0)
                else:
                    val = z * r[(t, u, v - 1)] + ((v - 1) * r[(t, u, v - 2)] if v > 1 else 0.0)
                nr[(t, u, v)] = val
        r = nr
    return r


def _e1(la, lb, p, pa, pb):
    """E[(i, j, t)] of one direction."""
    e = {(0, 0, 0): torch.ones_like(p)}
    h = 0.5 / p
    get = lambda i, j, t: e.get((i, j, t), 0.0)
    for i in range(la + 1):
        for j in range(lb + 1):
            if i == j == 0:
                continue
            a, b, w = (i - 1, j, pa) if i else (i, j - 1, pb)
            for t in range(i + j + 1):
                e[(i, j, t)] = w * get(a, b, t) + h * get(a, b, t - 1) + (t + 1) * get(a, b, t + 1)
    return e


class _Prims:
    """Primitive shells by angular momentum and the map from the primitive
    functions (spherical) to the contracted ones."""

    def __init__(self, bs, xyz):
        self.dev = xyz.device
        off, self.l, self.off, at, ex, rows = 0, [], [], [], [], []
        for i in range(bs.nblock):
            l, c = int(bs.block_l[i]), bs.block_coefs(i)
            nf = 2 * l + 1
            for k, a in enumerate(bs.block_exps(i)):
                self.l.append(l)
                self.off.append(off)
                at.append(int(bs.block_atom[i]))
                ex.append(float(a))
                for m in range(nf):
                    rows.append([(int(bs.block_ao_offset[i]) + q * nf + m, c[k, q]) for q in range(c.shape[1])])
                off += nf
        self.n = off
        self.l, self.off = np.array(self.l), np.array(self.off)
        self.at = torch.tensor(at, device=self.dev)
        self.a = torch.tensor(ex, dtype=torch.float64, device=self.dev)
        self.x = xyz[self.at]
        C = np.zeros((off, bs.nbf))
        for p, r in enumerate(rows):
            for mu, v in r:
                C[p, mu] += v
        self.C = torch.tensor(C, device=self.dev)

    def pairs(self, ordered=False):
        """Shell pairs by (la, lb): every pair once with la >= lb (ordered:
        both orders), as dicts of tensors with the spherical Hermite
        coefficients E[pair, function pair, tuv]."""
        out = {}
        n = len(self.l)
        i, j = (v.reshape(-1) for v in np.meshgrid(np.arange(n), np.arange(n), indexing="ij"))
        if not ordered:
            keep = (self.l[i] > self.l[j]) | ((self.l[i] == self.l[j]) & (i >= j))
            i, j = i[keep], j[keep]
        for la in range(4):
            for lb in range(4):
                sel = (self.l[i] == la) & (self.l[j] == lb)
                if not sel.any():
                    continue
                I = torch.tensor(i[sel], device=self.dev)
                J = torch.tensor(j[sel], device=self.dev)
                out[(la, lb)] = self._pair(la, lb, I, J)
        return out

    def _pair(self, la, lb, I, J, extra=0):
        a, b, A, B = self.a[I], self.a[J], self.x[I], self.x[J]
        p = a + b
        P = (a[:, None] * A + b[:, None] * B) / p[:, None]
        K = torch.exp(-a * b / p * ((A - B) ** 2).sum(1))
        e = [_e1(la, lb + extra, p, P[:, k] - A[:, k], P[:, k] - B[:, k]) for k in range(3)]
        ca, cb, tuv = _carts(la), _carts(lb), _tuv(la + lb)
        zero = torch.zeros_like(p)
        E = torch.stack([torch.stack([
            e[0][(x[0], y[0], t)] * e[1][(x[1], y[1], u)] * e[2][(x[2], y[2], v)]
            if (t <= x[0] + y[0] and u <= x[1] + y[1] and v <= x[2] + y[2]) else zero
            for t, u, v in tuv], 1) for x in ca for y in cb], 1)
        E = E.reshape(len(p), len(ca), len(cb), len(tuv))
        sa = torch.tensor(_solid(la), device=self.dev)
        sb = torch.tensor(_solid(lb), device=self.dev)
        E = torch.einsum("mx,ny,pxyt->pmnt", sa, sb, E) * K[:, None, None, None]
        off = torch.tensor(self.off, device=self.dev)
        fa = off[I][:, None] + torch.arange(2 * la + 1, device=self.dev)
        fb = off[J][:, None] + torch.arange(2 * lb + 1, device=self.dev)
        return dict(p=p, P=P, E=E, fa=fa, fb=fb, same=(I == J), e=e, K=K, b=b, la=la, lb=lb)


def _blocks(bra, ket, mu=0.0, limit=3e7):
    """Chunks (slice of bra pairs, g[p, a, b, q, c, d]) of a class pair."""
    la, lb, lc, ld = bra["la"], bra["lb"], ket["la"], ket["lb"]
    tb, tk = _tuv(la + lb), _tuv(lc + ld)
    sign = torch.tensor([(-1.0) ** (t + u + v) for t, u, v in tk], device=bra["p"].device, dtype=torch.float64)
    nq = len(ket["p"])
    step = max(1, int(limit / (nq * max(len(tb) * len(tk), 16))))
    for s in range(0, len(bra["p"]), step):
        sl = slice(s, s + step)
        p, q = bra["p"][sl][:, None], ket["p"][None, :]
        alpha = p * q / (p + q)
        fac = 2.0 * math.pi ** 2.5 / (p * q * torch.sqrt(p + q))
        if mu:
            beta = mu * mu / (alpha + mu * mu)
            alpha, fac = alpha * beta, fac * torch.sqrt(beta)
        d = bra["P"][sl][:, None, :] - ket["P"][None, :, :]
        R = _hermite_r(la + lb + lc + ld, fac, alpha, d[..., 0], d[..., 1], d[..., 2])
        rows = [torch.stack([R[(t + x, u + y, v + z)] for x, y, z in tk], -1) for t, u, v in tb]
        M = torch.stack(rows, -2) * sign                       # p q e f
        X = torch.einsum("pqef,qcdf->pqecd", M, ket["E"])
        yield sl, torch.einsum("pabe,pqecd->pabqcd", bra["E"][sl], X)


def _jk(pr, pairs, D, mu=0.0):
    """J and K (lists over densities) in the primitive basis, every ordered
    bra x ket combination of unordered shell pairs."""
    n = pr.n
    nd = len(D)
    J = [torch.zeros(n * n, dtype=torch.float64, device=pr.dev) for _ in range(nd)]
    K = [torch.zeros(n * n, dtype=torch.float64, device=pr.dev) for _ in range(nd)]

    def add(M, r, c, v):
        M.index_add_(0, (r * n + c).expand_as(v).reshape(-1), v.reshape(-1))

    for bra in pairs.values():
        for ket in pairs.values():
            kc, kd = ket["fa"], ket["fb"]
            wk = torch.where(ket["same"], 0.5, 1.0).to(torch.float64)
            for sl, g in _blocks(bra, ket, mu):
                a, b = bra["fa"][sl], bra["fb"][sl]
                wb = torch.where(bra["same"][sl], 0.5, 1.0).to(torch.float64)
                g = g * wb[:, None, None, None, None, None] * wk[None, None, None, :, None, None]
                ix = lambda r, c: (r[:, None, :, None], c[None, :, None, :])  # [p, q, row, col]
                for k in range(nd):
                    Ds = D[k] + D[k].T
                    cd = Ds[kc[:, :, None], kd[:, None, :]]
                    jab = torch.einsum("pabqcd,qcd->pab", g, cd)
                    add(J[k], a[:, :, None], b[:, None, :], jab)
                    add(J[k], b[:, None, :], a[:, :, None], jab)
                    for eq, r, c, x, y in (("pabqcd,pqbd->pqac", a, kc, b, kd), ("pabqcd,pqbc->pqad", a, kd, b, kc),
                                           ("pabqcd,pqad->pqbc", b, kc, a, kd), ("pabqcd,pqac->pqbd", b, kd, a, kc)):
                        v = torch.einsum(eq, g, D[k][ix(x, y)])
                        add(K[k], *ix(r, c), v)
    return [m.reshape(n, n) for m in J], [m.reshape(n, n) for m in K]


def _exact_fock(bs, dens, ifctyp, hfx=1.0, mu=0.0, att=0.0):
    dev = _dev()
    pr = _Prims(bs, torch.tensor(bs.molecule.coords, device=dev))
    pairs = pr.pairs()
    C = pr.C
    sym = {0: lambda d: d, 1: lambda d: 0.5 * (d + d.T), 2: lambda d: 0.5 * (d - d.T)}
    D = [sym[t // 10](torch.tensor(d, device=dev)) for d, t in zip(dens, ifctyp)]
    Dp = [C @ d @ C.T for d in D]
    J, K = _jk(pr, pairs, Dp)
    out = []
    Ka = _jk(pr, pairs, Dp, mu)[1] if mu else None
    for k, t in enumerate(ifctyp):
        f = torch.zeros_like(D[k])
        if t % 10 & 1 and t // 10 != 2:
            f = f + C.T @ J[k] @ C
        if t % 10 & 2:
            f = f - 0.5 * hfx * (C.T @ K[k] @ C)
        if mu:
            f = f - 0.5 * att * (C.T @ Ka[k] @ C)
        out.append(f)
    return out


def _exact_oneint(bs, xyz=None):
    dev = _dev()
    xyz = torch.tensor(bs.molecule.coords, device=dev) if xyz is None else xyz
    pr = _Prims(bs, xyz)
    n = pr.n
    S, T, V = (torch.zeros(n, n, dtype=torch.float64, device=dev) for _ in range(3))
    Z = torch.tensor(bs.molecule.charges, device=dev)
    sh = np.arange(len(pr.l))
    for la in range(4):
        for lb in range(4):
            i, j = sh[pr.l == la], sh[pr.l == lb]
            if not len(i) or not len(j):
                continue
            I, J = (torch.tensor(v.reshape(-1), device=dev) for v in np.meshgrid(i, j, indexing="ij"))
            q = pr._pair(la, lb, I, J, extra=2)
            s0 = (math.pi / q["p"]) ** 1.5 * q["K"]
            e, b = q["e"], q["b"]
            sx = [lambda x, y, k=k: e[k][(x, y, 0)] if y >= 0 else 0.0 for k in range(3)]

            def kin(k, x, y):
                return -0.5 * (y * (y - 1) * sx[k](x, y - 2) - 2.0 * b * (2 * y + 1) * sx[k](x, y) +
                               4.0 * b * b * sx[k](x, y + 2))

            ov, ke = [], []
            for x in _carts(la):
                for y in _carts(lb):
                    o = [sx[k](x[k], y[k]) for k in range(3)]
                    ov.append(s0 * o[0] * o[1] * o[2])
                    ke.append(s0 * (kin(0, x[0], y[0]) * o[1] * o[2] + o[0] * kin(1, x[1], y[1]) * o[2] +
                                    o[0] * o[1] * kin(2, x[2], y[2])))
            sa, sb = (torch.tensor(_solid(l), device=dev) for l in (la, lb))
            sph = lambda v: torch.einsum("mx,ny,pxy->pmn", sa, sb, torch.stack(v, 1).reshape(
                len(s0), (la + 1) * (la + 2) // 2, (lb + 1) * (lb + 2) // 2))
            d = q["P"][:, None, :] - xyz[None, :, :]
            p = q["p"][:, None].expand(d.shape[:2])
            fac = -Z[None, :] * 2.0 * math.pi / p
            R = _hermite_r(la + lb, fac, p, d[..., 0], d[..., 1], d[..., 2])
            Rs = torch.stack([R[k].sum(1) for k in _tuv(la + lb)], 1)
            at = (q["fa"][:, :, None], q["fb"][:, None, :])
            S = S.index_put(at, sph(ov))
            T = T.index_put(at, sph(ke))
            V = V.index_put(at, torch.einsum("pmnt,pt->pmn", q["E"], Rs))
    C = pr.C
    return [C.T @ m @ C for m in (S, T, V)]


def _nuclear(charges, xyz):
    n = len(charges)
    i, j = np.triu_indices(n, 1)
    z = torch.tensor(charges[i] * charges[j], device=xyz.device)
    return (z / torch.linalg.norm(xyz[i] - xyz[j], dim=1)).sum()


def _exact_grad1e(bs, d, w):
    """sum D dh - sum W dS + dVnn, by differentiating the integrals above."""
    dev = _dev()
    xyz = torch.tensor(bs.molecule.coords, device=dev, requires_grad=True)
    S, T, V = _exact_oneint(bs, xyz)
    d, w = torch.tensor(d, device=dev), torch.tensor(w, device=dev)
    e = (d * (T + V)).sum() - (w * S).sum() + (_nuclear(bs.molecule.charges, xyz) if len(bs.molecule.charges) > 1 else 0)
    return torch.autograd.grad(e, xyz)[0]


def _exact_gradient(bs, d1, d2):
    """d <D2, G(D1)> / dR for symmetric D1, D2, by differentiating the
    contraction of the Hermite integrals."""
    dev = _dev()
    xyz = torch.tensor(bs.molecule.coords, device=dev, requires_grad=True)
    grad = torch.zeros_like(xyz)
    C = _Prims(bs, xyz.detach()).C
    D1, D2 = (C @ torch.tensor(d, device=dev) @ C.T for d in (d1, d2))
    keys = list(_Prims(bs, xyz.detach()).pairs())
    for kb in keys:
        for kk in keys:
            pairs = _Prims(bs, xyz).pairs()
            bra, ket = pairs[kb], pairs[kk]
            e = 0.0
            c, dd = ket["fa"], ket["fb"]
            wk = torch.where(ket["same"], 1.0, 2.0).to(torch.float64)
            for sl, g in _blocks(bra, ket):
                a, b = bra["fa"][sl], bra["fb"][sl]
                wb = torch.where(bra["same"][sl], 1.0, 2.0).to(torch.float64)
                ab = lambda M: M[a[:, :, None], b[:, None, :]]
                cd = lambda M: M[c[:, :, None], dd[:, None, :]]
                x = lambda M, r, s: M[r[:, None, :, None], s[None, :, None, :]]
                g = g * wb[:, None, None, None, None, None] * wk[None, None, None, :, None, None]
                e = e + torch.einsum("pabqcd,pab,qcd->", g, ab(D2), cd(D1))
                for s1, s2 in (("pqac,pqbd", (a, c, b, dd)), ("pqad,pqbc", (a, dd, b, c)),
                               ("pqbc,pqad", (b, c, a, dd)), ("pqbd,pqac", (b, dd, a, c))):
                    e = e - 0.125 * torch.einsum("pabqcd,%s->" % s1, g, x(D2, *s2[:2]), x(D1, *s2[2:]))
            grad = grad + torch.autograd.grad(e, xyz)[0]
    return grad


def _exact_scf(bs, iters):
    """The RHF driver's iterations with the full integral tensor."""
    dev = _dev()
    S, T, V = _exact_oneint(bs)
    pr = _Prims(bs, torch.tensor(bs.molecule.coords, device=dev))
    pairs = pr.pairs()
    H = T + V
    nocc = bs.molecule.nelectrons() // 2
    s, U = torch.linalg.eigh(S)
    X = U / torch.sqrt(s)

    def dens(F):
        c = X @ torch.linalg.eigh(X.T @ F @ X)[1]
        return 2.0 * c[:, :nocc] @ c[:, :nocc].T

    D = dens(H)
    errs, focks = [], []
    for it in range(iters):
        J, K = _jk(pr, pairs, [pr.C @ D @ pr.C.T])
        F = H + pr.C.T @ (J[0] - 0.5 * K[0]) @ pr.C
        err = X.T @ (F @ D @ S - S @ D @ F) @ X
        energy = float(0.5 * (D * (H + F)).sum()) + bs.molecule.nuclear_repulsion()
        errs, focks = (errs + [err])[-8:], (focks + [F])[-8:]
        if it + 1 == iters:
            break
        m = len(errs)
        Fx = F
        if m >= 2:
            B = -torch.ones(m + 1, m + 1, dtype=torch.float64, device=dev)
            B[m, m] = 0.0
            for i in range(m):
                for j in range(m):
                    B[i, j] = (errs[i] * errs[j]).sum()
            r = torch.zeros(m + 1, dtype=torch.float64, device=dev)
            r[m] = -1.0
            c = torch.linalg.solve(B, r)[:m]
            Fx = sum(ci * f for ci, f in zip(c, focks))
        D = dens(Fx)
    return energy, D, F


def exact(case, seed):
    kind = case["kind"]
    bs, x = _inputs(case, seed)
    if kind == "batch":
        if sum(int(b.block_nprim.sum()) ** 2 for b in bs) > 2 * EXACT_SHELLS ** 2:
            return None
        return torch.cat([_exact_fock(b, [d], [13])[0].reshape(-1) for b, d in zip(bs, x)])
    shells = int(bs.block_nprim.sum())
    if kind == "oneel":
        if shells > 6 * EXACT_SHELLS:
            return None
        s, t, v = _exact_oneint(bs)
        return s, t, v, (_exact_grad1e(bs, *x) if shells <= 2 * EXACT_SHELLS else None)
    if shells > EXACT_SHELLS or (kind == "scf" and shells > EXACT_SHELLS // 2):
        return None
    if kind in ("fock", "host", "incr", "stored"):
        return _exact_fock(bs, [x], [13], hfx=case.get("hfx", 1.0))[0]
    if kind == "rsh":
        return _exact_fock(bs, [x], [13], hfx=0.2, mu=case["mu"], att=0.6)[0]
    if kind == "multi":
        return torch.stack(_exact_fock(bs, list(x), MULTI_IFCTYP))
    if kind == "autograd":
        g, gd = (_exact_fock(bs, [d], [13])[0] for d in x)
        return g, gd, (_exact_gradient(bs, x[0], x[1]) if shells <= EXACT_SHELLS_GRAD else None)
    return _exact_scf(bs, 12)
