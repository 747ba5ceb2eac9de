"""Timed cases of the SCF framework's public entry points.

Each case names one entry a user's program calls, with its sizes: the drop-in ``nanoDFT`` call,
the fixed-iteration SCF loop of an engine, and the batched pieces of dataset generation (device
setup, ERIs, J/K, exchange-correlation, nuclear gradients, whole batches to convergence).
Molecules are seeded random trees of 1-9 heavy atoms (C/N/O/F, hydrogens to valence) with
several jittered conformers each, as dataset generation runs several conformers of one
molecule.  The mixed-precision path holds its integrals and grid work in float32, so its
results are returned as float32; the float64 path's are returned as they are.
"""
import itertools
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "pyscf-ipu_b200"))

from b200dft._lib import check, lib, ptr, stream_handle                     # noqa: E402
from b200dft.engine import NMO, RKSEngine, nuclear_gradient, run_batches    # noqa: E402
from b200dft.mole import Mole                                               # noqa: E402
from b200dft.molgen import random_molecule                                  # noqa: E402
from b200dft.nanodft import nanoDFT, nanoDFT_options                        # noqa: E402
from b200dft.train_guess import load as load_guess_net                      # noqa: E402

CONFORMERS = 8        # conformers per random tree
HYB = 0.2             # exact-exchange fraction of B3LYP
LEVEL_POINTS = {0: 230, 1: 950, 2: 4100, 3: 6500}    # grid points per orbital, about


def listed():
    return [
        # the smallest call a user makes: the drop-in on one water-sized molecule, default options
        dict(name="nanodft-fp64-1", kind="nanodft", precision="fp64", nmol=1, lo=1, hi=1, level=0),
        # the drop-in on a molecule of QM1B's larger half, with its float32 option
        dict(name="nanodft-mixed-7", kind="nanodft", precision="mixed", nmol=1, lo=7, hi=7, level=0),
        # one molecule at the size cap on the command line's default grid (level 2), 20 iterations
        dict(name="scf-fp64-9-l2", kind="scf", precision="fp64", nmol=1, lo=9, hi=9, level=2),
        # device setup of a generation batch: one-electron integrals, grid, guess, L
        dict(name="setup-1500", kind="setup", precision="mixed", nmol=1500, lo=1, hi=9, level=0),
        # integrals of a generation batch (float32 lists, exchange list)
        dict(name="eri-mixed-2048", kind="eri", precision="mixed", nmol=2048, lo=1, hi=9, level=0),
        # integrals of a small batch at the reference's float64
        dict(name="eri-fp64-50", kind="eri", precision="fp64", nmol=50, lo=1, hi=9, level=0),
        # J/K of one SCF iteration of a generation batch
        dict(name="jk-mixed-1024", kind="jk", precision="mixed", nmol=1024, lo=1, hi=9, level=0),
        # exchange-correlation of one SCF iteration of a generation batch
        dict(name="xc-mixed-2048", kind="xc", precision="mixed", nmol=2048, lo=1, hi=9, level=0),
        # the same at float64 on the command line's default grid, a few uneven molecules
        dict(name="xc-fp64-7-l2", kind="xc", precision="fp64", nmol=7, lo=2, hi=9, level=2),
        # forces of one molecule after its SCF
        dict(name="grad-1", kind="grad", precision="fp64", nmol=1, lo=5, hi=5, level=0),
        # force labels of a batch
        dict(name="grad-160", kind="grad", precision="fp64", nmol=160, lo=1, hi=9, level=0),
        # dataset generation: two batches through the pipelined driver, learned guess, converged
        dict(name="generate-2x1024", kind="generate", precision="mixed", nmol=2048, lo=1, hi=9, level=0),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["nanodft", "scf", "setup", "eri", "jk", "xc", "grad", "generate"])
    prec = rng.choice(["fp64", "mixed"])
    lo, hi = rng.choice([(1, 3), (1, 9), (4, 9), (7, 9)])
    level = 0
    if kind == "nanodft":
        nmol, level = 1, rng.choice([0, 0, 1])
        lo = hi = rng.randint(1, 6 if level else 8)
    elif kind == "scf":
        level = rng.choice([0, 1, 2])
        nmol = _log_int(rng, 1, {0: 40, 1: 10, 2: 3}[level])
    elif kind == "setup":
        nmol, prec = _log_int(rng, 1, 1400), "mixed"
    elif kind == "eri":
        nmol = _log_int(rng, 1, 1000 if prec == "mixed" else 50)
    elif kind == "jk":
        nmol = _log_int(rng, 1, 500 if prec == "mixed" else 150)
    elif kind == "xc":
        level = rng.choice([0, 1, 2, 3])
        nmol = _log_int(rng, 1, {0: 1500, 1: 400, 2: 100, 3: 60}[level] // (1 if prec == "mixed" else 16))
    elif kind == "grad":
        nmol, prec = _log_int(rng, 1, 80), "fp64"
    else:
        nmol, prec = 2 * _log_int(rng, 8, 500), "mixed"
    return dict(kind=kind, precision=prec, nmol=nmol, lo=lo, hi=hi, level=level)


# ---------------------------------------------------------------------------- inputs

def _families(case, seed):
    """molecules as a list of conformer groups: the trees follow from the case (so its sizes do),
    the conformers' coordinates from the seed"""
    tree = np.random.default_rng([case["nmol"], case["lo"], case["hi"]])
    rng = np.random.default_rng(seed)
    out, left = [], case["nmol"]
    while left:
        k = min(CONFORMERS, left)
        base = Mole(random_molecule(tree, int(tree.integers(case["lo"], case["hi"] + 1))))
        group = []
        for _ in range(k):
            xyz = base.coords + rng.normal(scale=0.08, size=base.coords.shape)
            group.append(Mole(list(zip(base.symbols, xyz.tolist())), unit="Bohr"))
        out.append(group)
        left -= k
    return out


def _molecules(case, seed):
    return [m for g in _families(case, seed) for m in g]


def _tables(group):
    """AO tables of a conformer group on the GPU: centres (k, n, 3), directions (n, 3; zero for
    s), exponents and coefficients (n, 3)"""
    t = group[0].ao_table()
    n = group[0].nao
    dirs = np.zeros((n, 3))
    p = t["l"] == 1
    dirs[p, t["comp"][p]] = 1.0
    R = np.stack([m.coords[t["atom"]] for m in group])
    gpu = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    return gpu(R), gpu(dirs), gpu(t["exps"]), gpu(t["coef"]), t


def _pairs(R, dirs, ex, cf):
    """primitive-pair quantities over (k, n, n, 9): zeta, weight, P, and the linear factors"""
    n = ex.shape[0]
    a = ex[:, None, :, None].expand(n, n, 3, 3).reshape(n, n, 9)
    b = ex[None, :, None, :].expand(n, n, 3, 3).reshape(n, n, 9)
    c = (cf[:, None, :, None] * cf[None, :, None, :]).reshape(n, n, 9)
    z = a + b
    A, B = R[:, :, None, None, :], R[:, None, :, None, :]
    P = (a[..., None] * A + b[..., None] * B) / z[..., None]
    w = c * torch.exp(-a * b / z * ((A - B) ** 2).sum(-1))
    isp = dirs.abs().sum(-1)
    da, db = dirs[:, None, None, :], dirs[None, :, None, :]
    sa = ((P - A) * da).sum(-1) + (1.0 - isp)[:, None, None]
    sb = ((P - B) * db).sum(-1) + (1.0 - isp)[None, :, None]
    return z, w, P, sa, sb


def _overlap(R, dirs, ex, cf):
    z, w, _, sa, sb = _pairs(R, dirs, ex, cf)
    dd = (dirs @ dirs.T)[:, :, None]
    return (w * (math.pi / z) ** 1.5 * (sa * sb + dd * 0.5 / z)).sum(-1)


_EPS = {1: (-0.5,), 6: (-11.3, -0.75, -0.40), 7: (-15.6, -0.95, -0.50), 8: (-20.7, -1.2, -0.60),
        9: (-26.4, -1.5, -0.70)}                       # orbital energies (1s, 2s, 2p), about


def _orbitals(families):
    """bonding orbitals of every molecule from an extended-Hueckel matrix, in plain torch: lists
    of (C, energies, D) per molecule (numpy, column k = orbital k, S-orthonormal)"""
    out = []
    for group in families:
        R, dirs, ex, cf, t = _tables(group)
        S = _overlap(R, dirs, ex, cf)
        z = group[0].charges[t["atom"]]
        first = np.concatenate([[True], t["atom"][1:] != t["atom"][:-1]])      # an atom's 1s
        shell = np.where(t["l"] == 1, 2, np.where(first, 0, 1))
        e = torch.tensor([_EPS[int(q)][int(s)] for q, s in zip(z, shell)], dtype=torch.float64, device="cuda")
        H = 0.875 * (e[:, None] + e[None, :]) * S
        H.diagonal(dim1=-2, dim2=-1).copy_(e.expand(S.shape[:-1]))
        Li = torch.linalg.inv(torch.linalg.cholesky(S))
        eps, U = torch.linalg.eigh(Li @ H @ Li.mT)
        C = Li.mT @ U
        occ = C[:, :, :group[0].nelectron // 2]
        D = 2.0 * occ @ occ.mT
        out += list(zip(C.cpu().numpy(), eps.cpu().numpy(), D.cpu().numpy()))
    return out


def _engine(case, mols):
    return RKSEngine(mols, level=case["level"], precision=case["precision"])


def _flat(eng, mats):
    return torch.from_numpy(eng.plan.pack(mats)).cuda()


def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case}
    if kind == "nanodft":
        s["mol"] = _molecules(case, seed)[0]
        s["opts"] = nanoDFT_options(float32=case["precision"] == "mixed", level=case["level"])[0]
        return s
    if kind == "generate":
        mols = _molecules(case, seed)
        h = len(mols) // 2
        # neighbours in the list are conformers of one tree: deal them out to both batches
        s["batches"] = [mols[0::2], mols[1::2]] if h else [mols]
        s["net"] = load_guess_net()
        return s
    fam = _families(case, seed)
    s["mols"] = mols = [m for g in fam for m in g]
    s["eng"] = eng = _engine(case, mols)
    if kind == "scf":
        eng.prepare()
    elif kind == "eri":
        eng.eri.zero_()                 # the lists' padding is never written
        eng.eri_x.zero_()
    elif kind == "jk":
        # integral lists whose values spread over several decades, as real ones do
        gen = torch.Generator(device="cuda").manual_seed(seed)
        n = eng.eri.numel()
        r = dict(generator=gen, device="cuda", dtype=torch.float32)
        eng.eri.copy_(torch.randn(n, **r) * torch.exp(-9.0 * torch.rand(n, **r)))
        eng.eri_x.zero_()
        check(lib().b2_jk_exchange(eng.plan.h, eng.prec, ptr(eng.eri), ptr(eng.eri_x), stream_handle()),
              "b2_jk_exchange")
        s["D"] = _flat(eng, [o[2] for o in _orbitals(fam)])
    elif kind == "xc":
        eng.device_setup()
        s["D"] = _flat(eng, [o[2] for o in _orbitals(fam)])
    elif kind == "grad":
        eng.device_setup()
        orb = _orbitals(fam)
        s["C"] = _flat(eng, [o[0] for o in orb])
        mo = np.zeros((len(mols), NMO))
        for k, o in enumerate(orb):
            mo[k, :len(o[1])] = o[1]
        s["mo"] = torch.from_numpy(mo.reshape(-1)).cuda()
    return s


# ---------------------------------------------------------------------------- one pass

def _typed(case, x):
    """the mixed path's float64 buffers hold float32-accurate results"""
    if case["precision"] == "fp64":
        return x
    return x.astype(np.float32) if isinstance(x, np.ndarray) else x.float()


def run(state):
    case = state["case"]
    kind = case["kind"]
    f = lambda x: _typed(case, x)
    if kind == "nanodft":
        mol = state["mol"]
        E, (logged, gaps, mo_energy, mo_coeff, coords, weights) = nanoDFT(mol, state["opts"])
        occ = mo_coeff[:, :mol.nelectron // 2]
        return {"energies": f(E), "logged": f(logged), "hlgap": f(gaps), "mo_energy": f(mo_energy),
                "density": f(2.0 * occ @ occ.T), "coords": coords, "weights": weights}
    if kind == "generate":
        out = {}
        for k, (_, r) in enumerate(run_batches(state["batches"], net=state["net"])):
            out["energy%d" % k], out["mo_energy%d" % k] = f(r["energy"]), f(r["mo_energy"])
        return out
    eng = state["eng"]
    if kind == "scf":
        r = eng.run(its=20, log=False)
        return {"energies": f(r["energies"]), "mo_energy": f(r["mo_energy"]), "D": f(eng.D)}
    if kind == "setup":
        e = RKSEngine(state["mols"], level=case["level"], precision=case["precision"], plan=eng.plan)
        e.device_setup()
        return {"S": e.S, "T": e.T, "V": e.V, "Linv": e.Linv, "D0": e.D0, "enuc": e.enuc,
                "coords": e.coords, "weights": e.weights}
    if kind == "eri":
        eng.compute_eri()
        return {"eri": eng.eri, "exchange": eng.eri_x}
    if kind == "jk":
        eng.jk(D=state["D"])
        return {"J": f(eng.J), "K": f(eng.K)}
    if kind == "xc":
        eng.xc(D=state["D"])
        return {"V": f(eng.Vxc), "E": f(eng.exc)}
    return nuclear_gradient(eng.plan, state["C"], state["mo"], eng.coords, eng.weights)


# ---------------------------------------------------------------------------- what a pass needs

def work(case):
    """bytes and operations of one pass, from the sizes of one seeded set of such molecules"""
    kind, prec = case["kind"], 8 if case["precision"] == "fp64" else 4
    sample = dict(case, nmol=min(case["nmol"], 16 * CONFORMERS))
    scale = case["nmol"] / sample["nmol"]
    n = np.array([m.nao for m in _molecules(sample, 0)], np.float64)
    n4 = (scale * (n * (n + 1) / 2) ** 2 / 2).sum()
    n2 = scale * (n * n).sum()
    pts = scale * (n * LEVEL_POINTS[case["level"]]).sum()
    gn2 = scale * (LEVEL_POINTS[case["level"]] * n ** 3).sum()
    eri = dict(bytes=2 * n4 * prec, flops=27 * 30 * n4)     # 81 primitive quartets, a third screened away
    jk = dict(bytes=n4 * prec + 3 * n2 * 8, flops=8 * n4)
    xc = dict(bytes=pts * 32 + 2 * n2 * 8, flops=4 * gn2)
    setup = dict(bytes=pts * 32 + 6 * n2 * 8, flops=pts * 600 + n2 * 9 * 400)
    eig = dict(bytes=8 * n2 * 8, flops=scale * 15 * (n ** 3).sum())
    its = 20 if kind in ("nanodft", "scf") else 7
    parts = {
        "nanodft": [(1, setup), (1, eri), (its, jk), (its, xc), (its, eig)],
        "scf": [(its, jk), (its, xc), (its, eig)],
        "generate": [(1, setup), (1, eri), (its, jk), (its, xc), (its, eig)],
        "setup": [(1, setup)], "eri": [(1, eri)], "jk": [(1, jk)], "xc": [(1, xc)],
        "grad": [(1, dict(bytes=pts * 32 + 3 * n2 * 8, flops=54 * 60 * n4 + 16 * gn2))],
    }[kind]
    return {k: float(sum(c * p[k] for c, p in parts)) for k in ("bytes", "flops")}


# ---------------------------------------------------------------------------- 64-bit values

def _b3lyp(rho, sigma):
    """B3LYP energy per volume of closed-shell rho and sigma = |grad rho|^2: 0.08 Slater,
    0.72 B88 (with its Slater part), 0.19 VWN, 0.81 LYP"""
    slater = -rho ** (4.0 / 3.0) * math.exp(-0.30305460484554375)
    n = rho / 2
    x = torch.sqrt(sigma / 4 * n ** (-8.0 / 3.0))
    b88 = -1.5 * (6 / math.pi) ** (1.0 / 3.0) * n ** (4.0 / 3.0) - \
        2 * 0.0042 * n ** (4.0 / 3.0) * x * x / (1 + 6 * 0.0042 * x * torch.asinh(x))
    p0, p1, p2, p3 = -0.10498, 0.0621813817393097900698817274255, 3.72744, 12.9352
    q0 = p0 * p0 + p0 * p2 + p3
    f = p0 * p2 / q0 - 1.0
    sq = math.sqrt(4 * p3 - p2 * p2)
    pre = p2 * (1 / sq - p0 / (q0 * sq / (p2 + 2 * p0)))
    s = (3 / (4 * math.pi * rho)) ** (1.0 / 6.0)
    vwn = rho * p1 * (torch.log(s) + f * (0.5 * torch.log(s * s + p2 * s + p3) - (1 / f + 1) * torch.log(s - p0)) +
                      pre * torch.atan(sq / (2 * s + p2)))
    A, B, C, D = 0.04918, 0.132, 0.2533, 0.349
    t = rho ** (-1.0 / 3.0)
    P = 1 / (1 + D * t)
    om = torch.exp(-C * t) * P
    dl = t * (C + D * P)
    cf = 0.3 * (3 * math.pi ** 2) ** (2.0 / 3.0)
    lyp = -A * rho * P - A * B * cf * om * rho + A * B / 72 * om * sigma * t ** 5 * (3 + 7 * dl)
    return 0.08 * slater + 0.72 * b88 + 0.19 * vwn + 0.81 * lyp


def _exact_xc(case, seed):
    s = prepare(case, seed)
    eng, V, E = s["eng"], [], []
    m = 0
    for group in _families(case, seed):
        R, dirs, ex, cf, _ = _tables(group)
        isp = dirs.abs().sum(-1)
        for k in range(len(group)):
            g0, g1 = int(eng.plan.grid_off[m]), int(eng.plan.grid_off[m + 1])
            xyz, w = eng.coords.view(-1, 3)[g0:g1], eng.weights[g0:g1]
            D = eng.plan.unpack(s["D"], m)
            v, e = torch.zeros_like(D), D.new_zeros(())
            for c0 in range(0, g1 - g0, 65536):
                d = xyz[c0:c0 + 65536, None, :] - R[k][None]
                wt = w[c0:c0 + 65536]
                prim = cf * torch.exp(-(d * d).sum(-1)[..., None] * ex)
                g, dg = prim.sum(-1), -2.0 * (prim * ex).sum(-1)
                ang = (d * dirs).sum(-1) + (1.0 - isp)
                ao = [ang * g] + [ang * d[..., x] * dg + dirs[:, x] * g for x in range(3)]
                X = ao[0] @ D
                r = [(X * a).sum(-1) for a in ao]
                rho = r[0].clamp(1e-9, 1e12).requires_grad_()
                sig = (4 * (r[1] ** 2 + r[2] ** 2 + r[3] ** 2) + 1e-20).requires_grad_()
                en = _b3lyp(rho, sig)
                vr, vg = torch.autograd.grad(en.sum(), (rho, sig))
                e = e + (r[0] * wt * (en / rho).detach()).sum()
                Y = (0.5 * vr * wt)[:, None] * ao[0]
                for x in range(3):
                    Y = Y + (4 * vg * r[1 + x] * wt)[:, None] * ao[1 + x]
                v = v + ao[0].T @ Y
            V.append((v + v.T).reshape(-1))
            E.append(e)
            m += 1
    return {"V": torch.cat(V), "E": torch.stack(E)}


def _packed(m):
    """index of pair (i, j) in the packed triangle, (m, m)"""
    i = torch.arange(m, device="cuda")
    hi, lo = torch.maximum(i[:, None], i[None]), torch.minimum(i[:, None], i[None])
    return hi * (hi + 1) // 2 + lo


def _exact_jk(case, seed):
    s = prepare(case, seed)
    eng, J, K = s["eng"], [], []
    for m in range(eng.plan.nmol):
        n = int(eng.plan.nao[m])
        n2 = n * (n + 1) // 2
        o = int(eng.plan.eri_off[m])
        M = eng.eri[o:o + n2 * (n2 + 1) // 2].double()[_packed(n2)]
        D = eng.plan.unpack(s["D"], m)
        pair = _packed(n).reshape(-1)
        G = M[pair][:, pair].view(n, n, n, n)
        J.append(torch.einsum("ijkl,ij->kl", G, D).reshape(-1))
        K.append(torch.einsum("ijkl,jk->il", G, D).reshape(-1))
    return {"J": torch.cat(J), "K": torch.cat(K)}


def _boys(m, t):
    """F_0..F_m(t): the incomplete gamma function for F_m, downward recursion"""
    ts = t.clamp_min(1e-14)
    a = torch.full_like(ts, m + 0.5)
    F = [math.gamma(m + 0.5) * torch.special.gammainc(a, ts) / (2 * ts ** (m + 0.5))]
    F[0] = torch.where(t < 1e-5, 1.0 / (2 * m + 1) - t / (2 * m + 3) + t * t / (4 * m + 10), F[0])
    e = torch.exp(-t)
    for k in range(m - 1, -1, -1):
        F.insert(0, (2 * t * F[0] + e) / (2 * k + 1))
    return F


def _eri_rows(P, quart):
    """(ij|kl) of one molecule for index vectors quart = (bra pair, ket pair): Hermite expansion,
    the derivatives of F_0 along the p directions summed over pairings"""
    z, w, C, sa, sb, di, dj = P
    b, k = quart
    dv = [di[b], dj[b], di[k], dj[k]]
    some = [bool(d.any()) for d in dv]
    dot = {(x, y): (dv[x] * dv[y]).sum(-1) for x, y in itertools.combinations(range(4), 2)}
    tot = torch.zeros(b.shape, dtype=torch.float64, device="cuda")
    for p in range(9):
        for q in range(9):
            ze, et = z[b, p], z[k, q]
            rho = ze * et / (ze + et)
            X = C[b, p] - C[k, q]
            F = _boys(sum(some), rho * (X * X).sum(-1))
            f = [F[n] * (-2 * rho) ** n for n in range(len(F))]
            f += [torch.zeros_like(rho)] * (5 - len(f))
            xd = [(X * d).sum(-1) for d in dv]
            u, v = 0.5 / ze, -0.5 / et          # derivatives with respect to Q are -d/dX
            ss = [sa[b, p], sb[b, p], sa[k, q], sb[k, q]]
            val = 0.0
            for pick in itertools.product(*[(0, 1) if s else (0,) for s in some]):
                on = [x for x in range(4) if pick[x]]
                c = 1.0
                for x in range(4):
                    # a p function's linear factor is its shift plus u d/dP
                    c = c * ((u if x < 2 else v) if pick[x] else ss[x])
                val = val + c * _pairings(on, xd, dot, f)
            # products of two linear factors on one side also meet at the same point
            if some[0] and some[1]:
                val = val + _same(dot[0, 1] * u, 2, 3, ss, v, xd, dot, f, some)
            if some[2] and some[3]:
                val = val - _same(dot[2, 3] * v, 0, 1, ss, u, xd, dot, f, some)
            if all(some):
                val = val - dot[0, 1] * u * dot[2, 3] * v * f[0]
            tot += w[b, p] * w[k, q] * 2 * math.pi ** 2.5 / (ze * et * torch.sqrt(ze + et)) * val
    return tot


def _pairings(on, xd, dot, f):
    """derivative of f_0(X) along the directions ``on``: sums over pairings of the directions"""
    r = 0.0
    for npair in range(len(on) // 2 + 1):
        for ps in _pair_sets(on, npair):
            used = [x for p in ps for x in p]
            t = f[len(on) - npair]
            for p in ps:
                t = t * dot[p]
            for x in on:
                if x not in used:
                    t = t * xd[x]
            r = r + t
    return r


def _pair_sets(on, npair):
    if npair == 0:
        return [[]]
    sets = []
    for a, b in itertools.combinations(on, 2):
        rest = [x for x in on if x not in (a, b) and x > a]
        sets += [[(a, b)] + r for r in _pair_sets(rest, npair - 1)]
    return sets


def _same(c, x, y, ss, u, xd, dot, f, some):
    r = 0.0
    for pick in itertools.product((0, 1) if some[x] else (0,), (0, 1) if some[y] else (0,)):
        on = [a for a, p in zip((x, y), pick) if p]
        t = 1.0
        for a, p in zip((x, y), pick):
            t = t * (u if p else ss[a])
        r = r + t * _pairings(on, xd, dot, f)
    return c * r


def _exact_eri(case, seed):
    fam = _families(case, seed)
    if sum(((g[0].nao * (g[0].nao + 1) / 2) ** 2) / 2 * len(g) for g in fam) > 4e7:
        return None
    eri, exch = [], []
    for group in fam:
        R, dirs, ex, cf, _ = _tables(group)
        n = group[0].nao
        i, j = torch.tril_indices(n, n, device="cuda")
        n2 = i.numel()
        bra, ket = torch.tril_indices(n2, n2, device="cuda")
        isp = dirs.abs().sum(-1) > 0
        cls = (isp[i].int() + 2 * isp[j].int())
        for k in range(len(group)):
            z, w, P, sa, sb = (a[i, j] for a in (lambda q: (q[0], q[1][0], q[2][0], q[3][0], q[4][0]))(
                _pairs(R[k:k + 1], dirs, ex, cf)))
            pairs = (z, w, P, sa, sb, dirs[i], dirs[j])
            vals = torch.zeros(bra.numel(), dtype=torch.float64, device="cuda")
            for cb, ck in itertools.product(range(4), range(4)):
                sel = ((cls[bra] == cb) & (cls[ket] == ck)).nonzero().flatten()
                for c0 in range(0, sel.numel(), 1 << 20):
                    part = sel[c0:c0 + (1 << 20)]
                    vals[part] = _eri_rows(pairs, (bra[part], ket[part]))
            M, pi = vals[_packed(n2)], _packed(n)
            # exchange list: H[(il),(jk)] = (ij|kl) + (ik|jl)
            a, l, b, c = i[bra], j[bra], i[ket], j[ket]
            H = M[pi[a, b], pi[c, l]] + M[pi[a, c], pi[b, l]]
            pad = torch.zeros((-vals.numel()) % 32, dtype=torch.float64, device="cuda")
            eri += [vals, pad]
            exch += [H, pad]
    return {"eri": torch.cat(eri), "exchange": torch.cat(exch)}


def _exact_setup(case, seed):
    S, L, enuc = [], [], []
    for group in _families(case, seed):
        R, dirs, ex, cf, _ = _tables(group)
        o = _overlap(R, dirs, ex, cf)
        li = torch.linalg.inv(torch.linalg.cholesky(o))
        S.append(o.reshape(-1))
        L.append(li.tril().reshape(-1))
        for m in group:
            d = np.sqrt(((m.coords[:, None] - m.coords[None]) ** 2).sum(-1))
            iu = np.triu_indices(m.natm, 1)
            enuc.append(float((np.outer(m.charges, m.charges)[iu] / d[iu]).sum()))
    return {"S": torch.cat(S), "T": None, "V": None, "Linv": torch.cat(L), "D0": None,
            "enuc": torch.tensor(enuc, dtype=torch.float64), "coords": None, "weights": None}


def exact(case, seed):
    """64-bit values of the single pieces, in plain torch; whole SCF runs and gradients have none"""
    f = {"xc": _exact_xc, "jk": _exact_jk, "eri": _exact_eri, "setup": _exact_setup}.get(case["kind"])
    return f(case, seed) if f else None
