"""Nuclear gradients on the B200 (b2_grad): every kernel against the host build of the same
math on the same densities, batched over uneven molecules, and the nanoDFT.grad drop-in against
the gradient oracle."""
import ctypes

import numpy as np
import pytest

from b200dft.mole import Mole, methane

pytestmark = pytest.mark.gpu

HYB = 0.2


def _mols():
    return [Mole("O 0 0 0.1173; H 0 0.7572 -0.4692; H 0 -0.7532 -0.4792"), Mole(methane(1.05)),
            Mole("N 0 0 0; C 0 0 2.6; O 2.1 0 3.9; H 0 1.9 -0.8", unit="Bohr")]


def _host_parts(hc, mol, D, W, coords, w):
    """one-electron, two-electron, exchange-correlation and nuclear parts by the host build"""
    from test_hostcheck import _p
    atm = np.ascontiguousarray(mol._atm, np.int32)
    bas = np.ascontiguousarray(mol._bas, np.int32)
    env = np.ascontiguousarray(mol._env, np.float64)
    args = (mol.natm, len(bas), _p(atm, ctypes.c_int), _p(bas, ctypes.c_int), _p(env, ctypes.c_double))
    D, W = np.ascontiguousarray(D), np.ascontiguousarray(W)
    coords, w = np.ascontiguousarray(coords), np.ascontiguousarray(w)
    g1, g2, gx = (np.zeros((mol.natm, 3)) for _ in range(3))
    assert hc.b2hc_grad_1e(*args, _p(D, ctypes.c_double), _p(W, ctypes.c_double), _p(g1, ctypes.c_double)) == 0
    assert hc.b2hc_grad_2e(*args, _p(D, ctypes.c_double), ctypes.c_double(HYB), _p(g2, ctypes.c_double)) == 0
    assert hc.b2hc_grad_xc(*args, _p(D, ctypes.c_double), ctypes.c_longlong(len(w)), _p(coords, ctypes.c_double),
                           _p(w, ctypes.c_double), _p(gx, ctypes.c_double)) == 0
    Z = mol.charges.astype(np.float64)
    dR = mol.coords[:, None, :] - mol.coords[None, :, :]
    dist = np.linalg.norm(dR, axis=2)
    np.fill_diagonal(dist, np.inf)
    gn = -(Z[:, None, None] * Z[None, :, None] * dR / dist[:, :, None] ** 3).sum(1)
    return {1: g1, 2: g2, 4: gx, 8: gn}


def test_gradient_kernels_match_host_math_batched():
    from test_hostcheck import _hc
    from b200dft.engine import RKSEngine, nuclear_gradient
    mols = _mols()
    eng = RKSEngine(mols, precision="fp64", guess="minao")
    try:
        r = eng.run_converged()
        assert bool(r["converged"].all())
        dm = []
        full = nuclear_gradient(eng.plan, eng.C, eng.mo_energy, eng.coords, eng.weights, parts=15,
                                hyb=HYB, out_dm=dm).cpu().numpy()
        parts = {p: eng.gradient(parts=p, hyb=HYB).cpu().numpy() for p in (1, 2, 4, 8)}
        P = eng.plan
        D, W = (x.cpu().numpy() for x in dm)
        # dm0 from the final orbitals is the final density of the SCF
        np.testing.assert_allclose(D[:P.n_mat], eng.D.cpu().numpy(), atol=1e-12, rtol=0)
        coords = eng.coords.cpu().numpy().reshape(-1, 3)
        w = eng.weights.cpu().numpy()
    finally:
        eng.close()
    np.testing.assert_allclose(sum(parts.values()), full, atol=1e-10, rtol=0)
    hc = _hc()
    a0 = 0
    for m, mol in enumerate(mols):
        g0, g1 = P.grid_off[m], P.grid_off[m + 1]
        ref = _host_parts(hc, mol, P.unpack(D, m), P.unpack(W, m), coords[g0:g1], w[g0:g1])
        for p, gr in ref.items():
            got = parts[p][a0:a0 + mol.natm]
            np.testing.assert_allclose(got, gr, atol=1e-9 * max(1.0, np.abs(gr).max()), rtol=0,
                                       err_msg=f"molecule {m} part {p}")
        # translation invariance holds for the integral terms; the XC term is taken on a grid that
        # does not move with the atoms (no grid response, as in the reference), so it breaks it
        analytic = sum(parts[p][a0:a0 + mol.natm] for p in (1, 2, 8))
        assert np.abs(analytic.sum(0)).max() < 1e-8
        a0 += mol.natm


def test_nanodft_grad_drop_in_matches_oracle():
    """nanoDFT(mol, opts) then grad(mol, coords, weight, mo_coeff, mo_energy) (nanoDFT.py:636)"""
    from oracle import grad as ograd
    from b200dft.nanodft import grad, nanoDFT, nanoDFT_options
    mol = _mols()[0]
    opts, _ = nanoDFT_options(its=30, mol_str="water")
    _, (_, _, mo_energy, mo_coeff, coords, weights) = nanoDFT(mol, opts)
    g = grad(mol, coords, weights, mo_coeff, mo_energy)
    ref = ograd.gradient(mol, mo_coeff, mo_energy, coords, weights)
    assert np.abs(ref).max() > 1e-2
    np.testing.assert_allclose(g, ref, atol=1e-6, rtol=0)     # oracle truncation ~1e-8


@pytest.mark.parametrize("heavy, odd", [(1, True), (2, False), (4, True), (9, False)])
def test_gradient_slices_over_sizes(heavy, odd):
    """two- and one-electron parts against the host build of the same slices: one to several
    32-ket chunks per class, 8 / 16 / 32 lanes of nuclei, shells off the STO-3G pattern, a random
    density.  Same formulas in another order of float64 sums: 1e-10 of the largest component."""
    import torch
    from test_hostcheck import _gs_args, _hc, _p, odd_shells
    from b200dft.engine import Plan
    from b200dft._lib import check, lib, ptr, stream_handle
    from b200dft.molgen import random_molecule
    mol = Mole(random_molecule(np.random.default_rng(heavy), heavy))
    mol = odd_shells(mol) if odd else mol
    hc, N = _hc(), mol.nao
    rng = np.random.default_rng(5)
    D, W = (np.ascontiguousarray(a + a.T) for a in rng.normal(size=(2, N, N)) * 0.3)
    plan = Plan([mol])
    try:
        t = lambda a: torch.from_numpy(a.reshape(-1)).cuda()
        d, w = t(D), t(W)
        got = []
        for parts in (1, 2):
            g = torch.full((mol.natm, 3), float("nan"), dtype=torch.float64, device="cuda")
            check(lib().b2_grad(plan.h, parts, HYB, None, None, None, None, ptr(d), ptr(w), ptr(g), stream_handle()),
                  "b2_grad")
            got.append(g.cpu().numpy())
    finally:
        plan.close()
    ref1, ref2, n = np.zeros((mol.natm, 3)), np.zeros((mol.natm, 3)), np.zeros(2, np.int32)
    keep, a = _gs_args(mol, D, W)
    assert hc.b2hc_grad_1e_super(*a, _p(ref1, ctypes.c_double)) == 0
    keep, a = _gs_args(mol, D)
    assert hc.b2hc_grad_2e_super(*a, ctypes.c_double(HYB), _p(ref2, ctypes.c_double), _p(n, ctypes.c_int)) == 0
    for g, ref in zip(got, (ref1, ref2)):
        np.testing.assert_allclose(g, ref, atol=1e-10 * max(1.0, np.abs(ref).max()), rtol=0)


def test_gradient_xc_odd_shells():
    """the exchange-correlation part with shells off the STO-3G pattern against the host math, same
    tolerance as for the regular ones"""
    import torch
    from test_gpu_kernels import _odd_mols
    from test_hostcheck import _gs_args, _hc, _p
    from b200dft.engine import RKSEngine
    from b200dft._lib import check, lib, ptr, stream_handle
    mols = _odd_mols()
    eng = RKSEngine(mols, level=0, precision="fp64")
    eng.device_setup()
    P, rng, hc = eng.plan, np.random.default_rng(25), _hc()
    Ds = []
    for m in mols:
        C = rng.normal(size=(m.nao, m.nao)) * 0.1 + np.diag(rng.uniform(0.5, 1.0, m.nao))
        Ds.append(2.0 * C[:, :m.nelectron // 2] @ C[:, :m.nelectron // 2].T)
    d = torch.from_numpy(P.pack(Ds)).cuda()
    w, g = torch.zeros_like(d), torch.zeros(sum(m.natm for m in mols), 3, dtype=torch.float64, device="cuda")
    check(lib().b2_grad(P.h, 4, HYB, None, None, ptr(eng.coords), ptr(eng.weights), ptr(d), ptr(w), ptr(g),
                        stream_handle()), "b2_grad")
    got, a0, xyz, wt = g.cpu().numpy(), 0, eng.coords.cpu().numpy().reshape(-1, 3), eng.weights.cpu().numpy()
    for k, (m, D) in enumerate(zip(mols, Ds)):
        gp = slice(P.grid_off[k], P.grid_off[k + 1])
        ref, (x, q, D) = np.zeros((m.natm, 3)), (np.ascontiguousarray(a) for a in (xyz[gp], wt[gp], D))
        keep, a = _gs_args(m, D)
        assert hc.b2hc_grad_xc(*a, ctypes.c_longlong(len(q)), _p(x, ctypes.c_double), _p(q, ctypes.c_double),
                               _p(ref, ctypes.c_double)) == 0
        np.testing.assert_allclose(got[a0:a0 + m.natm], ref, atol=1e-9 * max(1.0, np.abs(ref).max()), rtol=0)
        a0 += m.natm
    eng.close()


def test_gradient_many_tasks():
    """two- and one-electron parts of a batch in which every warp takes several slices, neighbours of
    other sizes: each molecule as alone.  Sums of the same float64 terms in another order (atomics)."""
    import torch
    from test_gpu_kernels import _big_batch
    from b200dft.engine import Plan
    from b200dft._lib import check, lib, ptr, stream_handle
    kinds, order = _big_batch()
    rng = np.random.default_rng(31)
    mats = [[a + a.T for a in rng.normal(size=(2, m.nao, m.nao)) * 0.3] for m in kinds]

    def parts(which):
        plan = Plan([kinds[k] for k in which])
        d, w = (torch.from_numpy(plan.pack([mats[k][i] for k in which])).cuda() for i in (0, 1))
        g = torch.zeros(2, sum(kinds[k].natm for k in which), 3, dtype=torch.float64, device="cuda")
        for i, part in enumerate((1, 2)):
            check(lib().b2_grad(plan.h, part, HYB, None, None, None, None, ptr(d), ptr(w), ptr(g[i]),
                                stream_handle()), "b2_grad")
        out = g.cpu().numpy()
        plan.close()
        return out

    alone = [parts([k]) for k in range(len(kinds))]
    got, a0 = parts(order), 0
    for k in order:
        n = kinds[k].natm
        for i in (0, 1):
            np.testing.assert_allclose(got[i, a0:a0 + n], alone[k][i], rtol=0,
                                       atol=1e-11 * max(1.0, np.abs(alone[k][i]).max()))
        a0 += n
