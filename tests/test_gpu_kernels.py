"""GPU parity: every kernel through the C ABI against the oracle / reference golden data."""
import ctypes
import numpy as np
import pytest
import torch

from conftest import golden
from oracle import eri as oeri, rks
from b200dft.mole import Mole, methane
from b200dft.molgen import config2_molecule, random_molecule
from b200dft.engine import RKSEngine, HostSetup, Plan
from b200dft._lib import lib, check, ptr, stream_handle

pytestmark = pytest.mark.gpu

NAMES = ("h2", "ch4", "water", "tree3")


def _mols():
    gs = [golden(f"eri_ref_{n}.npz") for n in NAMES]
    return [Mole(str(g["atom"]), unit=str(g["unit"])) for g in gs], gs


def _eri(mols, prec, cuda, raw=False):
    """device s8 lists; the plan pads each molecule's list to 32 entries"""
    P = Plan(mols)
    out = torch.full((P.n_eri,), float("nan"), dtype=torch.float64 if prec == 64 else torch.float32,
                     device=cuda)
    check(lib().b2_eri_s8(P.h, prec, ptr(out), stream_handle()), "eri")
    torch.cuda.synchronize()
    v = out.double().cpu().numpy()
    if raw:
        return P, v
    return P, np.concatenate([v[P.eri_off[i]:P.eri_off[i] + oeri.n_s8(int(P.nao[i]))] for i in range(P.nmol)])


def test_eri_s8_fp64_vs_reference(cuda):
    mols, gs = _mols()
    P, v = _eri(mols, 64, cuda)
    assert not np.isnan(v).any()
    ref = np.concatenate([g["s8"] for g in gs])
    err = np.abs(v - ref).max()
    assert err <= 1e-10, err                       # north-star gate: 1e-10 abs


def test_eri_s8_fp32(cuda):
    mols, gs = _mols()
    P, v = _eri(mols, 32, cuda)
    ref = np.concatenate([g["s8"] for g in gs])
    assert np.abs(v - ref).max() < 5e-6


def test_eri_config2_full(cuda):
    g = golden("eri_ref_sample_config2.npz")
    m = Mole(str(g["atom"]))
    P, v = _eri([m], 64, cuda)
    assert len(v) == int(g["n"])
    np.testing.assert_allclose(v[g["idx"]], g["val"], atol=1e-10, rtol=0)
    assert abs(v.sum() - float(g["total"])) <= 1e-9 * abs(float(g["total"]))
    assert abs((v * v).sum() - float(g["sumsq"])) <= 1e-9 * float(g["sumsq"])
    ref = oeri.eri_s8(m)
    assert np.abs(v - ref).max() <= 1e-10


def test_int2e_sph_s8_single(cuda):
    m = Mole(methane())
    out = torch.zeros(oeri.n_s8(m.nao), dtype=torch.float64, device=cuda)
    atm = np.ascontiguousarray(m._atm, np.int32)
    bas = np.ascontiguousarray(m._bas, np.int32)
    env = np.ascontiguousarray(m._env)
    check(lib().b2_int2e_sph_s8(ptr(atm), m.natm, ptr(bas), m.nbas, ptr(env), len(env), 64, ptr(out),
                                stream_handle()), "int2e")
    np.testing.assert_allclose(out.cpu().numpy(), golden("eri_ref_ch4.npz")["s8"], atol=1e-10)


def _sym_random(n, rng):
    a = rng.normal(size=(n, n))
    return (a + a.T) / 2


@pytest.mark.parametrize("prec", [64, 32])
def test_jk_parity(cuda, prec):
    mols, gs = _mols()
    P, v = _eri(mols, prec, cuda, raw=True)
    rng = np.random.default_rng(0)
    Ds = [_sym_random(m.nao, rng) for m in mols]
    eri_t = torch.from_numpy(v).to(cuda).to(torch.float64 if prec == 64 else torch.float32)
    D = torch.from_numpy(P.pack(Ds)).to(cuda)
    J = torch.zeros(P.n_mat, dtype=torch.float64, device=cuda)
    K = torch.zeros_like(J)
    for chunk in (0, 64, 1000):               # several work splits give the same answer
        if chunk:
            P.set_jk_chunk(chunk)
        check(lib().b2_jk_s8(P.h, prec, None, ptr(eri_t), ptr(D), ptr(J), ptr(K), stream_handle()), "jk")
        torch.cuda.synchronize()
        Jh, Kh = J.cpu().numpy(), K.cpu().numpy()
        for mi, (m, g) in enumerate(zip(mols, gs)):
            _, Jr, Kr = rks.jk_from_s8(Ds[mi], g["s8"], m.nao)
            tol = 1e-10 if prec == 64 else 2e-5 * max(1.0, np.abs(Jr).max())
            np.testing.assert_allclose(P.unpack(Jh, mi), Jr, atol=tol)
            np.testing.assert_allclose(P.unpack(Kh, mi), Kr, atol=tol)


@pytest.mark.parametrize("prec", [64, 32])
def test_jk_pairs_parity(cuda, prec):
    # J/K as two products over the s8 list and the exchange list, vs the s8 semantics oracle;
    # inactive molecules keep their previous J/K
    mols, gs = _mols()
    P, v = _eri(mols, prec, cuda, raw=True)
    dt = torch.float64 if prec == 64 else torch.float32
    eri_t = torch.from_numpy(v).to(cuda).to(dt)
    exch = torch.full_like(eri_t, float("nan"))
    check(lib().b2_jk_exchange(P.h, prec, ptr(eri_t), ptr(exch), stream_handle()), "exchange")
    rng = np.random.default_rng(1)
    Ds = [_sym_random(m.nao, rng) for m in mols]
    D = torch.from_numpy(P.pack(Ds)).to(cuda)
    J = torch.full((P.n_mat,), 7.0, dtype=torch.float64, device=cuda)
    K = torch.full_like(J, 7.0)
    active = torch.tensor([1, 0, 1, 1], dtype=torch.int32, device=cuda)
    check(lib().b2_jk_pairs(P.h, prec, ptr(active), ptr(eri_t), ptr(exch), ptr(D), ptr(J), ptr(K),
                            stream_handle()), "jk_pairs")
    torch.cuda.synchronize()
    st = ctypes.c_int(-1)
    check(lib().b2_jk_status(1, ctypes.byref(st)), "b2_jk_status")
    assert st.value == 0                       # no row-group copy wait gave up
    Jh, Kh = J.cpu().numpy(), K.cpu().numpy()
    for mi, (m, g) in enumerate(zip(mols, gs)):
        if mi == 1:
            assert np.all(P.unpack(Jh, mi) == 7.0) and np.all(P.unpack(Kh, mi) == 7.0)
            continue
        _, Jr, Kr = rks.jk_from_s8(Ds[mi], g["s8"], m.nao)
        tol = 1e-10 if prec == 64 else 2e-5 * max(1.0, np.abs(Jr).max())
        np.testing.assert_allclose(P.unpack(Jh, mi), Jr, atol=tol)
        np.testing.assert_allclose(P.unpack(Kh, mi), Kr, atol=tol)
    # exchange list entries: H[(il),(jk)] = (ij|kl) + (ik|jl)
    m, g = mols[2], gs[2]
    N = m.nao
    full = oeri.unpack_s8(g["s8"], N)
    o = int(P.eri_off[2])
    X = exch[o:o + oeri.n_s8(N)].double().cpu().numpy()
    pr = [(i, l) for i in range(N) for l in range(i + 1)]
    e = 0
    for a, (i, l) in enumerate(pr):
        for (j, k) in pr[:a + 1]:
            ref = full[i, j, k, l] + full[i, k, j, l]
            assert abs(X[e] - ref) <= (1e-12 if prec == 64 else 1e-6) * max(1.0, abs(ref))
            e += 1


def test_ao_eval_and_xc(cuda):
    mols = [Mole(methane()), Mole("O 0 0 0.1173; H 0 0.7572 -0.4692; H 0 -0.7572 -0.4692")]
    eng = RKSEngine(mols, level=0, precision="fp64", setups=[HostSetup(m, 0) for m in mols])
    eng.compute_ao()
    torch.cuda.synchronize()
    ao = eng.ao.cpu().numpy()
    for mi, (m, s) in enumerate(zip(mols, eng.setups)):
        G, N = len(s.weights), m.nao
        a = ao[eng.plan.ao_off[mi]:eng.plan.ao_off[mi] + 4 * G * N].reshape(4, G, N)
        np.testing.assert_allclose(a, rks.ao_values(m, s.coords), atol=1e-12)
    eng.D.copy_(eng.D0)
    for fn in (eng.xc_from_ao, eng.xc):          # stored-AO and on-the-fly-AO paths
        eng.Vxc.zero_()
        fn()
        torch.cuda.synchronize()
        for mi, (m, s) in enumerate(zip(mols, eng.setups)):
            exc, V, _ = rks.exchange_correlation(s.D0, rks.ao_values(m, s.coords), s.weights)
            assert abs(eng.exc[mi].item() - exc) < 1e-10
            np.testing.assert_allclose(eng.plan.unpack(eng.Vxc.cpu().numpy(), mi), V, atol=1e-10)
    eng.close()


@pytest.mark.parametrize("prec", ["fp64", "mixed"])
def test_xc_direct_sizes(cuda, prec):
    # molecules in every orbital bucket (nao 5..65) through the on-the-fly AO path
    rng = np.random.default_rng(4)
    mols = [Mole(random_molecule(rng, k)) for k in (1, 3, 5, 7, 9)]
    setups = [HostSetup(m, 0) for m in mols]
    eng = RKSEngine(mols, level=0, precision=prec, setups=setups)
    eng.D.copy_(eng.D0)
    eng.xc()
    torch.cuda.synchronize()
    tol = 1e-9 if prec == "fp64" else 2e-5
    for mi, (m, s) in enumerate(zip(mols, setups)):
        exc, V, _ = rks.exchange_correlation(s.D0, rks.ao_values(m, s.coords), s.weights)
        assert abs(eng.exc[mi].item() - exc) < tol * max(1, abs(exc))
        np.testing.assert_allclose(eng.plan.unpack(eng.Vxc.cpu().numpy(), mi), V, atol=tol * 10)
    eng.close()


def test_xc_tensor_core_vs_cuda_core(cuda):
    # tcgen05 split-TF32 kernel against the float32 CUDA-core kernel and the float64 oracle,
    # every orbital bucket (nao 5..65), several 128-point tiles per CTA, a converged-like D
    rng = np.random.default_rng(11)
    mols = [Mole(random_molecule(rng, k)) for k in (1, 2, 4, 6, 8, 9)]
    setups = [HostSetup(m, 0) for m in mols]
    eng = RKSEngine(mols, level=0, precision="mixed", setups=setups)
    eng.D.copy_(eng.D0)
    got = {}
    for impl in (1, 2, 0):               # CUDA-core, one-launch tensor-core, per-bucket persistent
        check(lib().b2_plan_set_xc_impl(eng.plan.h, impl), "b2_plan_set_xc_impl")
        eng.xc()
        torch.cuda.synchronize()
        got[impl] = (eng.exc.cpu().numpy().copy(), eng.Vxc.cpu().numpy().copy())
    st = ctypes.c_int(-1)
    check(lib().b2_xc_tc_status(1, ctypes.byref(st)), "b2_xc_tc_status")
    assert st.value == 0
    for mi, (m, s) in enumerate(zip(mols, setups)):
        exc, V, _ = rks.exchange_correlation(s.D0, rks.ao_values(m, s.coords), s.weights)
        Vt = eng.plan.unpack(got[0][1], mi)
        Vs = eng.plan.unpack(got[1][1], mi)
        # float32 quality: relative 2e-6 on E_xc, 2e-5 * max|V| on V
        assert abs(got[0][0][mi] - exc) < 2e-6 * abs(exc)
        np.testing.assert_allclose(Vt, V, atol=2e-5 * np.abs(V).max())
        np.testing.assert_allclose(Vt, Vs, atol=2e-5 * np.abs(V).max())
        np.testing.assert_allclose(Vt, Vt.T, atol=1e-12)
        assert abs(got[2][0][mi] - exc) < 2e-6 * abs(exc)
        np.testing.assert_allclose(eng.plan.unpack(got[2][1], mi), V, atol=2e-5 * np.abs(V).max())
    eng.close()


def test_xc_work_queue_items_active_and_subset(cuda):
    # the per-bucket persistent kernel: several tile counts per work item, inactive molecules
    # left untouched, and a molecule subset (compacted items) give the same V and E_xc
    rng = np.random.default_rng(12)
    mols = [Mole(random_molecule(rng, k)) for k in (9, 1, 5, 3, 7, 2, 8)]
    eng = RKSEngine(mols, level=0, precision="mixed", guess="minao")
    eng.device_setup()
    eng.D.copy_(eng.D0)
    P = eng.plan
    eng.xc()
    torch.cuda.synchronize()
    ref_e, ref_v = eng.exc.cpu().numpy().copy(), eng.Vxc.cpu().numpy().copy()
    for tiles in (1, 3, 16):
        check(lib().b2_plan_set_xc_tiles(P.h, tiles), "b2_plan_set_xc_tiles")
        eng.xc()
        torch.cuda.synchronize()
        np.testing.assert_allclose(eng.exc.cpu().numpy(), ref_e, rtol=1e-6)
        np.testing.assert_allclose(eng.Vxc.cpu().numpy(), ref_v, atol=1e-5 * np.abs(ref_v).max())
    check(lib().b2_plan_set_xc_tiles(P.h, 0), "b2_plan_set_xc_tiles")
    act = torch.tensor([1, 0, 1, 0, 1, 1, 0], dtype=torch.int32, device=cuda)
    eng.Vxc.fill_(7.0)
    eng.exc.fill_(7.0)
    eng.xc(active=act)
    torch.cuda.synchronize()
    V, E = eng.Vxc.cpu().numpy(), eng.exc.cpu().numpy()
    for mi in range(len(mols)):
        if act[mi].item():
            assert abs(E[mi] - ref_e[mi]) <= 1e-6 * abs(ref_e[mi])
            np.testing.assert_allclose(P.unpack(V, mi), P.unpack(ref_v, mi), atol=1e-5 * np.abs(ref_v).max())
        else:
            assert E[mi] == 7.0 and np.all(P.unpack(V, mi) == 7.0)
    idx = np.array([0, 3, 6], np.int32)
    check(lib().b2_plan_set_subset(P.h, ptr(idx), len(idx)), "b2_plan_set_subset")
    sub_act = torch.zeros(len(mols), dtype=torch.int32, device=cuda)
    sub_act[torch.from_numpy(idx.astype(np.int64)).to(cuda)] = 1
    eng.xc(active=sub_act)
    torch.cuda.synchronize()
    check(lib().b2_plan_set_subset(P.h, None, 0), "b2_plan_set_subset")
    for mi in idx:
        np.testing.assert_allclose(P.unpack(eng.Vxc.cpu().numpy(), mi), P.unpack(ref_v, mi),
                                   atol=1e-5 * np.abs(ref_v).max())
    st = ctypes.c_int(-1)
    check(lib().b2_xc_tc_status(1, ctypes.byref(st)), "b2_xc_tc_status")
    assert st.value == 0
    eng.close()


def test_b3lyp_entry(cuda):
    rng = np.random.default_rng(0)
    n = 10000
    rho = np.zeros((4, n))
    rho[0] = 10 ** rng.uniform(-12, 3, n)
    rho[1:] = rng.normal(size=(3, n)) * rho[0] ** (4 / 3)
    r = torch.from_numpy(rho).to(cuda)
    e, vr, vg = (torch.zeros(n, dtype=torch.float64, device=cuda) for _ in range(3))
    check(lib().b2_b3lyp(n, ptr(r), ptr(e), ptr(vr), ptr(vg), stream_handle()), "b3lyp")
    torch.cuda.synchronize()
    e0, vr0, vg0 = rks.b3lyp(rho)
    np.testing.assert_allclose(e.cpu().numpy(), e0, rtol=1e-12)
    np.testing.assert_allclose(vr.cpu().numpy(), vr0, rtol=1e-12)
    np.testing.assert_allclose(vg.cpu().numpy(), vg0, rtol=1e-10)


def test_chol_inv(cuda):
    mols, _ = _mols()
    eng_setups = [HostSetup(m, 0) for m in mols]
    P = Plan(mols)
    S = torch.from_numpy(P.pack([s.S for s in eng_setups])).to(cuda)
    L = torch.zeros_like(S)
    st = torch.zeros(len(mols), dtype=torch.int32, device=cuda)
    check(lib().b2_chol_inv(P.h, ptr(S), ptr(L), ptr(st), stream_handle()), "chol")
    torch.cuda.synchronize()
    assert (st.cpu().numpy() == 0).all()
    for mi, s in enumerate(eng_setups):
        np.testing.assert_allclose(P.unpack(L.cpu().numpy(), mi), s.L_inv, atol=1e-10)


@pytest.mark.parametrize("heavy", [0, 1, 2, 3, 5, 7, 9])
def test_xc_float64_sizes(cuda, heavy):
    """float64 XC (matrix-instruction products over orbitals rounded up to 8, tiles of 32 points)
    for molecules of every orbital bucket beside a water molecule, all molecules and a subset
    active, against the oracle.  Sums of ~1e4 float64 terms of the size of V: 1e-11 relative."""
    rng = np.random.default_rng(40 + heavy)
    mols = [Mole("H 0 0 0; H 0 0 0.74") if heavy == 0 else Mole(random_molecule(rng, heavy)),
            Mole("O 0 0 0.1173; H 0 0.7572 -0.4692; H 0 -0.7572 -0.4692")]
    setups = [HostSetup(m, 0) for m in mols]
    eng = RKSEngine(mols, level=0, precision="fp64", setups=setups)
    ref, Ds = [], []
    for m, s in zip(mols, setups):
        C = rng.normal(size=(m.nao, m.nao)) * 0.1 + np.diag(rng.uniform(0.5, 1.0, m.nao))
        D = 2.0 * C[:, :m.nelectron // 2] @ C[:, :m.nelectron // 2].T
        Ds.append(D)
        ref.append(rks.exchange_correlation(D, rks.ao_values(m, s.coords), s.weights)[:2])
    D = torch.from_numpy(eng.plan.pack(Ds)).to(cuda)
    for act in ((1, 1), (0, 1)):
        eng.Vxc.fill_(-7.0)
        eng.exc.fill_(-7.0)
        eng.xc(D, active=torch.tensor(act, dtype=torch.int32, device=cuda))
        V, E = eng.Vxc.cpu().numpy(), eng.exc.cpu().numpy()
        for k, (Er, Vr) in enumerate(ref):
            if act[k]:
                np.testing.assert_allclose(eng.plan.unpack(V, k), Vr, atol=1e-11 * max(1.0, np.abs(Vr).max()), rtol=0)
                assert abs(E[k] - Er) <= 1e-11 * abs(Er)
            else:
                assert (eng.plan.unpack(V, k) == -7.0).all() and E[k] == -7.0
    eng.close()


@pytest.mark.parametrize("nmol", [1, 2, 5, 24])
def test_xc_run_lengths(cuda, nmol):
    """runs of tiles shortened to a small batch's share of the GPU (half the configured length and
    more, with short last runs) against items of exactly one tile, whole batch and last molecule
    alone.  float32 accumulators over at most 16 tiles: 1e-6 of E_xc, 1e-5 of
    max|V|, as for the tile counts above."""
    rng = np.random.default_rng(60 + nmol)
    mols = [Mole(random_molecule(rng, int(k))) for k in rng.integers(1, 10, size=nmol)]
    eng = RKSEngine(mols, level=0, precision="mixed", guess="minao", tuned=False)
    eng.device_setup()
    eng.D.copy_(eng.D0)
    P, got = eng.plan, {}
    for tiles in (16, 1):
        if tiles > 1:
            counts = np.full(5, tiles, np.int32)
            check(lib().b2_plan_set_xc_bucket_tiles(P.h, ptr(counts)), "b2_plan_set_xc_bucket_tiles")
        else:
            check(lib().b2_plan_set_xc_tiles(P.h, tiles), "b2_plan_set_xc_tiles")
        eng.xc()
        torch.cuda.synchronize()
        got[tiles] = (eng.exc.cpu().numpy().copy(), eng.Vxc.cpu().numpy().copy())
        idx = np.array([nmol - 1], np.int32)
        check(lib().b2_plan_set_subset(P.h, ptr(idx), 1), "b2_plan_set_subset")
        act = torch.zeros(nmol, dtype=torch.int32, device=cuda)
        act[nmol - 1] = 1
        eng.xc(active=act)
        torch.cuda.synchronize()
        check(lib().b2_plan_set_subset(P.h, None, 0), "b2_plan_set_subset")
        got[tiles] += (eng.exc.cpu().numpy().copy(), eng.Vxc.cpu().numpy().copy())
    vmax = np.abs(got[1][1]).max()
    for k in (0, 2):
        np.testing.assert_allclose(got[16][k], got[1][k], rtol=1e-6)
        np.testing.assert_allclose(got[16][k + 1], got[1][k + 1], atol=1e-5 * vmax)
    st = ctypes.c_int(-1)
    check(lib().b2_xc_tc_status(1, ctypes.byref(st)), "b2_xc_tc_status")
    assert st.value == 0
    eng.close()


@pytest.mark.parametrize("prec, tol", [(64, 1e-11), (32, 5e-6)])
def test_eri_batch_sizes(cuda, prec, tol):
    """batched integrals at the edges of the super-shell kernels: s shells only, one sp shell, more
    than one chunk of 32 kets in every class, shells off the STO-3G pattern; each entry written
    and the padding between the lists left alone"""
    from test_hostcheck import odd_shells
    water = Mole("O 0 0 0.1173; H 0 0.7572 -0.4692; H 0 -0.7572 -0.4692")
    rng = np.random.default_rng(17)
    mols = [Mole("H 0 0 0; H 0 0 0.74"), water, odd_shells(water),
            Mole("; ".join(f"H {0.9 * (k % 3)} {0.8 * (k // 3)} 0" for k in range(9)) + "; H 0 0 1.1"),
            odd_shells(Mole(random_molecule(rng, 4))), Mole(random_molecule(rng, 9))]
    P = Plan(mols)
    dt = torch.float64 if prec == 64 else torch.float32
    out = torch.full((P.n_eri,), float("nan"), dtype=dt, device=cuda)
    check(lib().b2_eri_s8(P.h, prec, ptr(out), stream_handle()), "b2_eri_s8")
    v = out.double().cpu().numpy()
    ends = list(P.eri_off[1:]) + [P.n_eri]
    for k, m in enumerate(mols):
        ref, o = oeri.eri_s8(m), int(P.eri_off[k])
        np.testing.assert_allclose(v[o:o + len(ref)], ref, atol=tol, rtol=0)
        assert np.isnan(v[o + len(ref):ends[k]]).all()
    P.close()


@pytest.mark.parametrize("heavy", [1, 3, 5, 7, 9])
def test_xc_float32_independent_of_batch(cuda, heavy):
    """a molecule's float32 V and E_xc alone, in a batch that fills the GPU and with all but it
    compacted away: its tiles are cut and summed the same way in all three, and only the order of
    float64 additions of whole sums differs (N <= 5 per entry at 16 tiles or more: 1e-14 of max|V|,
    1e-13 of E_xc over ~2e3 tiles' points)"""
    rng = np.random.default_rng(70 + heavy)
    one = Mole(random_molecule(rng, heavy))
    got = []
    for mols in ([one], [one] + [Mole(random_molecule(rng, int(k))) for k in rng.integers(1, 10, size=96)]):
        eng = RKSEngine(mols, level=1, precision="mixed", guess="minao", tuned=False)
        eng.device_setup()
        P, counts = eng.plan, np.full(5, 32, np.int32)
        check(lib().b2_plan_set_xc_bucket_tiles(P.h, ptr(counts)), "b2_plan_set_xc_bucket_tiles")
        for subset in (0, 1):
            act = None
            if subset:
                idx = np.zeros(1, np.int32)
                check(lib().b2_plan_set_subset(P.h, ptr(idx), 1), "b2_plan_set_subset")
                act = torch.zeros(len(mols), dtype=torch.int32, device=cuda)
                act[0] = 1
            eng.xc(eng.D0, active=act)
            torch.cuda.synchronize()
            got.append((eng.exc[0].item(), P.unpack(eng.Vxc.cpu().numpy(), 0).copy()))
        check(lib().b2_plan_set_subset(P.h, None, 0), "b2_plan_set_subset")
        eng.close()
    for e, v in got[1:]:
        assert abs(e - got[0][0]) <= 1e-13 * abs(e)
        np.testing.assert_allclose(v, got[0][1], atol=1e-14 * np.abs(v).max(), rtol=0)


@pytest.fixture(scope="module")
def both_precisions(cuda):
    """float32 and float64 engines of 256 molecules, and the float64 path's converged densities"""
    from b200dft.molgen import config3_batch
    mols = [Mole(s) for s in config3_batch(256, seed=7)]
    e64, e32 = (RKSEngine(mols, level=0, precision=p, guess="minao") for p in ("fp64", "mixed"))
    e64.prepare()
    assert bool(e64.run_converged()["converged"].all())
    e32.prepare()
    yield e64, e32, e64.D.clone()
    e64.close()
    e32.close()


def test_eri_float32_error(both_precisions):
    """float32 integrals no further from float64 than kernels that sum one l class at a time are,
    over the same 256 molecules: 7.1e-7 at most, 9.0e-8 in the 2-norm (measured on those kernels)"""
    e64, e32, _ = both_precisions
    P, err, norm = e64.plan, 0.0, [0.0, 0.0]
    for m in range(P.nmol):
        o = int(P.eri_off[m])
        ref = e64.eri[o:o + oeri.n_s8(int(P.nao[m]))]
        d = e32.eri[o:o + len(ref)].double() - ref
        err = max(err, d.abs().max().item())
        norm[0] += d.pow(2).sum().item()
        norm[1] += ref.pow(2).sum().item()
    assert err <= 7.1e-7 and norm[0] ** 0.5 <= 9.0e-8 * norm[1] ** 0.5


def _energies(eng, mats, D):
    """sum over each molecule's entries of mats o D"""
    P, a, d = eng.plan, mats.cpu().numpy(), D.cpu().numpy()
    return np.array([(P.unpack(a, m) * P.unpack(d, m)).sum() for m in range(P.nmol)])


def test_jk_energy_float32_error(both_precisions):
    """Coulomb and exchange energy of float32 lists at a float64 density: errors that add up with one
    sign show here.  No further from float64 than lists summed one l class at a time: mean error
    of E_J 5.9e-6 Ha, of E_K 2.0e-7 Ha (measured on those kernels, the same molecules)"""
    e64, e32, D = both_precisions
    for e in (e64, e32):
        e.jk(D=D)
    dj = 0.5 * (_energies(e32, e32.J, D) - _energies(e64, e64.J, D))
    dk = -0.25 * 0.2 * (_energies(e32, e32.K, D) - _energies(e64, e64.K, D))
    assert np.abs(dj).mean() <= 5.9e-6 and np.abs(dk).mean() <= 2.0e-7


def test_xc_energy_float32_error(both_precisions):
    """E_xc of the tensor-core path at a float64 density: the mean error, which has one sign, no
    larger than with the tile's columns in the order of the orbitals (8.7e-6 Ha, measured on the
    same molecules)"""
    e64, e32, D = both_precisions
    for e in (e64, e32):
        e.xc(D=D)
    assert (e32.exc - e64.exc).abs().mean().item() <= 8.7e-6


def _odd_mols():
    """shells off the STO-3G pattern (a p shell without its s, s shells of one and two primitives)
    in every orbital bucket: the float32 kernel's columns then hold p functions of their own"""
    from test_hostcheck import odd_shells
    rng = np.random.default_rng(23)
    return [odd_shells(Mole("O 0 0 0.1173; H 0 0.7572 -0.4692; H 0 -0.7572 -0.4692"))] + \
        [odd_shells(Mole(random_molecule(rng, k))) for k in (2, 4, 6, 8, 9)]


@pytest.mark.parametrize("prec, etol, vtol", [("fp64", 1e-11, 1e-11), ("mixed", 2e-6, 2e-5)])
def test_xc_odd_shells(cuda, prec, etol, vtol):
    """XC with shells off the STO-3G pattern against the oracle (tolerances as for the regular ones)"""
    mols = _odd_mols()
    eng = RKSEngine(mols, level=0, precision=prec)
    eng.device_setup()
    P, w = eng.plan, eng.weights.cpu().numpy()
    xyz = eng.coords.cpu().numpy().reshape(-1, 3)
    assert len({(n - 1) // 16 for n in P.nao}) >= 4
    rng = np.random.default_rng(24)
    Ds = []
    for m in mols:
        C = rng.normal(size=(m.nao, m.nao)) * 0.1 + np.diag(rng.uniform(0.5, 1.0, m.nao))
        Ds.append(2.0 * C[:, :m.nelectron // 2] @ C[:, :m.nelectron // 2].T)
    eng.xc(torch.from_numpy(P.pack(Ds)).to(cuda))
    V, E = eng.Vxc.cpu().numpy(), eng.exc.cpu().numpy()
    for k, m in enumerate(mols):
        g = slice(P.grid_off[k], P.grid_off[k + 1])
        Er, Vr, _ = rks.exchange_correlation(Ds[k], rks.ao_values(m, xyz[g]), w[g])
        np.testing.assert_allclose(P.unpack(V, k), Vr, atol=vtol * max(1.0, np.abs(Vr).max()), rtol=0)
        assert abs(E[k] - Er) <= etol * abs(Er)
    eng.close()


def _three_primitives(m):
    """the molecule with its shorter contractions filled up with primitives of coefficient zero (the
    host formulas take three)"""
    t = Mole.__new__(Mole)
    t.__dict__.update(m.__dict__)
    t._bas, env = m._bas.copy(), m._env
    for b in t._bas:
        ex, c = env[b[5]:b[5] + b[2]], env[b[6]:b[6] + b[2]]
        b[5], b[6] = len(env), len(env) + 3
        env = np.concatenate([env, ex, np.ones(3 - b[2]), c, np.zeros(3 - b[2])])
        b[2] = 3
    t._env = env
    return t


def test_int1e_odd_shells(cuda):
    """one-electron matrices with shells off the STO-3G pattern against the host formulas"""
    from b200dft.int1e import int1e
    mols = _odd_mols()
    eng = RKSEngine(mols, level=0, precision="fp64")
    eng.device_setup()
    for k, m in enumerate(mols):
        for name, ref in zip("STV", int1e(_three_primitives(m))):
            got = eng.plan.unpack(getattr(eng, name).cpu().numpy(), k)
            np.testing.assert_allclose(got, ref, atol=1e-11 * max(1.0, np.abs(ref).max()), rtol=0, err_msg=name)
    eng.close()


def _super_shells(m):
    """(s-only, sp) super shells of a molecule with STO-3G shells or those of odd_shells"""
    e = [tuple(m._env[b[5]:b[5] + b[2]]) + (b[0], b[2]) for b in m._bas]
    s = {x for x, b in zip(e, m._bas) if b[1] == 0}
    p = [x for x, b in zip(e, m._bas) if b[1] == 1]
    merged = sum(x in s for x in p)
    return int((m._bas[:, 1] == 0).sum()) - merged, len(p)


def _big_batch():
    """a batch in which every resident warp of the integral and gradient kernels takes several tasks
    (148 x 8 CTAs of 4 warps) and one of the one-electron kernel eight pairs (148 x 4 x 8 warps), its
    neighbours of other sizes"""
    from test_hostcheck import odd_shells
    rng = np.random.default_rng(29)
    kinds = [Mole("H 0 0 0; H 0 0 0.74"), Mole(random_molecule(rng, 9)), odd_shells(Mole(random_molecule(rng, 4))),
             Mole(random_molecule(rng, 9)), Mole("O 0 0 0.1173; H 0 0.7572 -0.4692; H 0 -0.7572 -0.4692"),
             odd_shells(Mole(random_molecule(rng, 9)))]
    order = [k for _ in range(20) for k in range(len(kinds))]
    pairs, tasks = 0, np.zeros(6, int)
    for k in order:
        ns, np_ = _super_shells(kinds[k])
        n = [ns * (ns + 1) // 2, ns * np_, np_ * (np_ + 1) // 2]
        pairs += sum(n)
        for c, (bra, ket) in enumerate(((n[0], n[0]), (n[0], n[1]), (n[1], n[1]), (n[0], n[2]), (n[1] + n[2], n[2]),
                                        (3 * n[2], n[2]))):
            tasks[c] += bra * -(-ket // 32)
    assert pairs >= 8 * 148 * 4 * 8 and (tasks > 2 * 148 * 8 * 4).all()
    return kinds, order


@pytest.mark.parametrize("prec", [64, 32])
def test_eri_many_tasks(cuda, prec):
    """integrals of a batch in which every warp takes several tasks: the same bits as each molecule
    alone, where no warp takes a second one in the classes with p bras"""
    kinds, order = _big_batch()
    dt = torch.float64 if prec == 64 else torch.float32
    alone = [torch.from_numpy(_eri([m], prec, cuda)[1]).to(cuda) for m in kinds]
    P = Plan([kinds[k] for k in order])
    out = torch.full((P.n_eri,), float("nan"), dtype=dt, device=cuda)
    check(lib().b2_eri_s8(P.h, prec, ptr(out), stream_handle()), "b2_eri_s8")
    for i, k in enumerate(order):
        o = int(P.eri_off[i])
        assert torch.equal(out[o:o + len(alone[k])].double(), alone[k])
    P.close()


def test_int1e_many_pairs(cuda):
    """one-electron matrices of a batch with eight pairs per warp, chunks crossing molecules: the same
    bits as each molecule alone"""
    kinds, order = _big_batch()

    def matrices(mols):
        P = Plan(mols)
        a = [torch.full((P.n_mat,), float("nan"), dtype=torch.float64, device=cuda) for _ in range(3)]
        check(lib().b2_int1e(P.h, *[ptr(x) for x in a], stream_handle()), "b2_int1e")
        out = [[P.unpack(x.cpu().numpy(), k).copy() for x in a] for k in range(len(mols))]
        P.close()
        return out

    alone = [matrices([m])[0] for m in kinds]
    for got, k in zip(matrices([kinds[k] for k in order]), order):
        for a, b in zip(got, alone[k]):
            assert (a == b).all()
