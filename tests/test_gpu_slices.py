"""Sliced J/K work queues and the block-per-quartet engine on s, p, d shells.

A small molecule's J/K build splits the primitive quartets of its contracted
shell quartets over several work entries, and runs the d-rich launches of few
quartets on the engine of the f shells.  Both are checked at primitive counts
that divide unevenly, against the oracle and against a batch (whose plans
slice more coarsely), and the exact work counts must not see the slices.
"""
import numpy as np
import pytest

import oracle as O
from hfgpu import CartesianBasis, Context, JKOptions
from hfgpu.clusters import water_cluster

pytestmark = pytest.mark.gpu

ATOMS = [("He", (0.0, 0.1, -0.2)), ("He", (1.3, -0.4, 0.5)), ("He", (-0.3, 1.1, 0.9))]


def shells(counts):
    return [(l, 0.35 * 2.1 ** np.arange(k)[::-1], np.linspace(0.3, 0.7, k), None) for l, k in enumerate(counts)]


def rand_sym(n, seed):
    a = np.random.default_rng(seed).standard_normal((n, n)) * 0.3
    return a + a.T


def oracle_basis(atoms, sh):
    text = "HE     0\n"
    for l, e, c, _ in sh:
        text += "%s   %d   1.00\n" % ("SPD"[l], len(e))
        text += "".join("%.17g %.17g\n" % x for x in zip(e, c))
    return O.build_basis(atoms, O.parse_gaussian94(text + "****\n"))


@pytest.mark.parametrize("counts", [(1, 1, 1), (7, 1, 1), (5, 3, 2), (11, 2, 3)])
def test_sliced_builds_match_the_oracle(counts):
    sh = shells(counts)
    ctx = Context(CartesianBasis(ATOMS, {"HE": sh}))
    ref = oracle_basis(ATOMS, sh)
    Pa, Pb = rand_sym(ctx.n, 1), rand_sym(ctx.n, 2)
    for prim in (0.0, 1e-14):
        J, K = ctx.jk(Pa + Pb, [Pa, Pb], opts=JKOptions.make(prim=prim))
        Jr, Kr = O.direct_jk(ref, Pa + Pb, [Pa, Pb])
        scale = np.max(np.abs(Jr))
        # primitive screening drops products below prim, at most 1e6 of them
        tol = 1e-12 * scale + 1e6 * prim
        assert np.max(np.abs(J - Jr)) < tol and np.max(np.abs(np.stack(K) - np.stack(Kr))) < tol, (counts, prim)
    ctx.close()


@pytest.mark.parametrize("nw", [1, 3])
def test_work_counts_do_not_see_the_slices(nw):
    # every unique significant quartet once, with all its primitive quartets
    basis = CartesianBasis.build(water_cluster(nw), "cc-pvdz")
    ctx = Context(basis)
    ctx.jk(rand_sym(ctx.n, 3))
    s = ctx.last_stats()
    Q = ctx.schwarz()
    k = np.array([basis.prim_off[f + 1] - basis.prim_off[f] for f, _, _ in basis.shells])
    a, b = np.tril_indices(len(k))
    npp = (k[a] * k[b]).astype(float)
    i, j = np.tril_indices(len(Q))
    on = Q[i] * Q[j] > 1e-12
    assert s["quartets_fp64"] == np.count_nonzero(on)
    assert s["prim_quartets_fp64"] == np.sum((npp[i] * npp[j])[on])
    ctx.close()


def test_batch_and_single_builds_of_sliced_molecules_agree():
    import torch
    dev = torch.device("cuda", 0)
    ctxs = [Context(CartesianBasis.build(water_cluster(1 + k % 3, seed=k), "cc-pvdz")) for k in range(5)]
    P = [torch.from_numpy(rand_sym(c.n, k)).to(dev) for k, c in enumerate(ctxs)]
    J, K = [torch.empty_like(p) for p in P], [torch.empty_like(p) for p in P]
    torch.cuda.synchronize()
    Context.jk_device_batch(ctxs, *[[t.data_ptr() for t in x] for x in (P, J, K)])
    torch.cuda.synchronize()
    for c, p, j, k in zip(ctxs, P, J, K):
        Jr, Kr = c.jk(p.cpu().numpy())
        assert np.max(np.abs(j.cpu().numpy() - Jr)) < 1e-12 * np.max(np.abs(Jr))
        assert np.max(np.abs(k.cpu().numpy() - Kr[0])) < 1e-12 * np.max(np.abs(Jr))
        c.close()


def test_packed_tensor_and_gradient_after_a_sliced_build():
    # consumers of whole quartets on a context whose J/K plan slices them
    atoms = water_cluster(1)
    ctx = Context(CartesianBasis.build(atoms, "cc-pvdz"))
    P = rand_sym(ctx.n, 5)
    g0 = ctx.eri_gradient(P)
    J, K = ctx.jk(P)
    ref = O.eri_packed(O.build_basis(atoms, O.load_basis("cc-pvdz")))
    assert np.max(np.abs(ctx.eri_packed(1e-12) - ref)) < 1e-12
    assert np.max(np.abs(ctx.eri_gradient(P) - g0)) < 1e-12 * np.max(np.abs(g0))
    ctx.close()


def test_packed_tensor_does_not_depend_on_an_earlier_build():
    # 666 (dd|dd) quartets of one primitive each: the J/K plan slices nothing
    # and takes its generated kernel there, the packed tensor's the block engine
    atoms = [("He", (1.6 * (i % 2), 1.7 * (i // 2 % 2), 1.5 * (i // 4) + 0.1 * i)) for i in range(8)]
    basis = CartesianBasis(atoms, {"HE": [(2, np.array([0.8]), np.array([1.0]), None),
                                          (0, np.array([1.1]), np.array([1.0]), None)]})
    fresh, used = Context(basis), Context(basis)
    used.jk(rand_sym(basis.n, 6))
    assert np.array_equal(fresh.eri_packed(1e-12), used.eri_packed(1e-12))
    fresh.close()
    used.close()


def test_deterministic_builds_take_whole_quartets():
    # one warp (or block) runs a deterministic build's queue: its plan has no
    # slices, so it agrees to the bit with a build on the packed tensor's plan
    # (s, p and f shells: no class that only one of the two gives the block engine)
    import ctypes

    import torch
    sh = [(l, np.array([2.4, 1.1, 0.5]), np.array([0.4, 0.5, 0.3]), None) for l in (0, 1, 3)]
    basis = CartesianBasis(ATOMS[:2], {"HE": sh})
    n, det = basis.n, JKOptions.make(deterministic=True)
    ctx, other = Context(basis), Context(basis)
    P = rand_sym(n, 7)
    J, K = ctx.jk(P, opts=det)
    other.eri_packed(1e-12)
    dP = torch.from_numpy(P).cuda()
    dJ, dK = torch.empty_like(dP), torch.empty_like(dP)
    torch.cuda.synchronize()
    assert other.lib.hfg_jk_device_noalloc(other.h, ctypes.byref(det), 1, dP.data_ptr(), dP.data_ptr(), dJ.data_ptr(),
                                           dK.data_ptr()) == 0
    torch.cuda.synchronize()
    assert np.array_equal(dJ.cpu().numpy(), J) and np.array_equal(dK.cpu().numpy(), K[0])
    ctx.close()
    other.close()
