"""Density-fitting kernels at the sizes where their paths split."""
import numpy as np
import pytest

from hfgpu import CartesianBasis, Context
from hfgpu.clusters import water_cluster
from hfgpu.lib import HFG_DF_BF16, HFG_DF_FP32, HFG_DF_FP64, DFTensor

pytestmark = pytest.mark.gpu

AUX = "def2-universal-jkfit"


@pytest.fixture(scope="module")
def cluster():
    atoms = water_cluster(11)
    ctx = Context(CartesianBasis.build(atoms, "cc-pvdz"))
    df = DFTensor(ctx, CartesianBasis.build(atoms, AUX), storage=HFG_DF_FP32)
    yield ctx, df
    df.close()
    ctx.close()


# column tiles of 16, 32, 128, 144 and 256 rows (8 to 4 ring stages), and two
# tiles; n = 275 leaves ragged row blocks and column blocks
@pytest.mark.parametrize("nocc", [1, 16, 17, 128, 130, 256, 275])
@pytest.mark.parametrize("mma,tol", [(HFG_DF_BF16, 6e-3), (HFG_DF_FP32, 1e-3)])
def test_tensor_core_exchange_over_occupied_counts(cluster, nocc, mma, tol):
    ctx, df = cluster
    C = np.random.default_rng(nocc).standard_normal((ctx.n, nocc)) * 0.1
    J0, K0 = df.jk(C, mma=HFG_DF_FP64)
    J, K = df.jk(C, mma=mma)
    assert np.max(np.abs(J - J0)) <= 1e-12 * np.max(np.abs(J0))
    assert np.linalg.norm(K - K0) < tol * np.linalg.norm(K0)
    assert np.array_equal(K, K.T)


def test_three_centre_integrals_agree_between_launch_sizes():
    # a monomer's launches are small (lanes per combination, a block per
    # combination in the high classes); inside the cluster the same shells are
    # part of launches large enough for one lane each
    atoms = water_cluster(9)
    big, small = CartesianBasis.build(atoms, "cc-pvdz"), CartesianBasis.build(atoms[:3], "cc-pvdz")
    auxb, auxs = CartesianBasis.build(atoms, AUX), CartesianBasis.build(atoms[:3], AUX)
    cb, cs = Context(big), Context(small)
    want = cs.df_three_center(auxs)
    got = cb.df_three_center(auxb)[:auxs.n, :want.shape[1]]
    # 1e-14 relative per integral, cancellation within a contraction up to 1e2
    assert np.max(np.abs(got - want)) < 1e-12 * np.max(np.abs(want))
    cb.close()
    cs.close()


@pytest.mark.parametrize("n_occ,frozen", [(1, 0), (10, 0), (10, 3), (33, 1), (49, 0)])
@pytest.mark.parametrize("storage", [HFG_DF_FP64, HFG_DF_FP32])
def test_ri_mp2_matches_its_definition_on_the_transformed_factor(n_occ, frozen, storage):
    # blocks of 15 to 768 occupied orbitals, whole and ragged
    atoms = water_cluster(2)
    ctx = Context(CartesianBasis.build(atoms, "cc-pvdz"))
    df = DFTensor(ctx, CartesianBasis.build(atoms, AUX), storage=storage)
    n = ctx.n
    rng = np.random.default_rng(n_occ)
    C = np.linalg.qr(rng.standard_normal((n, n)))[0]
    eps = np.concatenate([np.sort(rng.uniform(-3, -0.5, n_occ)), np.sort(rng.uniform(0.3, 3, n - n_occ))])
    B = np.zeros((df.sizes()[1], n, n))
    i, j = np.tril_indices(n)
    B[:, i, j] = df.transform(C)
    B[:, j, i] = B[:, i, j]
    L = B[:, frozen:n_occ, n_occ:]
    v = np.einsum("qia,qjb->iajb", L, L, optimize=True)
    eo, ev = eps[frozen:n_occ], eps[n_occ:]
    gap = eo[:, None, None, None] - ev[None, :, None, None] + eo[None, None, :, None] - ev[None, None, None, :]
    want = np.sum(v * (2.0 * v - v.transpose(0, 3, 2, 1)) / gap)
    got = df.mp2_energy(C, eps, n_occ, frozen)
    # n_occ^2 n_virt^2 products of 64-bit sums over ~260 functions
    assert abs(got - want) < 1e-11 * abs(want)
    df.close()
    ctx.close()


def test_exchange_time_of_a_large_system_is_the_exchange_alone():
    # hfg_df_last_stats gives the device time of the exchange.  Above 1,100 AOs
    # J, which reads the factor twice (all but what the 126 MB L2 keeps) at no
    # more than 8 TB/s, runs outside it
    import torch
    nw = 48
    atoms = water_cluster(nw)
    stream = torch.cuda.Stream()
    ctx = Context(CartesianBasis.build(atoms, "cc-pvdz"), stream=stream.cuda_stream)
    df = DFTensor(ctx, CartesianBasis.build(atoms, AUX), pair_threshold=1e-10, storage=HFG_DF_BF16)
    nocc = 5 * nw
    C = torch.from_numpy(np.random.default_rng(3).standard_normal((nocc, ctx.n)) * 0.1).cuda()
    J, K = (torch.empty(ctx.n, ctx.n, dtype=torch.float64, device="cuda") for _ in range(2))
    torch.cuda.synchronize()
    rest = []
    for _ in range(6):
        t0, t1 = (torch.cuda.Event(enable_timing=True) for _ in range(2))
        t0.record(stream)
        df.jk_device_shard(C.data_ptr(), nocc, J.data_ptr(), K.data_ptr(), 0, 1, mma=HFG_DF_BF16)
        t1.record(stream)
        torch.cuda.synchronize()
        rest.append(t0.elapsed_time(t1) - df.last_stats()["k_ms"])
    _, rank, ncol = df.sizes()
    assert min(rest) > (2 * 2.0 * rank * ncol - 126e6) / 8e12 * 1e3
    df.close()
    ctx.close()
