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
