"""Pivoted Cholesky over column counts below, at and beyond one tile per block."""
import numpy as np
import pytest

from hfgpu import CartesianBasis, Context, HfgError
from hfgpu.clusters import water_cluster
from hfgpu.lib import DFTensor

pytestmark = pytest.mark.gpu


# 28 pairs (less than one tile of 32 columns), 325 (a tile per block, the last
# short), and 5,050 (two tiles per block, more than one on each of 148 SMs)
@pytest.mark.parametrize("nw,basis,threshold", [(1, "sto-3g", 1e-8), (1, "cc-pvdz", 1e-7), (4, "cc-pvdz", 1e-4)])
def test_factor_reproduces_the_supermatrix_within_its_residual(nw, basis, threshold):
    ctx = Context(CartesianBasis.build(water_cluster(nw), basis))
    n = ctx.n
    f, piv, res = DFTensor.cholesky(ctx, threshold)
    assert len(piv) == f.sizes()[1] == len(set(piv)) and res <= threshold
    L = f.transform(np.eye(n))
    npair = n * (n + 1) // 2
    eri = ctx.eri_packed(1e-15)
    idx = np.arange(npair, dtype=np.int64)
    diag = eri[idx * (idx + 1) // 2 + idx]
    resid = diag - np.einsum("kp,kp->p", L, L)
    assert np.min(resid) > -1e-12 and abs(np.max(resid) - res) < 1e-12
    # the pivots' own columns are exact
    cols = np.array(piv[:8])
    hi, lo = np.maximum(idx[:, None], cols), np.minimum(idx[:, None], cols)
    assert np.max(np.abs(L.T @ L[:, cols] - eri[hi * (hi + 1) // 2 + lo])) < 1e-11
    f.close()
    # a budget short of the last vector is refused, as before
    with pytest.raises(HfgError, match="budget"):
        DFTensor.cholesky(ctx, threshold, budget=8 * npair * (len(piv) - 1))
    ctx.close()


def test_an_infinite_diagonal_is_refused():
    # a contraction coefficient so large that (ss|ss) overflows: no bound holds
    # for an infinite residual, so no block owns the pivot
    basis = CartesianBasis([("He", (0.0, 0.0, 0.0)), ("He", (0.0, 0.0, 1.2))], {"HE": [(0, np.array([0.9]), np.array([1.0]),
                                                                                      None)]})
    basis.coefs[0] = 1e80
    ctx = Context(basis)
    assert np.isinf(ctx.eri_packed(1e-15)[0])
    with pytest.raises(HfgError, match="residual Coulomb diagonal"):
        DFTensor.cholesky(ctx, 1e-6)
    ctx.close()
