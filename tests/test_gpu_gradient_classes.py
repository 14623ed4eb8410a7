"""The two gradient kernels over the ranges that their launches split on.

Every class of s, p and d shells at primitive counts that fill a group of
lanes, leave it ragged and leave it nearly empty (the lane kernel gives a
shell quartet the largest power of two of lanes that its primitive quartets
fill), against fourth-order central differences of E2, and per-atom sums held
in shared memory (up to 512 atoms) against sums in device memory.
"""
import os

import numpy as np
import pytest

from hfgpu import CartesianBasis, Context
from hfgpu.lib import _dp

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "hf-rs_b200", "csrc")


def basis_of(atoms, counts):
    """s, p and d shells with the given primitive counts on every atom."""
    shells = []
    for l, k in enumerate(counts):
        shells.append((l, 0.35 * 2.3 ** np.arange(k)[::-1], np.linspace(0.3, 0.7, k), None))
    return CartesianBasis(atoms, {"HE": shells})


ATOMS = [("He", (0.0, 0.1, -0.2)), ("He", (1.3, -0.4, 0.5)), ("He", (-0.3, 1.1, 0.9))]


def e2(atoms, counts, P):
    ctx = Context(basis_of(atoms, counts))
    J, K = ctx.jk(P)
    ctx.close()
    return 0.5 * np.sum(P * J) - 0.25 * np.sum(P * K[0])


def density(n, seed):
    a = np.random.default_rng(seed).standard_normal((n, n)) * 0.3
    return a + a.T


@pytest.mark.gpu
@pytest.mark.parametrize("counts", [(1, 1, 1), (3, 2, 1), (5, 3, 2), (8, 1, 3)])
def test_every_class_and_primitive_count_matches_finite_differences(counts):
    ctx = Context(basis_of(ATOMS, counts))
    P = density(ctx.n, 7)
    g = ctx.eri_gradient(P)
    ctx.close()
    scale = np.max(np.abs(g))
    assert np.max(np.abs(g.sum(axis=0))) < 1e-11 * scale
    h = 1e-3
    for at, ax in ((0, 0), (1, 1), (2, 2)):
        f = {}
        for k in (-2, -1, 1, 2):
            moved = [list(p) for _, p in ATOMS]
            moved[at][ax] += k * h
            f[k] = e2([("He", tuple(p)) for p in moved], counts, P)
        fd = (8.0 * (f[1] - f[-1]) - (f[2] - f[-2])) / (12.0 * h)
        # truncation h^4 / 30 of the fifth derivative, rounding 1e-15 |E2| / h
        assert abs(fd - g[at, ax]) < 1e-8 * scale, (at, ax, fd, g[at, ax])


@pytest.mark.gpu
@pytest.mark.parametrize("natom", [3, 512, 513])
def test_atom_sums_in_shared_and_device_memory_agree(natom):
    ctx = Context(basis_of(ATOMS, (3, 2, 1)))
    P = density(ctx.n, 8)
    want = ctx.eri_gradient(P)
    g = np.ones((natom, 3))
    assert ctx.lib.hfg_eri_gradient(ctx.h, 1e-12, 1, _dp(P), _dp(P), natom, _dp(g)) == 0
    ctx.close()
    assert np.max(np.abs(g[:3] - want)) < 1e-12 * np.max(np.abs(want))
    assert np.all(g[3:] == 0.0)


def test_generated_gradient_code_matches_its_generator():
    import importlib.util
    import sys
    sys.path.insert(0, CSRC)
    spec = importlib.util.spec_from_file_location("gen_grad", os.path.join(CSRC, "gen_grad.py"))
    gen = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(gen)
    sys.path.remove(CSRC)
    assert gen.render() == open(os.path.join(CSRC, "grad_gen.cuh")).read()
