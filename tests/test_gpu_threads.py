"""Contexts on several threads whose launches share a kernel at different sizes.

The block-per-quartet engine and the gradient kernels are one function for
many classes or atom counts, each launch with its own dynamic shared memory.
Different contexts may run concurrently, so no launch may disturb another's.
"""
import threading

import numpy as np
import pytest

from hfgpu import CartesianBasis, Context, HfgError
from hfgpu.clusters import water_cluster

pytestmark = pytest.mark.gpu


def rand_sym(n, seed):
    a = np.random.default_rng(seed).standard_normal((n, n)) * 0.3
    return a + a.T


def spdf():
    return CartesianBasis([("He", (0.0, 0.1, -0.2))], {"HE": [(l, np.array([2.1, 0.5]), np.array([0.4, 0.7]), None)
                                                             for l in range(4)]})


def test_concurrent_eager_calls_of_different_classes_succeed():
    import torch
    water, small = (CartesianBasis.build(water_cluster(1), b) for b in ("cc-pvdz", "6-31g*"))
    pair = CartesianBasis.build(water_cluster(2), "6-31g*")
    jobs = []

    def shards(basis):
        # sharded builds run eagerly, never from a graph
        ctx = Context(basis)
        P = torch.from_numpy(rand_sym(basis.n, 1)).cuda()
        J, K = torch.empty_like(P), torch.empty_like(P)
        jobs.append((ctx, 300, (P, J, K), lambda: ctx.jk_device_shard(P.data_ptr(), P.data_ptr(), J.data_ptr(),
                                                                      K.data_ptr(), 0, 2)))

    def gradients(basis):
        ctx = Context(basis)
        P = rand_sym(basis.n, 2)
        jobs.append((ctx, 60, P, lambda: ctx.gradient(P, P)))

    def packed(basis):
        ctx = Context(basis)
        jobs.append((ctx, 60, None, lambda: ctx.eri_packed(1e-12)))

    for basis in (water, spdf(), pair):
        shards(basis)
    for basis in (small, pair):
        gradients(basis)
    packed(water)
    torch.cuda.synchronize()
    errors = []

    def run(job):
        _, rounds, _, call = job
        for _ in range(rounds):
            try:
                call()
            except HfgError as e:
                errors.append(str(e))

    threads = [threading.Thread(target=run, args=(job,)) for job in jobs]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    for job in jobs:
        job[0].close()
    assert not errors, (len(errors), errors[:3])
