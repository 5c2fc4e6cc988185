"""Gram matrices above 32 columns are factored by a cluster with a CTA for every 32 of them (csrc/bsq_cholesky_cluster.cuh): ranks at the edges
of its blocks of 32 and its steps of 8 columns, through the tests of the core kernels, which compare with FP64."""
import numpy as np
import pytest

import test_gpu_core_kernels as core

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [33, 39, 41, 63, 96, 97, 128, 129, 161, 192, 193, 224, 225, 248, 255, 256])
def test_ranks_at_the_edges_of_blocks(lib, k):
    core.test_core_edges(core.CodedFactors(lib), k, "noise")
    core.test_core_of_deficient_and_zero_matrices(core.CodedFactors(lib), k)


@pytest.mark.parametrize("k", [33, 40, 63, 64, 97, 128, 131, 192, 200, 225, 256])
@pytest.mark.parametrize("coded", [False, True])
def test_devices_that_cannot_place_the_cluster_get_the_same_bits(lib, monkeypatch, k, coded):
    """cholesky_kernel, one CTA that factors and those of the inverse beside it, makes the same sums in the same order."""
    rng = np.random.default_rng(k)
    a = (rng.standard_normal((640, 528)) @ np.diag(1.0 / np.arange(1, 529)) + 0.02 * rng.standard_normal((640, 528))).astype(np.float32)
    side = core.CodedFactors(lib) if coded else lib
    cluster = core.svd_gpu(side, a, k)
    monkeypatch.setenv("BSQ_CHOL_CLUSTER", "0")
    assert all(np.array_equal(x, y) for x, y in zip(cluster, core.svd_gpu(side, a, k)))
