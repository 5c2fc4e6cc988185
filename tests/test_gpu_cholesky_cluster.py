"""Gram matrices above 32 columns are factored by a cluster with a CTA for every 32 of them (csrc/bsq_cholesky_cluster.cuh): ranks at the edges
of its blocks of 32 and its steps of 8 columns, through the tests of the core kernels, which compare with FP64."""
import pytest

import test_gpu_core_kernels as core

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [33, 39, 41, 63, 96, 97, 128, 129, 161, 192, 193, 224, 225, 248, 255, 256])
def test_ranks_at_the_edges_of_blocks(lib, k):
    core.test_core_edges(core.CodedFactors(lib), k, "noise")
    core.test_core_of_deficient_and_zero_matrices(core.CodedFactors(lib), k)
