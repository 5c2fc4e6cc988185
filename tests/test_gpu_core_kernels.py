"""The k x k kernels of the randomized SVD (Cholesky factor and inverse by 32 x 32 blocks, block Jacobi on 1 to 8 CTAs) at the edges
of their blocks, clusters and paddings, through bsq_svd_lowrank, against FP64 numpy; and the kernels that take the core's SVD where factors are
coded (one CTA up to 48 columns, columns on a ring of warps above, over a cluster above 64) by the same checks and those of test_gpu_svd.py, through bsq_svd_lowrank_coded.

Bounds.  Each QR pass factors G + 1e-5 max(diag G) I, so columns are orthonormal to a few 1e-5, up to 2e-4 for the weakest
direction of a wide sketch (the bounds of test_gpu_svd.py).  With orthonormal Q the residual of Q Q^T A has the squared norm
|A|^2 - sum S^2: both sides are compared to 1e-3 of |A|^2 (twice the orthonormality bound for the two factors, and FP32 sums)."""
import ctypes as C
import ctypes.util
import glob
import os

import numpy as np
import pytest

import test_gpu_svd

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def svd_gpu(lib, a, k, niter=2):
    m, n = a.shape
    d_a = torch.from_numpy(a).cuda()
    u, s, v = torch.zeros(m, k, device="cuda"), torch.zeros(k, device="cuda"), torch.zeros(n, k, device="cuda")
    torch.cuda.synchronize()
    assert lib.bsq_svd_lowrank(d_a.data_ptr(), m, n, k, niter, 1241, u.data_ptr(), s.data_ptr(), v.data_ptr(), None) == 0
    torch.cuda.synchronize()
    return u.cpu().numpy().astype(np.float64), s.cpu().numpy().astype(np.float64), v.cpu().numpy().astype(np.float64)


@pytest.mark.parametrize("k", [1, 2, 3, 15, 16, 17, 31, 32, 33, 48, 63, 64, 65, 96, 97, 127, 128, 129, 160, 192, 224, 255, 256])
@pytest.mark.parametrize("kind", ["noise", "small", "large"])
def test_core_edges(lib, k, kind):
    m, n = 640, 528
    rng = np.random.default_rng(k)
    a = rng.standard_normal((m, n)) @ np.diag(1.0 / np.arange(1, n + 1)) + 0.02 * rng.standard_normal((m, n))
    a = (a * {"noise": 1.0, "small": 1e-9, "large": 1e9}[kind]).astype(np.float32)
    u, s, v = svd_gpu(lib, a, k)
    exact = np.linalg.svd(a.astype(np.float64), compute_uv=False)
    norm2 = float((a.astype(np.float64) ** 2).sum())
    assert np.all(np.diff(s) <= 1e-6 * s[0]) and np.all(s >= 0)
    assert np.all(s <= exact[:k] * (1 + 2e-4))
    tol = 1e-4 if k <= 128 else 2e-4
    assert np.abs(u.T @ u - np.eye(k)).max() <= tol and np.abs(v.T @ v - np.eye(k)).max() <= tol
    res2 = float(((a - (u * s) @ v.T) ** 2).sum())
    assert abs(res2 - (norm2 - float((s ** 2).sum()))) <= 1e-3 * norm2
    u2, s2, v2 = svd_gpu(lib, a, k)                          # the same input gives the same bits
    assert np.array_equal(u, u2) and np.array_equal(s, s2) and np.array_equal(v, v2)


@pytest.mark.parametrize("k", [5, 32, 40, 64, 100, 200, 256])
def test_core_of_deficient_and_zero_matrices(lib, k):
    m, n, r = 512, 448, 3
    rng = np.random.default_rng(k)
    a = (rng.standard_normal((m, r)) @ rng.standard_normal((r, n))).astype(np.float32)
    u, s, v = svd_gpu(lib, a, k)
    exact = np.linalg.svd(a.astype(np.float64), compute_uv=False)[:r]
    assert np.isfinite(u).all() and np.isfinite(s).all() and np.isfinite(v).all()
    assert np.max(np.abs(s[:r] - exact) / exact) <= 1e-4     # well-separated values: the contract's bound
    assert np.all(s[r:] <= 1e-3 * s[0])
    assert np.linalg.norm(a - (u * s) @ v.T) <= 1e-4 * np.linalg.norm(a)
    u, s, v = svd_gpu(lib, np.zeros((m, n), np.float32), k)
    assert np.isfinite(u).all() and np.isfinite(v).all() and not s.any()


@pytest.mark.parametrize("k", [8, 16, 17, 33, 48, 64, 65, 100, 128, 200, 256])
@pytest.mark.parametrize("kind", ["1/i", "flat"])
def test_rotations_of_fp32_factors_keep_lengths(lib, k, kind):
    """A matrix of k columns at rank k: its row space is captured whole, so S are its singular values but for rounding.  2e-6 of
    |S|: a sweep rotates a column k times and there are 8 or 9, and where each rotation rounds an element once, without a bias,
    that is sqrt(9 * 256) * 2^-25 = 1.4e-6 at 256 columns, with half as much again for the sums of the panel products.  (A rounded
    cosine in every rotation is a bias: 3e-5 to 6e-5 at 256 columns.)"""
    rng = np.random.default_rng(k)
    m = 2 * k + 64
    q1, q2 = np.linalg.qr(rng.standard_normal((m, k)))[0], np.linalg.qr(rng.standard_normal((k, k)))[0]
    sv = 1.0 / np.arange(1, k + 1) + 0.05 if kind == "1/i" else 1.0 + 0.1 * rng.random(k)
    a = ((q1 * sv) @ q2.T).astype(np.float32)
    exact = np.linalg.svd(a.astype(np.float64), compute_uv=False)
    s = svd_gpu(lib, a, k)[1]
    assert np.linalg.norm(s - exact) <= 2e-6 * np.linalg.norm(exact)


@pytest.mark.parametrize("k", [7, 9, 23, 24, 25, 34, 47, 49, 71, 72, 73])
def test_shapes_of_blocks_follow_the_rank(lib, k):
    """Full blocks of 8 and 12 columns, and the ranks on either side of each line of block_jacobi_shape."""
    for kind in ("noise", "small"):
        test_core_edges(lib, k, kind)
    test_core_of_deficient_and_zero_matrices(lib, k)
    for kind in ("1/i", "flat"):
        test_rotations_of_fp32_factors_keep_lengths(lib, k, kind)


class CodedFactors:
    """The library with bsq_svd_lowrank standing for the kernels of coded factors."""

    def __init__(self, lib):
        self.bsq_svd_lowrank = lib.bsq_svd_lowrank_coded


@pytest.mark.parametrize("k", [1, 2, 3, 8, 15, 16, 17, 31, 32, 33, 48, 63, 64, 65, 96, 127, 128, 129, 131, 160, 200, 255, 256])
@pytest.mark.parametrize("kind", ["noise", "large"])
def test_core_edges_of_coded_factors(lib, k, kind):
    test_core_edges(CodedFactors(lib), k, kind)


@pytest.mark.parametrize("k", [5, 32, 40, 64, 65, 100, 200, 256])
def test_coded_core_of_deficient_and_zero_matrices(lib, k):
    test_core_of_deficient_and_zero_matrices(CodedFactors(lib), k)


@pytest.mark.parametrize("case", [(1024, 512, 64, 2), (512, 2048, 32, 2), (2048, 1024, 128, 1), (300, 180, 20, 3), (1024, 768, 96, 2),
                                  (700, 900, 131, 2), (1024, 1024, 160, 2), (1536, 1024, 256, 2)])
def test_coded_factors_accuracy_against_exact(lib, case):
    test_gpu_svd.test_svd_accuracy_against_exact(CodedFactors(lib), case)


def test_coded_factors_of_rank_deficient_and_zero_inputs(lib):
    test_gpu_svd.test_svd_rank_deficient_and_zero_inputs(CodedFactors(lib))


@pytest.mark.parametrize("k", [49, 53, 54, 57, 62, 70, 101, 150, 197])
def test_core_of_coded_factors_with_partly_filled_warps(lib, k):
    """Ranks that leave one, two or three of the last warp's four column pairs empty, on one CTA (49 to 64 columns) and on clusters."""
    test_core_edges(CodedFactors(lib), k, "noise")
    test_core_of_deficient_and_zero_matrices(CodedFactors(lib), k)


def omega_of(n, k, seed):
    """The range finder's random matrix, n x k: cuRAND's default sequence, column-major."""
    found = glob.glob(os.path.join(os.path.dirname(torch.__file__), "..", "nvidia", "curand", "lib", "libcurand.so.10"))
    rand = C.CDLL(found[0] if found else ctypes.util.find_library("curand") or "libcurand.so.10")
    gen, count = C.c_void_p(), n * k + (n * k & 1)
    out = np.empty(count, np.float32)
    assert rand.curandCreateGeneratorHost(C.byref(gen), 100) == 0
    assert rand.curandSetPseudoRandomGeneratorSeed(gen, C.c_ulonglong(seed)) == 0
    assert rand.curandGenerateNormal(gen, C.c_void_p(out.ctypes.data), C.c_size_t(count), C.c_float(0.0), C.c_float(1.0)) == 0
    rand.curandDestroyGenerator(gen)
    return out[: n * k].reshape(k, n).T.astype(np.float64)


def orthonormalised(y, passes):
    factors = []
    for _ in range(passes):
        g = y.T @ y
        r = np.linalg.cholesky(g + 1e-5 * g.diagonal().max() * np.eye(len(g))).T
        y = y @ np.linalg.inv(r)
        factors.append(r)
    return y, factors


def rotated(m, first_round=0):
    """One-sided Jacobi of the columns of m in FP64, pairs in the order of the round-robin tournament that the kernels keep: columns, lengths
    (descending) and how far from a tie the closest decision on a rotation's sense was."""
    k = m.shape[1]
    kp, length = (k + 1) & ~1, 64 if k <= 64 else 128 if k <= 128 else 256
    m, margin = np.hstack([m, np.zeros((len(m), kp - k))]), np.inf
    for _ in range(30):
        norm, big = (m * m).sum(0), False
        for i in range(kp - 1):
            r, slot = (i + first_round) % (kp - 1), np.arange(1, kp // 2)
            p, q = np.append(kp - 1, (r + slot) % (kp - 1)), np.append(r, (r + kp - 1 - slot) % (kp - 1))
            a, b, g = norm[p], norm[q], (m[:, p] * m[:, q]).sum(0)
            on = (a > 0) & (b > 0) & (g * g > length * 2.0 ** -48 * a * b)
            p, q, a, b, g = p[on], q[on], a[on], b[on], g[on]
            if len(p) == 0:
                continue
            zeta = (b - a) / (2 * g)
            margin = min(margin, float((np.abs(b - a) / np.maximum(a, b)).min()))
            t = np.copysign(1.0, zeta) / (np.abs(zeta) + np.sqrt(1 + zeta * zeta))
            c = 1 / np.sqrt(1 + t * t)
            m[:, p], m[:, q] = c * m[:, p] - c * t * m[:, q], c * t * m[:, p] + c * m[:, q]
            norm[p], norm[q] = np.maximum(a - t * g, 0), b + t * g
            big |= bool((g * g > 1e-8 * a * b).any())
        if not big:
            break
    norm = np.sqrt((m * m).sum(0))
    order = np.argsort(-norm, kind="stable")[:k]
    return m[:, order] / norm[order], norm[order], margin


def coded_case(k, seed):
    """A matrix of rank k whose singular values are k distinct ones between 1 and 2, its SVD as the stage works it out, in FP64, and the matrix
    whose columns the core kernel rotates."""
    rng = np.random.default_rng(seed)
    m, n = 2 * k + 64, k + 37
    left, right = np.linalg.qr(rng.standard_normal((m, k)))[0], np.linalg.qr(rng.standard_normal((n, k)))[0]
    a = ((left * (2 - np.arange(k) / k)) @ right.T).astype(np.float32)
    w = a.astype(np.float64)
    q, _ = orthonormalised(w @ omega_of(n, k, 1241), 1)
    for it in range(2):
        z, _ = orthonormalised(w.T @ q, 1)
        q, _ = orthonormalised(w @ z, 1 + it)
    _, (r1, r2) = orthonormalised(w.T @ q, 2)
    return a, q, (r2 @ r1).T



@pytest.mark.parametrize("k,seed", [(33, 1000), (48, 1002), (49, 1002), (53, 1003), (64, 1003), (65, 1004), (70, 70), (101, 1003)])
def test_order_of_rotations_of_coded_factors(lib, k, seed):
    """Codes depend on the sign that each singular pair comes out with, and that on the order of the rotations.  Every pair has the sign that
    the restated order gives: left vectors within 0.05 of the FP64 ones (a core off by 3e-6 in every element, as FP32 products leave it, moves
    them by 1e-4, and the seeds are such that no rotation's sense is closer to a tie than 1e-4).  Begun one round later the order gives 9 to 42
    other signs.  Up to 101 columns: beyond, a core that far off takes other senses."""
    a, q, core = coded_case(k, seed)
    vec, s, margin = rotated(core.copy())
    assert margin > 1e-4
    assert ((vec * rotated(core.copy(), 1)[0]).sum(0) < 0).any()
    u, s_gpu, _ = svd_gpu(CodedFactors(lib), a, k)
    assert np.abs(s_gpu - s).max() <= 1e-4 * s[0]
    assert (np.abs(u - q @ vec).max(axis=0) <= 0.05).all()
