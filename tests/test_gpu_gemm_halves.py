"""Products of 16 to 240 columns whose caller gives a bound on |A| (csrc/bsq_gemm.cu, bsq_gemm_tc.cu, bsq_gemm_tma.cu): their operands are split into
halves whose exponents reach as far as FP32's, so that the rows of a result are as good however far they lie below the largest element.  Compared with FP64."""
import ctypes as C

import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("km", [1, 0])
@pytest.mark.parametrize("m,n,k", [(512, 16, 1024), (515, 48, 1088), (1000, 64, 2060), (640, 128, 1028), (2048, 128, 4100), (1024, 144, 1100), (700, 240, 3000)])
def test_halves_of_every_width_against_fp64(lib, km, m, n, k):
    """K ends inside a slot of 64, inside an image of 32 and with the first slot of a part (one accumulator unused); rows end inside a tile.
    The tensor core truncates each time it accumulates 16 of K: at most 2^-23 of what has come together, twice as much room given here; the
    split itself leaves 2^-21."""
    if not km:
        m = m // 4 * 4                                        # (the stored rows are m long then)
    g = torch.Generator(device="cuda").manual_seed(m + n + k)
    a = torch.randn((m, k) if km else (k, m), device="cuda", generator=g)
    b = torch.randn(k, n, device="cuda", generator=g)
    bound = a.abs().max().view(torch.int32).clone()
    out, status = torch.full((m, n), 7.0, device="cuda"), torch.zeros(4, dtype=torch.int32, device="cuda")
    ws = torch.empty(64 << 20, dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    assert lib.bsq_gemm_bounded(km, 0, a.data_ptr(), a.shape[1], b.data_ptr(), n, out.data_ptr(), n, m, n, k, ws.data_ptr(), ws.numel(), bound.data_ptr(),
                                status.data_ptr(), None) == 0
    torch.cuda.synchronize()
    want = (a if km else a.T).double() @ b.double()
    scale = float(want.square().mean().sqrt())
    err = (out.double() - want).abs()
    assert int(status[0]) == 0
    assert float(err.square().mean().sqrt()) <= scale * (2 * k / 16 * 2.0 ** -23 + 2.0 ** -21)
    assert float(err.max()) <= 8 * scale * (2 * k / 16 * 2.0 ** -23 + 2.0 ** -21)


EXPONENTS = (20, 24, 28, 32, 36, 40, 60)


@pytest.mark.parametrize("km", [1, 0])
@pytest.mark.parametrize("m,n,k", [(1024, 16, 1024), (1000, 48, 1088), (2048, 128, 4100), (1024, 144, 1100), (700, 240, 3000)])
def test_rows_far_below_the_largest_element(lib, km, m, n, k):
    """The bound of the test above, over each row's own norm (that of 16 columns and more of N(0,1) operands: no cancellation over a row)."""
    if not km:
        m = m // 4 * 4
    g = torch.Generator(device="cuda").manual_seed(m + n + k)
    a = torch.randn(m, k, device="cuda", generator=g)
    for i, e in enumerate(EXPONENTS):
        a[130 + i] *= 2.0 ** -e
    b = torch.randn(k, n, device="cuda", generator=g)
    stored = a if km else a.T.contiguous()
    bound = a.abs().max().view(torch.int32).clone()
    out, status = torch.full((m, n), 7.0, device="cuda"), torch.zeros(4, dtype=torch.int32, device="cuda")
    ws = torch.empty(64 << 20, dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    assert lib.bsq_gemm_bounded(km, 0, stored.data_ptr(), stored.shape[1], b.data_ptr(), n, out.data_ptr(), n, m, n, k, ws.data_ptr(), ws.numel(),
                                bound.data_ptr(), status.data_ptr(), None) == 0
    torch.cuda.synchronize()
    want = a.double() @ b.double()
    err = (out.double() - want).norm(dim=1) / want.norm(dim=1)
    assert int(status[0]) == 0 and float(err.max()) <= 2 * k / 16 * 2.0 ** -23 + 2.0 ** -21


@pytest.mark.parametrize("k", [16, 48, 64, 128, 240])
def test_factors_of_rows_far_below_the_largest_element(lib, k):
    """A matrix of rank k: each row of U diag(S) V^T is the matrix's, to what the orthonormalisation's shift of 1e-5 and the products leave of the row
    itself (seen 1e-5 to 3e-5 for rows of every size)."""
    m, n = 2048, 1024
    g = torch.Generator(device="cuda").manual_seed(k)
    a = torch.randn(m, k, device="cuda", generator=g) @ torch.randn(k, n, device="cuda", generator=g)
    for i, e in enumerate(EXPONENTS[:-1]):
        a[i] *= 2.0 ** -e
    u, s, v = torch.empty(m, k, device="cuda"), torch.empty(k, device="cuda"), torch.empty(n, k, device="cuda")
    torch.cuda.synchronize()
    assert lib.bsq_svd_lowrank(a.data_ptr(), m, n, k, 2, 1234, u.data_ptr(), s.data_ptr(), v.data_ptr(), None) == 0
    torch.cuda.synchronize()
    y = (u.double() * s.double()) @ v.double().T
    err = (y - a.double()).norm(dim=1) / a.double().norm(dim=1)
    assert float(err.max()) <= 1.2e-4
