"""Top-k and error stage on rows that no bulk copy can move (columns not a multiple of four, a matrix that starts off a 16-byte
boundary), bit for bit against the CPU oracle: edges of the padding, of the unrolled loads and of each group width, ties, zeros,
Inf and NaN, separation in place."""
import numpy as np
import pytest

from conftest import bits

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def matrix(rows, cols, seed):
    rng = np.random.default_rng(seed)
    x = rng.standard_normal((rows, cols)).astype(np.float32)
    if rows > 4:
        x[1] = np.round(x[1])                                # heavy ties
        x[2] = 0.0
        x[2, :: max(1, cols // 3)] = -0.0
        x[3, cols // 2] = np.inf
        x[3, -1] = -np.inf
        x[4, ::2] = np.nan
    return x


@pytest.mark.parametrize("cols", [1, 2, 3, 5, 63, 65, 513, 1001, 2047, 4097, 4099, 8191, 8193, 12287, 24575])
@pytest.mark.parametrize("shift", [0, 1, 3])
def test_ragged_topk_matches_oracle(lib, oracle, cols, shift):
    rows = 9
    x = matrix(rows, cols, cols + shift)
    buf = torch.zeros(rows * cols + 8, dtype=torch.float32, device="cuda")
    d_x = buf[shift: shift + rows * cols]
    for k in sorted({1, min(cols, 2), max(1, cols // 100), min(cols, 256)}):
        want_i, want_v, want_res = oracle.topk_rows(x, k, zero_selected=True)
        for in_place in (False, True):
            d_x.copy_(torch.from_numpy(x.ravel()))
            d_i = torch.zeros(rows, k, dtype=torch.int16, device="cuda")
            d_v = torch.zeros(rows, k, dtype=torch.float32, device="cuda")
            res_buf = torch.full((rows * cols + 8,), 7.0, dtype=torch.float32, device="cuda")
            res = d_x if in_place else res_buf[1: 1 + rows * cols]
            status = torch.zeros(4, dtype=torch.int32, device="cuda")
            torch.cuda.synchronize()
            assert lib.bsq_topk_rows(d_x.data_ptr(), res.data_ptr(), rows, cols, k, d_i.data_ptr(), d_v.data_ptr(), status.data_ptr(), None) == 0
            torch.cuda.synchronize()
            assert int(status[0]) == 0
            assert np.array_equal(d_i.cpu().numpy().view(np.uint16), want_i), (cols, k)
            assert np.array_equal(bits(d_v.cpu().numpy()), bits(want_v)), (cols, k)
            assert np.array_equal(bits(res.cpu().numpy().reshape(rows, cols)), bits(want_res)), (cols, k, in_place)
            if not in_place:
                assert float(res_buf[0]) == 7.0 and bool((res_buf[1 + rows * cols:] == 7.0).all())
            else:
                assert bool((buf[shift + rows * cols:] == 0).all())


@pytest.mark.parametrize("rows,cols,k", [(1023, 63, 16), (1023, 63, 17), (1024, 65, 17), (1024, 65, 18), (7, 129, 32), (7, 129, 33), (7, 166, 33),
                                         (699, 1001, 80), (699, 1001, 81), (1023, 1001, 100), (1023, 1001, 101), (1024, 1001, 108),
                                         (1024, 1001, 109), (2000, 515, 112), (2000, 515, 113), (40, 4099, 160), (40, 4099, 161),
                                         (1024, 4099, 168), (1024, 4099, 169), (2000, 4099, 176), (2000, 4099, 177), (5, 8195, 216), (5, 8195, 217)])
def test_ragged_topk_either_side_of_the_lines(lib, oracle, rows, cols, k):
    """Where the kernel for short lists of ragged rows ends and the one for any shape begins (ragged_rows_fit)."""
    x = np.random.default_rng(rows + cols + k).standard_normal((rows, cols)).astype(np.float32)
    x[rows // 2, : cols // 2] = 0.0
    x[rows - 1] = np.round(x[rows - 1])                       # ties
    want_i, want_v, want_res = oracle.topk_rows(x, k, zero_selected=True)
    d_x = torch.from_numpy(x).cuda()
    d_i, d_v = torch.zeros(rows, k, dtype=torch.int16, device="cuda"), torch.zeros(rows, k, device="cuda")
    res, status = torch.empty_like(d_x), torch.zeros(4, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    assert lib.bsq_topk_rows(d_x.data_ptr(), res.data_ptr(), rows, cols, k, d_i.data_ptr(), d_v.data_ptr(), status.data_ptr(), None) == 0
    torch.cuda.synchronize()
    assert int(status[0]) == 0
    assert np.array_equal(d_i.cpu().numpy().view(np.uint16), want_i) and np.array_equal(bits(d_v.cpu().numpy()), bits(want_v))
    assert np.array_equal(bits(res.cpu().numpy()), bits(want_res))


@pytest.mark.parametrize("shape", [(1, 1), (1, 63), (3, 65), (17, 1003), (64, 1024), (129, 515)])
@pytest.mark.parametrize("q", [10, 11])
def test_error_list_of_a_quantised_matrix_matches_oracle(pkg, lib, oracle, shape, q):
    """The quantiser hands the error stage x - dequantised itself: same lists, and the same answer to "is anything left"."""
    rows, cols = shape
    for kind in ("gauss", "exact", "special"):
        x = matrix(rows, cols, 5 * rows + cols)
        if kind == "exact":
            x = np.where(x > 0, np.float32(1.0), np.float32(-1.0))       # quantises without error: no error section
        elif kind == "gauss":
            x = np.random.default_rng(rows + cols).standard_normal(shape).astype(np.float32)
        for outlier in (0.0, 0.02):
            assert lib.bsq_compress_initialize(rows, cols, outlier, 0.03, -1, 1, -1, -1, q, pkg.INPUT_DEVICE) == 0
            d_x = torch.from_numpy(x).cuda()
            torch.cuda.synchronize()
            res = pkg.compress_to_bytes(d_x.data_ptr())
            assert res is not None
            got = res[1].copy()
            got[192:200] = 0
            want = oracle.compress_nosvd(x, outlier, 0.03, q)
            assert np.array_equal(got, want), (shape, q, kind, outlier)
    lib.bsq_compress_release()
