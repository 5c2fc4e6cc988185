"""Wide FP16 products leave through boxes of 32 x 32 values in shared memory, with and without a minuend (csrc/bsq_gemm_tma.cu): a reconstruction against
FP64, and a residual taken whole."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("rows,cols,rank", [(515, 3856, 64), (2049, 1328, 72), (1000, 2592, 80), (4097, 1200, 64), (2048, 5120, 128)])
def test_boxes_at_the_edges_of_tiles(pkg, lib, rows, cols, rank):
    """Rows end inside a tile, a quarter of one and with its first row; columns end with 16, 32, 48 or 176 of a tile's 256; the rank inside a slot of 64."""
    g = torch.Generator(device="cuda").manual_seed(rows)
    x = torch.randn(rows, cols, device="cuda", generator=g)
    y = torch.full((rows + 1, cols), 7.0, device="cuda")
    torch.cuda.synchronize()

    def round_trip(err):
        assert lib.bsq_compress_initialize(rows, cols, 0.0, err, rank, 2, -1, -1, -1, pkg.INPUT_DEVICE) == 0
        hdr, packed = pkg.compress_to_bytes(x.data_ptr())
        assert lib.bsq_decompress_initialize(rows, cols, 0.0, err, rank, -1, -1, -1) == 0
        assert pkg.decompress_packed(packed, y.data_ptr(), rows * cols) == 0
        torch.cuda.synchronize()
        assert bool((y[rows] == 7.0).all())                  # nothing behind the matrix
        return packed

    packed = round_trip(0.0)
    factors = packed[200:200 + (rows * rank + rank + cols * rank) * 4].copy().view(np.float32)     # U, S and V as they are, behind the header
    u, s, v = (torch.from_numpy(p.copy()).cuda().double() for p in np.split(factors, [rows * rank, rows * rank + rank]))
    u, v = u.view(rows, rank), v.view(cols, rank)
    want = (u * s) @ v.T
    # one product: the split leaves 2^-21 of its size, the tensor core's truncation 2^-23 for each 16 of K of three products, as much again for room
    bound = (u * s).norm(dim=1)[:, None] * v.norm(dim=1)[None, :] * (2.0 ** -21 + 2 * 3 * rank / 16 * 2.0 ** -23)
    assert bool(((y[:rows].double() - want).abs() <= bound).all())
    # every element of the residual kept: minuend - product + product, one rounding each, the product the same bits on both sides
    product = y[:rows].clone()
    round_trip(1.0)
    assert bool(((y[:rows] - x).abs() <= 2.0 ** -23 * (x.abs() + product.abs())).all())


@pytest.mark.parametrize("rows,cols,rank", [(515, 3856, 68), (1001, 2592, 100), (2050, 1328, 76)])
def test_wide_tiles_of_tf32_halves_at_the_edges(pkg, lib, rows, cols, rank):
    """Ranks that are not multiples of 8 keep TF32 halves and leave a row per lane; the last rows fill part of a warp."""
    test_boxes_at_the_edges_of_tiles(pkg, lib, rows, cols, rank)
