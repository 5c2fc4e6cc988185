"""Products whose tile width or reduction is chosen by size: 256-, 128- and 64-column tiles with ragged last tiles, K in one piece
and split, reductions of one and of four elements per thread, the scale pass over arrays with and without gaps between rows.

Bound: three tensor-core products of split operands leave at most a few 1e-7 of sum |a||b| (FP32 accumulation of up to 4096
terms in the tensor core's order); 4e-6 is allowed."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def check(lib, a_km, b_km, M, N, K, pad, workspace):
    g = torch.Generator(device="cuda").manual_seed(M + 3 * N + 7 * K)
    a_rows, a_cols = (M, K) if a_km else (K, M)
    b_rows, b_cols = (N, K) if b_km else (K, N)
    A = torch.randn(a_rows, a_cols + pad, device="cuda", generator=g)
    B = torch.randn(b_rows, b_cols + pad, device="cuda", generator=g)
    C = torch.full((M, N + pad), 3.0, device="cuda")
    ws = torch.empty(64 << 20, dtype=torch.uint8, device="cuda")
    status = torch.zeros(4, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    assert lib.bsq_gemm(int(a_km), int(b_km), A.data_ptr(), A.shape[1], B.data_ptr(), B.shape[1], C.data_ptr(), C.shape[1], M, N, K,
                        ws.data_ptr() if workspace else None, ws.numel() if workspace else 0, 1, status.data_ptr(), None) == 0
    torch.cuda.synchronize()
    a = A[:, :a_cols].double() if a_km else A[:, :a_cols].double().T
    b = B[:, :b_cols].double().T if b_km else B[:, :b_cols].double()
    want, scale = a @ b, a.abs() @ b.abs()
    assert int(status[0]) == 0
    assert bool(((C[:, :N].double() - want).abs() <= 4e-6 * scale).all())
    if pad:
        assert bool((C[:, N:] == 3.0).all())


@pytest.mark.parametrize("N", [16, 64, 112, 128, 144, 208, 240, 256])
@pytest.mark.parametrize("M", [128, 129, 777, 4096])
def test_panel_products(lib, M, N):
    check(lib, True, False, M, N, N if N >= 64 else 64, 0, True)
    check(lib, True, True, M, N, 256, 4, False)


@pytest.mark.parametrize("N", [128, 144, 208, 256])
@pytest.mark.parametrize("K", [512, 1031, 4096])
def test_gram_shaped_products(lib, N, K):
    check(lib, False, False, N, N, K, 0, True)
    check(lib, False, False, N, N, K, 4, True)


@pytest.mark.parametrize("shape", [(1024, 64, 2048), (4096, 48, 1536), (777, 33, 1031)])
def test_split_products(lib, shape):
    M, N, K = shape
    check(lib, True, False, M, N, K, 0, True)
    check(lib, True, False, M, N, K, 3, True)


@pytest.mark.parametrize("shape", [(4096, 4800, 256, 11), (4800, 8000, 144, 10), (8200, 4608, 128, -1)])
def test_objects_do_not_depend_on_the_matrices_in_flight(pkg, lib, shape):
    """A batch whose matrices fill the device keeps the panel products' tiles wide: same bytes as one matrix at a time."""
    rows, cols, rank, uv = shape
    mats = [torch.randn(rows, cols, device="cuda", generator=torch.Generator(device="cuda").manual_seed(i)) for i in range(8)]
    batch = lib.bsq_batch_create(rows, cols, 0.01, 0.0, rank, 1, uv, -1, -1, 8)
    assert batch
    try:
        cap = int(lib.bsq_lane_packed_capacity(lib.bsq_batch_lane(batch, 0)))
        want = []
        for m in mats:
            buf, size = torch.zeros(cap, dtype=torch.uint8, device="cuda"), C.c_uint64(0)
            torch.cuda.synchronize()
            assert lib.bsq_lane_compress_begin(lib.bsq_batch_lane(batch, 0), m.data_ptr(), 1, buf.data_ptr(), cap) == 0
            assert lib.bsq_lane_compress_end(lib.bsq_batch_lane(batch, 0), None, None, C.byref(size)) == 0
            want.append(buf[200: int(size.value)].clone())
        for count in (2, 4, 8):
            bufs = [torch.zeros(cap, dtype=torch.uint8, device="cuda") for _ in range(count)]
            vp = C.c_void_p * count
            torch.cuda.synchronize()
            assert lib.bsq_batch_compress(batch, vp(*[m.data_ptr() for m in mats[:count]]), count, 1, vp(*[b.data_ptr() for b in bufs]), cap,
                                          None, None, None) == 0
            for b, w in zip(bufs, want):
                assert torch.equal(b[200: 200 + w.numel()], w), count
    finally:
        lib.bsq_batch_destroy(batch)


@pytest.mark.parametrize("shape", [(1, 1, 1), (63, 64, 15), (64, 63, 16), (65, 64, 17), (64, 65, 63), (127, 48, 65), (128, 128, 64), (129, 129, 100), (300, 64, 48),
                                   (2000, 40, 4096), (777, 100, 1031), (40, 40, 2050)])
@pytest.mark.parametrize("a_km,b_km", [(1, 0), (1, 1), (0, 0), (0, 1)])
@pytest.mark.parametrize("off,pad", [(0, 0), (1, 0), (0, 1), (3, 4)])
def test_fp32_tiles(lib, shape, a_km, b_km, off, pad):
    """The FP32-pipe kernel at the edges of its tiles (64 and 128 rows and columns, 16 of K, K split and whole), operands on and off 16-byte
    boundaries.  A chain of up to 4096 multiply-adds per split and their sums: 4e-6 of sum |a||b| as above (about 64 2^-24 expected)."""
    M, N, K = shape
    g = torch.Generator(device="cuda").manual_seed(M + 3 * N + 7 * K)

    def operand(rows, cols):
        flat = torch.randn(off + rows * (cols + pad), device="cuda", generator=g)
        return flat[off:].view(rows, cols + pad)
    A = operand(*((M, K) if a_km else (K, M)))
    B = operand(*((N, K) if b_km else (K, N)))
    a = A[:, :K].double() if a_km else A[:, :M].double().T
    b = B[:, :K].double().T if b_km else B[:, :N].double()
    want, scale = a @ b, a.abs() @ b.abs()
    ws = torch.empty(64 << 20, dtype=torch.uint8, device="cuda")
    out = []
    for workspace in (True, False, True):
        C = torch.full((M, N + pad), 3.0, device="cuda")
        status = torch.zeros(4, dtype=torch.int32, device="cuda")
        torch.cuda.synchronize()
        assert lib.bsq_gemm(a_km, b_km, A.data_ptr(), A.shape[1], B.data_ptr(), B.shape[1], C.data_ptr(), C.shape[1], M, N, K,
                            ws.data_ptr() if workspace else None, ws.numel() if workspace else 0, 0, status.data_ptr(), None) == 0
        torch.cuda.synchronize()
        assert bool(((C[:, :N].double() - want).abs() <= 4e-6 * scale).all())
        assert bool((C[:, N:] == 3.0).all())
        out.append(C)
    assert torch.equal(out[0], out[2])
