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


def test_products_side_by_side_give_the_bits_of_products_alone(lib):
    """The products of a rank-256 range finder for two matrices on two streams, kernels of both on the same SMs: every product as when it
    ran alone, bit for bit.  Both orientations of A through the FP16 raw slots, Gram and panel products between them."""
    m, n, k = 4096, 4800, 256

    class Chain:
        def __init__(self, seed):
            g = torch.Generator(device="cuda").manual_seed(seed)
            self.stream = torch.cuda.Stream()
            self.a, self.omega = torch.randn(m, n, device="cuda", generator=g), torch.randn(k, m, device="cuda", generator=g)
            self.qn, self.qm = torch.randn(n, k, device="cuda", generator=g) / n ** 0.5, torch.randn(m, k, device="cuda", generator=g) / m ** 0.5
            self.t = torch.randn(k, k, device="cuda", generator=g).triu() / 16
            self.bound = self.a.abs().max().view(torch.int32).reshape(1).clone()
            self.ws, self.status = torch.empty(160 << 20, dtype=torch.uint8, device="cuda"), torch.zeros(4, dtype=torch.int32, device="cuda")
            self.out = [torch.empty(*shape, device="cuda") for shape in ((n, k), (k, k), (n, k), (m, k), (k, k), (m, k), (n, k))]
            self.wrong = torch.zeros(len(self.out), dtype=torch.int64, device="cuda")

        def product(self, a_km, b_km, A, B, C, M, N, K, bounded):
            tail = (self.bound.data_ptr() if bounded else 1, self.status.data_ptr(), self.stream.cuda_stream)
            call = lib.bsq_gemm_bounded if bounded else lib.bsq_gemm
            assert call(a_km, b_km, A.data_ptr(), A.shape[1], B.data_ptr(), B.shape[1], C.data_ptr(), N, M, N, K, self.ws.data_ptr(), self.ws.numel(), *tail) == 0

        def run(self):
            y, gy, qy, z, gz, qz, w = self.out
            self.product(0, 1, self.a, self.omega, y, n, k, m, True)
            self.product(0, 0, y, y, gy, k, k, n, False)
            self.product(1, 0, y, self.t, qy, n, k, k, False)
            self.product(1, 0, self.a, self.qn, z, m, k, n, True)
            self.product(0, 0, z, z, gz, k, k, m, False)
            self.product(1, 0, z, self.t, qz, m, k, k, False)
            self.product(0, 0, self.a, self.qm, w, n, k, m, True)

        def check(self):
            with torch.cuda.stream(self.stream):
                self.wrong += torch.stack([(o != r).any() for o, r in zip(self.out, self.want)])
                for o in self.out:
                    o.fill_(float("nan"))
    chains = [Chain(1), Chain(2)]
    torch.cuda.synchronize()
    for c in chains:
        c.run()
        torch.cuda.synchronize()
        c.want = [o.clone() for o in c.out]
        assert bool(((c.out[3].double() - c.a.double() @ c.qn.double()).abs() <= 4e-6 * (c.a.double().abs() @ c.qn.double().abs())).all())
    for i in range(150):
        for c in chains:
            c.run()
        for c in chains:
            c.check()
        if i % 8 == 7:
            torch.cuda.synchronize()
    torch.cuda.synchronize()
    for c in chains:
        assert c.wrong.tolist() == [0] * len(c.out) and int(c.status[0]) == 0
