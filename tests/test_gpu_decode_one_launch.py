"""A device-resident quantised matrix is checked, decoded and completed with its lists by one kernel (csrc/bsq_quant.cu): the bits of the
host object's route, at sizes around the kernel's batches of 1024 elements, with lists shorter and longer than what a batch brings with it."""
import ctypes as C
import importlib

import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

# rows, cols, outlier, error: one batch and a little less or more, several rows in a batch, several batches in a row, ragged rows (lists and
# codes off their alignment), lists of 1, 64, 65 and more than 128 entries, lists that name the same elements, more batches than warps
CASES = [
    (1, 1023, 0.01, 0.0), (1, 1025, 0.01, 0.02), (3, 341, 0.3, 0.3), (33, 31, 0.0, 0.1), (64, 64, 1.0, 1.0), (5, 2049, 0.04, 0.001),
    (16, 6400, 0.01, 0.0102), (7, 14335, 0.005, 0.01), (300, 14336, 0.0, 0.02), (1501, 3001, 0.005, 0.01),
]
# lists that a kernel of their own adds: one and two of them, in one launch and in two, ragged, all of a row
LONG_CASES = [(8, 11200, 0.036, 0.253), (64, 3136, 0.11, 0.33), (11, 5879, 0.0, 0.2), (33, 2047, 1.0, 0.0), (512, 1601, 0.4, 0.6), (5, 14335, 0.5, 1.0)]


@pytest.mark.parametrize("q", [10, 11])
@pytest.mark.parametrize("case", CASES)
def test_one_launch_gives_the_host_objects_bits(pkg, lib, case, q):
    rows, cols, outlier, error = case
    x = torch.randn(rows, cols, device="cuda", generator=torch.Generator(device="cuda").manual_seed(rows + cols))
    lane = lib.bsq_lane_create(rows, cols, outlier, error, -1, 1, -1, -1, q)
    assert lane
    try:
        cap = int(lib.bsq_lane_packed_capacity(lane))
        buf = torch.empty(cap, dtype=torch.uint8, device="cuda")
        room = torch.full((rows * cols + 8,), 7.0, device="cuda")
        torch.cuda.synchronize()
        hdr, out = pkg.Array(), C.c_void_p(None)
        assert lib.bsq_lane_compress_begin(lane, x.data_ptr(), 1, buf.data_ptr(), cap) == 0
        assert lib.bsq_lane_compress_end(lane, None, C.byref(hdr), None) == 0
        assert lib.bsq_lane_compress_begin(lane, x.data_ptr(), 1, None, 0) == 0
        assert lib.bsq_lane_compress_end(lane, C.byref(out), None, None) == 0
        want = torch.empty_like(x)
        torch.cuda.synchronize()
        assert lib.bsq_lane_decompress_begin(lane, out, 0, want.data_ptr(), rows * cols) == 0
        assert lib.bsq_lane_decompress_end(lane) == 0
        for off in (4, 1):                                    # on a 16-byte boundary and off it
            y = room[off: off + rows * cols]
            assert lib.bsq_lane_decompress_begin(lane, C.byref(hdr), 1, y.data_ptr(), rows * cols) == 0
            assert lib.bsq_lane_decompress_end(lane) == 0
            torch.cuda.synchronize()
            assert torch.equal(y.view(torch.int32), want.view(torch.int32).reshape(-1)), off
            assert (room[:off] == 7.0).all() and (room[off + rows * cols:] == 7.0).all()
            room.fill_(7.0)
            torch.cuda.synchronize()
        lib.bsq_free(out)
    finally:
        lib.bsq_lane_destroy(lane)


@pytest.mark.parametrize("q", [10, 11])
@pytest.mark.parametrize("case", LONG_CASES)
def test_long_lists_behind_the_decode_give_the_host_objects_bits(pkg, lib, case, q):
    test_one_launch_gives_the_host_objects_bits(pkg, lib, case, q)


@pytest.mark.parametrize("case,apart", [(c, True) for c in LONG_CASES] + [((8, 9216, 0.0074, 0.0015), False), ((256, 1024, 0.01, 0.0), False),
                                                                          ((1024, 4096, 0.01, 0.01), False)])
def test_long_lists_take_a_kernel_of_their_own(pkg, lib, case, apart):
    """A warp that looks through thousands of entries for each of its batches takes up to four times as long as the lists added behind the decode."""
    rows, cols, outlier, error = case
    x = torch.randn(rows, cols, device="cuda")
    comp = importlib.import_module(pkg.__name__ + ".torch_api").Compressor(rows, cols, outlier=outlier, error=error, q=10)
    packed = comp.compress(x)
    comp.decompress(packed)
    torch.cuda.synchronize()
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as trace:
        comp.decompress(packed)
        torch.cuda.synchronize()
    names = [e.key for e in trace.key_averages()]
    comp.close()
    assert any("decode_flat_kernel" in n for n in names) and any("topk_apply" in n for n in names) == apart, names


def test_refused_object_leaves_the_result_alone(pkg, lib):
    """The kernel is launched before the host knows what the payload's headers say; a header that differs in any checked byte keeps
    it from writing, and a column that the matrix does not have fails the call."""
    refused(pkg, lib, 0.02)


def test_refused_object_with_long_lists_leaves_the_result_alone(pkg, lib):
    """Here the lists' kernel is launched when the headers are known to be good."""
    refused(pkg, lib, 0.7)


def refused(pkg, lib, ratio):
    rows, cols = 96, 640
    x = torch.randn(rows, cols, device="cuda", generator=torch.Generator(device="cuda").manual_seed(3))
    lane = lib.bsq_lane_create(rows, cols, ratio, ratio, -1, 1, -1, -1, 10)
    assert lane
    try:
        cap = int(lib.bsq_lane_packed_capacity(lane))
        buf = torch.empty(cap, dtype=torch.uint8, device="cuda")
        torch.cuda.synchronize()
        hdr = pkg.Array()
        assert lib.bsq_lane_compress_begin(lane, x.data_ptr(), 1, buf.data_ptr(), cap) == 0
        assert lib.bsq_lane_compress_end(lane, None, C.byref(hdr), None) == 0
        y = torch.full_like(x, 7.0)
        direct, err = 200 + hdr.section_direct.offset, 200 + hdr.section_error_topk.offset
        for at in (direct + 3, direct + 4, direct + 8, direct + 17, direct + 39, 200 + hdr.section_outlier_topk.offset, err + 2, err + 5):
            good = int(buf[at])
            buf[at] = good ^ 0x10
            torch.cuda.synchronize()
            assert lib.bsq_lane_decompress_begin(lane, C.byref(hdr), 1, y.data_ptr(), rows * cols) == 1, at
            torch.cuda.synchronize()
            assert (y == 7.0).all(), at
            buf[at] = good
        good = buf[err + 8: err + 10].clone()
        buf[err + 8: err + 10] = 0xFF                         # column 65535 of 640
        torch.cuda.synchronize()
        assert lib.bsq_lane_decompress_begin(lane, C.byref(hdr), 1, y.data_ptr(), rows * cols) == 0
        assert lib.bsq_lane_decompress_end(lane) == 1
        buf[err + 8: err + 10] = good
        torch.cuda.synchronize()
        assert lib.bsq_lane_decompress_begin(lane, C.byref(hdr), 1, y.data_ptr(), rows * cols) == 0
        assert lib.bsq_lane_decompress_end(lane) == 0
    finally:
        lib.bsq_lane_destroy(lane)


# rows, cols, outlier, error, rank, uv: factors coded both ways and kept in FP32, off 8-byte boundaries, a rank with more singular values than
# the kernel keeps in shared memory, factors of less than a batch, with no, one and two lists
FACTOR_CASES = [
    (777, 1031, 0.005, 0.0, 48, -1), (1024, 640, 0.0, 0.0, 64, -1), (1100, 1090, 0.01, 0.0, 1030, -1), (96, 70, 0.02, 0.02, 7, 11),
    (1024, 1536, 0.01, 0.02, 64, 10), (640, 2048, 0.0, 0.02, 40, 11), (515, 1001, 0.01, 0.01, 33, 10), (1024, 1024, 0.0, 0.02, 32, -1),
]


@pytest.mark.parametrize("case", FACTOR_CASES)
def test_opened_factors_give_the_host_objects_bits(pkg, lib, case):
    """Factors opened in place by one kernel, their maxima taken on the way, against the route of a host object, which copies and decodes
    section by section and finds the maxima in passes of their own."""
    rows, cols, outlier, error, rank, uv = case
    x = torch.randn(rows, cols, device="cuda", generator=torch.Generator(device="cuda").manual_seed(rows + rank))
    lane = lib.bsq_lane_create(rows, cols, outlier, error, rank, 1, uv, -1, -1)
    assert lane
    try:
        cap = int(lib.bsq_lane_packed_capacity(lane))
        buf = torch.empty(cap, dtype=torch.uint8, device="cuda")
        torch.cuda.synchronize()
        hdr, out = pkg.Array(), C.c_void_p(None)
        assert lib.bsq_lane_compress_begin(lane, x.data_ptr(), 1, buf.data_ptr(), cap) == 0
        assert lib.bsq_lane_compress_end(lane, None, C.byref(hdr), None) == 0
        host = buf.cpu().numpy()
        out = lib.bsq_load_from_buffer(host.ctypes.data, host.size)
        assert out
        want, got = torch.empty_like(x), torch.full_like(x, 7.0)
        torch.cuda.synchronize()
        assert lib.bsq_lane_decompress_begin(lane, out, 0, want.data_ptr(), rows * cols) == 0
        assert lib.bsq_lane_decompress_end(lane) == 0
        if uv != -1:                                          # V's block count: refused before the result is touched
            at = 200 + hdr.section_v.offset + 24
            buf[at] ^= 1
            torch.cuda.synchronize()
            assert lib.bsq_lane_decompress_begin(lane, C.byref(hdr), 1, got.data_ptr(), rows * cols) == 1
            buf[at] ^= 1
            torch.cuda.synchronize()
            assert (got == 7.0).all()
        for _ in range(2):                                    # (the second call finds the words as the first one left them)
            torch.cuda.synchronize()
            assert lib.bsq_lane_decompress_begin(lane, C.byref(hdr), 1, got.data_ptr(), rows * cols) == 0
            assert lib.bsq_lane_decompress_end(lane) == 0
            torch.cuda.synchronize()
            assert torch.equal(got.view(torch.int32), want.view(torch.int32))
            got.fill_(7.0)
        lib.bsq_free(out)
    finally:
        lib.bsq_lane_destroy(lane)
