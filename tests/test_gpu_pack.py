"""Device-resident objects are assembled and read back by kernels of their own (csrc/bsq_pack.cu): the same bytes as the host
object, whatever the alignment of the caller's buffer and of the sections inside it, and the same matrix when they are read."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

# rows, cols, outlier, error, rank, uv, s, q: sections that end on every alignment (odd list lengths, odd code counts), objects
# of less than one 16-byte unit per piece and of more than one CTA's share (32 KB) per piece, with and without an error list
CASES = [
    (1, 1, 0.0, 0.0, -1, -1, -1, 11),
    (3, 5, 0.3, 0.3, -1, -1, -1, 10),
    (7, 64, 0.02, 0.0, -1, -1, -1, 10),
    (33, 77, 0.04, 0.04, -1, -1, -1, 11),
    (256, 1024, 0.01, 0.0, -1, -1, -1, 10),
    (515, 1001, 0.0, 0.0, -1, -1, -1, -1),
    (129, 203, 0.02, 0.02, 13, 10, 11, -1),
    (512, 640, 0.01, 0.0, 32, -1, -1, -1),
    (300, 257, 0.01, 0.01, 21, 11, -1, -1),
]


@pytest.mark.parametrize("case", CASES)
@pytest.mark.parametrize("off", [0, 1, 6, 12])
def test_device_object_equals_host_object_at_any_alignment(pkg, lib, case, off):
    rows, cols, outlier, error, rank, uv, s, q = case
    g = torch.Generator(device="cuda").manual_seed(rows * 7 + cols)
    x = torch.randn(rows, cols, device="cuda", generator=g)
    lane = lib.bsq_lane_create(rows, cols, outlier, error, rank, 2, uv, s, q)
    assert lane
    try:
        cap = int(lib.bsq_lane_packed_capacity(lane))
        buf = torch.full((cap + 64,), 0xA5, dtype=torch.uint8, device="cuda")
        torch.cuda.synchronize()
        hdr, size, out = pkg.Array(), C.c_uint64(0), C.c_void_p(None)
        assert lib.bsq_lane_compress_begin(lane, x.data_ptr(), 1, buf.data_ptr() + off, cap) == 0
        assert lib.bsq_lane_compress_end(lane, None, C.byref(hdr), C.byref(size)) == 0
        assert lib.bsq_lane_compress_begin(lane, x.data_ptr(), 1, None, 0) == 0
        assert lib.bsq_lane_compress_end(lane, C.byref(out), None, None) == 0
        n = int(lib.bsq_get_packed_size(out))
        host = np.frombuffer(C.string_at(out.value, n), np.uint8).copy()
        assert int(size.value) == n <= cap
        got = buf.cpu().numpy()
        assert (got[:off] == 0xA5).all() and (got[off + cap:] == 0xA5).all()       # nothing outside the object
        dev = got[off: off + n].copy()
        assert dev[192:200].view(np.uint64)[0] == buf.data_ptr() + off + 200
        dev[192:200] = 0
        host[192:200] = 0
        assert np.array_equal(dev, host)
        y_dev = torch.empty_like(x)
        y_host = torch.empty_like(x)
        torch.cuda.synchronize()
        assert lib.bsq_lane_decompress_begin(lane, C.byref(hdr), 1, y_dev.data_ptr(), rows * cols) == 0
        assert lib.bsq_lane_decompress_end(lane) == 0
        assert lib.bsq_lane_decompress_begin(lane, out, 0, y_host.data_ptr(), rows * cols) == 0
        assert lib.bsq_lane_decompress_end(lane) == 0
        torch.cuda.synchronize()
        assert torch.equal(y_dev.view(torch.int32), y_host.view(torch.int32))
        lib.bsq_free(out)
    finally:
        lib.bsq_lane_destroy(lane)


def test_damaged_device_object_is_refused(pkg, lib):
    """The headers inside a device-resident payload are checked as those of a host object are, before anything is decoded."""
    rows, cols = 64, 128
    x = torch.randn(rows, cols, device="cuda")
    lane = lib.bsq_lane_create(rows, cols, 0.02, 0.0, -1, 1, -1, -1, 11)
    try:
        cap = int(lib.bsq_lane_packed_capacity(lane))
        buf = torch.empty(cap, dtype=torch.uint8, device="cuda")
        torch.cuda.synchronize()
        hdr = pkg.Array()
        assert lib.bsq_lane_compress_begin(lane, x.data_ptr(), 1, buf.data_ptr(), cap) == 0
        assert lib.bsq_lane_compress_end(lane, None, C.byref(hdr), None) == 0
        y = torch.empty_like(x)
        for at in (200 + hdr.section_direct.offset, 200 + hdr.section_outlier_topk.offset + 4):      # magic number, list length
            good = int(buf[at])
            buf[at] = good ^ 0x80
            torch.cuda.synchronize()
            assert lib.bsq_lane_decompress_begin(lane, C.byref(hdr), 1, y.data_ptr(), rows * cols) == 1
            buf[at] = good
        torch.cuda.synchronize()
        assert lib.bsq_lane_decompress_begin(lane, C.byref(hdr), 1, y.data_ptr(), rows * cols) == 0
        assert lib.bsq_lane_decompress_end(lane) == 0
    finally:
        lib.bsq_lane_destroy(lane)


# quantised matrices with no, one and two lists, low-rank objects with lists, sections that are read in place and ones that are not
OVERLAP_CASES = [
    (64, 512, 0.0, 0.0, -1, -1, -1, 11),
    (192, 1024, 0.02, 0.0, -1, -1, -1, 10),
    (192, 1024, 0.0, 0.02, -1, -1, -1, 11),
    (256, 768, 0.01, 0.02, -1, -1, -1, 10),
    (33, 77, 0.04, 0.04, -1, -1, -1, 11),
    (512, 640, 0.01, 0.01, 32, 11, -1, -1),
    (512, 640, 0.01, 0.0, 16, -1, -1, -1),
]


@pytest.mark.parametrize("case", OVERLAP_CASES)
def test_result_may_lie_over_the_object(pkg, lib, case):
    """One buffer holds the object and receives the matrix: the object at the end, in the middle and at the front of it, and
    ending just inside and just outside.  Same bits as into a buffer of its own."""
    rows, cols, outlier, error, rank, uv, s, q = case
    g = torch.Generator(device="cuda").manual_seed(rows + cols)
    x = torch.randn(rows, cols, device="cuda", generator=g)
    lane = lib.bsq_lane_create(rows, cols, outlier, error, rank, 2, uv, s, q)
    assert lane
    try:
        cap = int(lib.bsq_lane_packed_capacity(lane))
        obj = torch.empty(cap, dtype=torch.uint8, device="cuda")
        hdr, size = pkg.Array(), C.c_uint64(0)
        torch.cuda.synchronize()
        assert lib.bsq_lane_compress_begin(lane, x.data_ptr(), 1, obj.data_ptr(), cap) == 0
        assert lib.bsq_lane_compress_end(lane, None, C.byref(hdr), C.byref(size)) == 0
        n = int(size.value)
        want = torch.empty_like(x)
        torch.cuda.synchronize()
        assert lib.bsq_lane_decompress_begin(lane, C.byref(hdr), 1, want.data_ptr(), rows * cols) == 0
        assert lib.bsq_lane_decompress_end(lane) == 0
        out_bytes, front = rows * cols * 4, (cap + 255) // 256 * 256
        # where the object starts, counted from the start of the matrix
        last = (out_bytes - n) // 16 * 16
        for at in (last, last // 2 // 4 * 4, 0, -200 + 4 * 64, 64 - n // 64 * 64, -((n + 63) // 64 * 64), out_bytes, last + 2):
            arena = torch.zeros(front + out_bytes + cap, dtype=torch.uint8, device="cuda")
            where = arena.data_ptr() + front + at
            arena[front + at: front + at + n] = obj[:n]
            moved = pkg.Array.from_buffer_copy(hdr)
            moved.payload = where + 200
            torch.cuda.synchronize()
            assert lib.bsq_lane_decompress_begin(lane, C.byref(moved), 1, arena.data_ptr() + front, rows * cols) == 0, at
            assert lib.bsq_lane_decompress_end(lane) == 0, at
            torch.cuda.synchronize()
            got = arena[front: front + out_bytes].view(torch.int32)
            assert torch.equal(got, want.view(torch.int32).reshape(-1)), at
    finally:
        lib.bsq_lane_destroy(lane)


@pytest.mark.parametrize("case", [(33, 77, 0.04, 0.04, -1, -1, -1, 11), (256, 1024, 0.01, 0.0, -1, -1, -1, 10), (129, 203, 0.02, 0.02, 13, 10, 11, -1),
                                  (515, 1001, 0.0, 0.0, -1, -1, -1, -1)])
def test_objects_in_memory_that_kernels_do_not_reach(pkg, lib, case):
    """Page-locked host memory handed over as the object's buffer stands for all memory that is not this device's own (another
    GPU's): stream copies move it, with the same bytes as ever.  Memory that CUDA does not know is refused on the host, both
    ways, before anything is launched on it, and the lane goes on working."""
    rows, cols, outlier, error, rank, uv, s, q = case
    g = torch.Generator(device="cuda").manual_seed(rows + cols)
    x = torch.randn(rows, cols, device="cuda", generator=g)
    lane = lib.bsq_lane_create(rows, cols, outlier, error, rank, 2, uv, s, q)
    assert lane
    try:
        cap = int(lib.bsq_lane_packed_capacity(lane))
        pinned = torch.full((cap,), 0xA5, dtype=torch.uint8).pin_memory()
        pageable = np.zeros(cap, np.uint8)
        hdr, size, out = pkg.Array(), C.c_uint64(0), C.c_void_p(None)
        torch.cuda.synchronize()
        assert lib.bsq_lane_compress_begin(lane, x.data_ptr(), 1, pageable.ctypes.data, cap) == 1
        assert not pageable.any()
        assert lib.bsq_lane_compress_begin(lane, x.data_ptr(), 1, pinned.data_ptr(), cap) == 0
        assert lib.bsq_lane_compress_end(lane, None, C.byref(hdr), C.byref(size)) == 0
        assert lib.bsq_lane_compress_begin(lane, x.data_ptr(), 1, None, 0) == 0
        assert lib.bsq_lane_compress_end(lane, C.byref(out), None, None) == 0
        n = int(size.value)
        host = np.frombuffer(C.string_at(out.value, n), np.uint8).copy()
        got = pinned.numpy()[:n].copy()
        assert int(lib.bsq_get_packed_size(out)) == n and hdr.payload == pinned.data_ptr() + 200
        host[192:200] = got[192:200]
        assert np.array_equal(got, host)
        y_host, y = torch.empty_like(x), torch.empty_like(x)
        torch.cuda.synchronize()
        assert lib.bsq_lane_decompress_begin(lane, out, 0, y_host.data_ptr(), rows * cols) == 0
        assert lib.bsq_lane_decompress_end(lane) == 0
        if q != pkg.NONE or rank > 0:                         # an object without inner headers was never looked into
            pageable[:n] = got
            bad = pkg.Array.from_buffer_copy(hdr)
            bad.payload = pageable.ctypes.data + 200
            assert lib.bsq_lane_decompress_begin(lane, C.byref(bad), 1, y.data_ptr(), rows * cols) == 1
        assert lib.bsq_lane_decompress_begin(lane, C.byref(hdr), 1, y.data_ptr(), rows * cols) == 0
        assert lib.bsq_lane_decompress_end(lane) == 0
        torch.cuda.synchronize()
        assert torch.equal(y.view(torch.int32), y_host.view(torch.int32))
        lib.bsq_free(out)
    finally:
        lib.bsq_lane_destroy(lane)


@pytest.mark.parametrize("where", ["device", "pinned"])
@pytest.mark.parametrize("case", [(256, 1024, 0.01, 0.0, -1, -1, -1, 10), (129, 203, 0.02, 0.02, 13, 10, 11, -1)])
def test_failed_compress_leaves_no_object(pkg, lib, case, where):
    """A call whose status word is set (from the host, no kernel fails) returns 1 and leaves a zeroed header, also in a buffer
    that held a good object before; the lane's next call is a good one again."""
    rows, cols, outlier, error, rank, uv, s, q = case
    x = torch.randn(rows, cols, device="cuda", generator=torch.Generator(device="cuda").manual_seed(rows))
    lane = lib.bsq_lane_create(rows, cols, outlier, error, rank, 2, uv, s, q)
    assert lane
    try:
        cap = int(lib.bsq_lane_packed_capacity(lane))
        buf = torch.zeros(cap, dtype=torch.uint8, device="cuda") if where == "device" else torch.zeros(cap, dtype=torch.uint8).pin_memory()
        hdr, size = pkg.Array(), C.c_uint64(0)

        def compress():
            torch.cuda.synchronize()
            assert lib.bsq_lane_compress_begin(lane, x.data_ptr(), 1, buf.data_ptr(), cap) == 0
            return lib.bsq_lane_compress_end(lane, None, C.byref(hdr), C.byref(size))
        assert compress() == 0
        good = buf.cpu().numpy().copy()
        lib.bsq_test_inject_lane_status(lane, 0, 1)           # "a bounded wait ran out"
        assert compress() == 1
        left = buf.cpu().numpy().copy()
        assert not left[:200].any()
        y = torch.empty_like(x)
        obj = lib.bsq_load_from_buffer(left.ctypes.data, left.size)
        if obj:
            assert lib.bsq_lane_decompress_begin(lane, obj, 0, y.data_ptr(), rows * cols) == 1
            lib.bsq_free(obj)
        assert compress() == 0
        assert np.array_equal(buf.cpu().numpy(), good)
        lib.bsq_test_inject_lane_status(lane, 1, 1)
        for want in (1, 0):
            assert lib.bsq_lane_decompress_begin(lane, C.byref(hdr), 1, y.data_ptr(), rows * cols) == 0
            assert lib.bsq_lane_decompress_end(lane) == want
    finally:
        lib.bsq_lane_destroy(lane)
