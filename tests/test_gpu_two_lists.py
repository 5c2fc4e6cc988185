"""Decompress with an error list and an outlier list: one launch (a warp per row) or two, chosen by the lists' lengths, the rows and the
entries in all (topk_apply_two).  Both against the CPU oracle, bit for bit, on both sides of every line of that rule."""
import ctypes as C

import numpy as np
import pytest

from conftest import bits

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

# rows, cols, error entries, outlier entries per row
SHAPES = [
    (2, 70, 1, 1), (3, 300, 1, 128), (9, 700, 127, 256), (9, 1000, 300, 200),       # up to five trips of 128 entries: one launch
    (9, 1000, 300, 300), (64, 1024, 700, 700),                             # more, few rows: two
    (511, 6000, 500, 400), (512, 6000, 500, 400), (512, 6000, 500, 600),   # eight trips from 512 rows on, nine
    (4100, 2048, 170, 171), (4108, 2048, 170, 171), (4100, 2048, 1, 370),         # 1.398 and 1.401 million entries, in four trips and three
    (511, 1000, 100, 100), (512, 1000, 100, 100), (512, 1000, 900, 700), (511, 1000, 1000, 700), (600, 2000, 399, 400),      # dense lists
]


@pytest.mark.parametrize("shape", SHAPES)
def test_two_lists_match_oracle(pkg, lib, oracle, shape):
    rows, cols, ke, ko = shape
    rng = np.random.default_rng(rows + cols + ke)
    x = rng.standard_normal((rows, cols)).astype(np.float32)
    outlier, error = np.float32(ko / cols), np.float32(ke / cols)
    assert oracle.topk_num_columns(cols, outlier) == ko and oracle.topk_num_columns(cols, error) == ke
    lane = lib.bsq_lane_create(rows, cols, float(outlier), float(error), -1, 1, -1, -1, 11)
    assert lane
    try:
        cap = int(lib.bsq_lane_packed_capacity(lane))
        buf = torch.empty(cap, dtype=torch.uint8, device="cuda")
        d_x = torch.from_numpy(x).cuda()
        torch.cuda.synchronize()
        hdr, size = pkg.Array(), C.c_uint64(0)
        assert lib.bsq_lane_compress_begin(lane, d_x.data_ptr(), 1, buf.data_ptr(), cap) == 0
        assert lib.bsq_lane_compress_end(lane, None, C.byref(hdr), C.byref(size)) == 0
        assert hdr.flags & pkg.FLAG_ERROR and hdr.flags & pkg.FLAG_OUTLIER
        packed = buf[: int(size.value)].cpu().numpy()
        sections = ((hdr.section_error_topk, ke), (hdr.section_outlier_topk, ko))
        # lists of our own: every row of both starts with the same columns, with values that round differently in the other order
        first = None
        for sec, k in sections:
            at = 200 + sec.offset + 8
            idx = np.argsort(rng.random((rows, cols)), axis=1)[:, :k].astype(np.uint16)
            if first is None:
                first = idx
            else:
                both = min(ke, ko)
                idx = np.concatenate([first[:, :both], np.stack([np.setdiff1d(np.arange(cols), first[r, :both])[: k - both] for r in range(rows)])],
                                     axis=1).astype(np.uint16) if k > both else first[:, :k].copy()
            val = (rng.standard_normal((rows, k)) * 10.0 ** rng.integers(-3, 4, (rows, k))).astype(np.float32)
            packed[at: at + rows * k * 2] = np.ascontiguousarray(idx).view(np.uint8).ravel()
            packed[at + rows * k * 2: at + rows * k * 6] = val.view(np.uint8).ravel()
        want = oracle.decompress_nosvd(packed, rows, cols)
        buf[: packed.size] = torch.from_numpy(packed).cuda()
        y = torch.empty(rows, cols, device="cuda")
        torch.cuda.synchronize()
        assert lib.bsq_lane_decompress_begin(lane, C.byref(hdr), 1, y.data_ptr(), rows * cols) == 0
        assert lib.bsq_lane_decompress_end(lane) == 0
        torch.cuda.synchronize()
        assert np.array_equal(bits(y.cpu().numpy()), bits(want))
        # a column out of range in either list, the last entry of the last row: skipped and reported
        for sec, k in sections:
            at = 200 + sec.offset + 8 + rows * k * 2 - 1                   # high byte
            good = int(buf[at])
            buf[at] = 0xFF
            torch.cuda.synchronize()
            assert lib.bsq_lane_decompress_begin(lane, C.byref(hdr), 1, y.data_ptr(), rows * cols) == 0
            assert lib.bsq_lane_decompress_end(lane) == 1
            buf[at] = good
        torch.cuda.synchronize()
        assert lib.bsq_lane_decompress_begin(lane, C.byref(hdr), 1, y.data_ptr(), rows * cols) == 0
        assert lib.bsq_lane_decompress_end(lane) == 0
        torch.cuda.synchronize()
        assert np.array_equal(bits(y.cpu().numpy()), bits(want))
    finally:
        lib.bsq_lane_destroy(lane)
