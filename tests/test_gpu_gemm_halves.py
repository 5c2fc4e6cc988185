"""Products with a bound on |A| split their operands into FP16 halves at every width up to 256 columns (csrc/bsq_gemm.cu, bsq_gemm_tma.cu); up to 128
columns the hi * hi terms go to two accumulators in turn.  Compared with FP64."""
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
