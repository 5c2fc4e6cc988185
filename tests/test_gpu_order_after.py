"""bsq_lane_order_after: a call comes behind the work that is on the caller's stream, and behind everything that an event recorded there would come behind:
the legacy default stream and blocking streams wait for one another.  Producers are still running when the call is made."""
import ctypes as C
import importlib
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

from conftest import ROOT  # noqa: E402

ROWS, COLS = 256, 1024


@pytest.fixture(scope="module")
def streams():
    s = C.c_void_p()
    assert int(torch.cuda.cudart().cudaStreamCreate(C.addressof(s))) == 0
    made = {"legacy": torch.cuda.default_stream(), "blocking": torch.cuda.ExternalStream(s.value), "nonblocking": torch.cuda.Stream()}
    assert made["legacy"].cuda_stream == 0
    return made


@pytest.fixture(scope="module")
def comp(pkg, lib):
    c = importlib.import_module(pkg.__name__ + ".torch_api").Compressor(ROWS, COLS, outlier=0.01, q=pkg.NF4_DQ)
    yield c
    c.close()


@pytest.mark.parametrize("producer,current", [("legacy", "legacy"), ("legacy", "blocking"), ("blocking", "legacy"), ("blocking", "blocking"),
                                              ("nonblocking", "nonblocking")])
def test_calls_come_behind_producers_that_still_run(comp, streams, producer, current):
    x = torch.randn(ROWS, COLS, device="cuda", generator=torch.Generator(device="cuda").manual_seed(3))
    want = comp.compress(x)
    back = comp.decompress(want)
    d_x, d_packed = torch.zeros_like(x), torch.zeros_like(want.data)
    late = type(want)(d_packed, type(want.header).from_buffer_copy(want.header), want.nbytes)
    late.header.payload = d_packed.data_ptr() + 200
    torch.cuda.synchronize()
    with torch.cuda.stream(streams[producer]):
        torch.cuda._sleep(100_000_000)                        # 50 ms
        d_x.copy_(x)
        d_packed.copy_(want.data)
    with torch.cuda.stream(streams[current]):
        got = comp.compress(d_x)
    torch.cuda.synchronize()
    assert torch.equal(got.data[200: got.nbytes], want.data[200: want.nbytes])
    d_packed.zero_()
    torch.cuda.synchronize()
    with torch.cuda.stream(streams[producer]):
        torch.cuda._sleep(100_000_000)
        d_packed.copy_(want.data)
    with torch.cuda.stream(streams[current]):
        y = comp.decompress(late)
    torch.cuda.synchronize()
    assert torch.equal(y.view(torch.int32), back.view(torch.int32))


def test_a_stream_that_is_being_captured_stays_so(comp, lib):
    """Asked for its state it would end the capture.  The lane's stream joins by the event and leaves by another one."""
    s, g = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    lane = torch.cuda.ExternalStream(lib.bsq_lane_stream(comp._lane, 0))
    a, b = torch.ones(64, device="cuda"), torch.zeros(64, device="cuda")
    torch.cuda.synchronize()
    with torch.cuda.stream(s):
        g.capture_begin()
        b.add_(a)
        assert lib.bsq_lane_order_after(comp._lane, 0, s.cuda_stream) == 0
        s.wait_stream(lane)
        b.add_(a)
        g.capture_end()
    g.replay()
    torch.cuda.synchronize()
    assert torch.equal(b, 2 * a)
    x = torch.randn(ROWS, COLS, device="cuda")                # the lane goes on as before
    assert torch.equal(comp.compress(x).data[200:1200], comp.compress(x).data[200:1200])


def test_waiting_for_other_work_is_left_to_the_device_flags():
    """A process whose context asks for waits that sleep: a decompress call behind 0.3 s of other work does not keep a core busy until its kernel's answer
    comes.  (The limit of a quarter: such a wait takes next to none of it, polling takes all.)"""
    code = """
import ctypes, time
cuda = ctypes.CDLL("libcuda.so.1")
assert cuda.cuInit(0) == 0 and cuda.cuDevicePrimaryCtxSetFlags_v2(0, 4) == 0         # CU_CTX_SCHED_BLOCKING_SYNC
import importlib, torch, __graft_entry__
pkg = __graft_entry__.load_package()
comp = importlib.import_module(pkg.__name__ + ".torch_api").Compressor(256, 1024, outlier=0.01, q=pkg.NF4_DQ)
x = torch.randn(256, 1024, device="cuda")
packed = comp.compress(x)
want = comp.decompress(packed)
torch.cuda.synchronize()
torch.cuda._sleep(600_000_000)
wall, cpu = time.perf_counter(), time.thread_time()
got = comp.decompress(packed)
wall, cpu = time.perf_counter() - wall, time.thread_time() - cpu
assert torch.equal(got, want) and wall > 0.1, wall
assert cpu < 0.25 * wall, (cpu, wall)
"""
    done = subprocess.run([sys.executable, "-c", code], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert done.returncode == 0, done.stderr[-2000:]
