"""The compress / decompress work that is timed, as a user's program calls it.

Each case is one setting of `bitsqz_llm_compress_initialize` (shape, top-k ratios, rank, formats) and what is done with
it.  Values follow the workloads of `bitsqueeze-llm_b200/workloads.py`: Gaussian activations with a few scaled-up columns
for the quantiser-only settings, a decaying spectrum plus noise (with outlier columns and heavy tails) for the low-rank ones.

  encode      matrix on the GPU -> packed object on the GPU           (Compressor.compress)
  decode      packed object on the GPU -> matrix on the GPU           (Compressor.decompress)
  roundtrip   both, for the low-rank settings: single singular vectors are defined up to sign and, in a flat spectrum, up
              to rounding, so what can be compared is the singular values, the outlier lists and the matrix that comes back
  dropin      pageable host matrix -> host object -> matrix on the GPU (bitsqz_llm_compress / bitsqz_llm_decompress)
  batch       several matrices in flight, compress all, decompress all (bsq_batch_compress / bsq_batch_decompress)
"""
import ctypes
import ctypes.util
import glob
import importlib
import os

import numpy as np
import torch

import __graft_entry__

PKG = __graft_entry__.load_package()
TORCH_API = importlib.import_module(PKG.__name__ + ".torch_api")
FORMATS = {"none": PKG.NONE, "nf4": PKG.NF4, "nf4_dq": PKG.NF4_DQ}


def _case(name, kind, rows, cols, outlier=0.0, error=0.0, rank=-1, niters=2, uv="none", s="none", q="none", count=1):
    c = dict(kind=kind, rows=rows, cols=cols, outlier=outlier, error=error, rank=rank, niters=niters, uv=uv, s=s, q=q, count=count)
    return dict(c, name=name) if name else c


def listed():
    return [
        # the smallest call: a decode step's activations of a few requests; launches and copies are all there is
        _case("encode_nf4dq_256x1024", "encode", 256, 1024, outlier=0.01, q="nf4_dq"),
        # the quantiser alone through the reference's own interface, on host data as its tests and example call it
        _case("dropin_nf4_1024x1024", "dropin", 1024, 1024, q="nf4"),
        # one layer's activations: outliers kept, the rest quantised; both directions
        _case("encode_nf4dq_4096x4096", "encode", 4096, 4096, outlier=0.01, q="nf4_dq"),
        _case("decode_nf4dq_4096x4096", "decode", 4096, 4096, outlier=0.01, q="nf4_dq"),
        # a ragged shape (not a multiple of the 64-element block, rows not 16-byte aligned), with error correction
        _case("encode_nf4_ec_1501x3001", "encode", 1501, 3001, outlier=0.005, error=0.01, q="nf4"),
        # small and ragged low-rank calls
        _case("roundtrip_r48_777x1031", "roundtrip", 777, 1031, outlier=0.005, rank=48),
        _case("roundtrip_r64_2048x5120", "roundtrip", 2048, 5120, outlier=0.005, error=0.01, rank=64, uv="nf4_dq"),
        # low-rank factors kept in FP32
        _case("roundtrip_r128_8192x4096", "roundtrip", 8192, 4096, rank=128),
        # everything on: outliers, rank 256, NF4 factors, error correction; and its decode (weights or a cache read often)
        _case("roundtrip_r256_8192x4096", "roundtrip", 8192, 4096, outlier=0.005, error=0.01, rank=256, uv="nf4"),
        _case("decode_r256_4096x14336", "decode", 4096, 14336, outlier=0.005, error=0.01, rank=256, uv="nf4"),
        # the layers of a model, eight MLP activations in flight
        _case("batch8_r256_4096x14336", "batch", 4096, 14336, outlier=0.005, error=0.01, rank=256, uv="nf4", count=8),
    ]


def _log(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(["encode", "encode", "decode", "decode", "roundtrip", "roundtrip", "dropin", "batch"])
    odd = rng.random() < 0.4                                  # any size; otherwise multiples of 64
    most = 4096 * 14336
    while True:
        rows, cols = _log(rng, 64, 8192), _log(rng, 256, 14336)
        if kind in ("dropin", "batch"):
            rows, cols = _log(rng, 64, 2048), _log(rng, 256, 4096)
        if not odd:
            rows, cols = max(64, rows // 64 * 64), cols // 64 * 64
        if rows * cols <= most:
            break
    outlier = rng.choice([0.0, 0.005, 0.01, 0.02])
    lowrank = kind in ("roundtrip", "batch") or (kind in ("decode", "dropin") and rng.random() < 0.5)
    if not lowrank:
        return _case(None, kind, rows, cols, outlier=outlier, error=rng.choice([0.0, 0.0, 0.01]), q=rng.choice(["nf4", "nf4_dq"]))
    rank = min(_log(rng, 8, 256), min(rows, cols) // 2)
    uv = rng.choice(["none", "nf4", "nf4_dq"])
    # error correction goes with quantised factors (it is what corrects their error)
    error = rng.choice([0.0, 0.01]) if uv != "none" else 0.0
    return _case(None, kind, rows, cols, outlier=outlier, error=error, rank=rank, niters=rng.choice([1, 2, 2]), uv=uv,
                 count=rng.choice([2, 4, 6]) if kind == "batch" else 1)


# ---- inputs ----------------------------------------------------------------------------------------------------------
def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _matrix(case, seed):
    """FP32 on the GPU.  Quantiser only: N(0,1), 0.1 % of the columns scaled by U[20,100].  Low rank: 1/i spectrum of up to
    512 components plus 0.01 N(0,1); with outlier separation also 0.05 % of the columns x 50 and 1 % Student-t(3) entries."""
    g, rows, cols = _generator(seed), case["rows"], case["cols"]

    def randn(*shape):
        return torch.randn(*shape, device="cuda", generator=g)

    if case["rank"] < 1:
        a = randn(rows, cols)
        chosen = torch.randperm(cols, device="cuda", generator=g)[: max(1, round(0.001 * cols))]
        a[:, chosen] *= 20.0 + 80.0 * torch.rand(chosen.numel(), device="cuda", generator=g)
        return a
    comp = min(512, rows, cols)
    sv = 1.0 / torch.arange(1, comp + 1, device="cuda", dtype=torch.float32)
    a = (randn(rows, comp) * (sv / (rows * cols) ** 0.5)) @ randn(cols, comp).T
    a += 0.01 * randn(rows, cols)
    if case["outlier"] > 0:
        chosen = torch.randperm(cols, device="cuda", generator=g)[: max(1, round(0.0005 * cols))]
        a[:, chosen] *= 50.0
        mask = torch.rand(rows, cols, device="cuda", generator=g) < 0.01
        chi = randn(rows, cols).square_().add_(randn(rows, cols).square_()).add_(randn(rows, cols).square_())
        a += torch.where(mask, 0.01 * randn(rows, cols) / (chi / 3.0).sqrt(), torch.zeros((), device="cuda"))
    return a


def _section_fill(case, packed, seed):
    """Gives an object made by the framework contents of its own, from the seed alone: codes, scales, factors and lists as a
    compressed matrix has them, so that what decode reads does not depend on the compress side."""
    g, data, hdr = _generator(seed + 77), packed.data, packed.header
    rows, cols, rank = case["rows"], case["cols"], hdr.effective_rank

    def put(at, tensor):
        raw = tensor.contiguous().view(torch.uint8).reshape(-1)
        data[200 + at: 200 + at + raw.numel()] = raw

    def quant(sec, fmt, n, size):
        nb, at = (n + 63) // 64, sec.offset + 48
        scales = size * (0.5 + torch.rand(nb, device="cuda", generator=g))
        if fmt == "nf4":
            put(at, scales)
            at += nb * 4
        else:
            put(sec.offset + 40, torch.full((1,), size * 1.5 / 448.0, device="cuda"))
            put(at, (scales / (size * 1.5 / 448.0)).to(torch.float8_e4m3fn))
            at += nb
        codes = torch.randint(0, 256, ((n + 1) // 2,), device="cuda", generator=g, dtype=torch.uint8)
        if n & 1:
            codes[-1] &= 0xF0
        put(at, codes)

    def fp32(sec, n, size):
        put(sec.offset, size * torch.randn(n, device="cuda", generator=g))

    def topk(sec, k, size):
        idx = torch.rand(rows, cols, device="cuda", generator=g).topk(k, dim=1).indices
        put(sec.offset + 8, idx.to(torch.int32).to(torch.int16))
        put(sec.offset + 8 + rows * k * 2, size * torch.randn(rows, k, device="cuda", generator=g))

    if rank:
        put(hdr.section_s.offset, 1.0 / torch.arange(1, rank + 1, device="cuda", dtype=torch.float32))
        for sec, n in ((hdr.section_u, rows), (hdr.section_v, cols)):
            if case["uv"] == "none":
                fp32(sec, n * rank, n ** -0.5)
            else:
                quant(sec, case["uv"], n * rank, 3.0 * n ** -0.5)
    else:
        quant(hdr.section_direct, case["q"], rows * cols, 3.0)
    if hdr.flags & PKG.FLAG_OUTLIER:
        topk(hdr.section_outlier_topk, _topk(cols, case["outlier"]), 20.0 if not rank else 1.0)
    if hdr.flags & PKG.FLAG_ERROR:
        topk(hdr.section_error_topk, _topk(cols, case["error"]), 0.5 if not rank else 0.05)


def _topk(cols, ratio):
    k = int(np.floor(np.float32(cols) * np.float32(ratio) + np.float32(0.5)))
    return max(1, min(cols, k)) if ratio > 0 else 0


class _Batch:
    """A set of lanes, its inputs and the buffers that its objects and results go to."""

    def __init__(self, case, mats):
        self.lib, self.mats, count, n = PKG.lib(), mats, case["count"], case["rows"] * case["cols"]
        self.handle = self.lib.bsq_batch_create(*_settings(case), min(8, count))
        if not self.handle:
            raise RuntimeError("bsq_batch_create failed")
        self.capacity = int(self.lib.bsq_lane_packed_capacity(self.lib.bsq_batch_lane(self.handle, 0)))
        self.packed = [torch.empty(self.capacity, dtype=torch.uint8, device="cuda") for _ in mats]
        self.out = [torch.empty_like(m) for m in mats]
        pointers = ctypes.c_void_p * count
        self.in_ptrs = pointers(*[m.data_ptr() for m in mats])
        self.packed_ptrs = pointers(*[p.data_ptr() for p in self.packed])
        self.out_ptrs = pointers(*[o.data_ptr() for o in self.out])
        self.headers = (PKG.Array * count)()
        self.header_ptrs = pointers(*[ctypes.addressof(h) for h in self.headers])
        self.sizes = (ctypes.c_uint64 * count)()
        self.count, self.n = count, n

    def run(self):
        if self.lib.bsq_batch_compress(self.handle, self.in_ptrs, self.count, PKG.INPUT_DEVICE, self.packed_ptrs, self.capacity,
                                       None, self.headers, self.sizes) != 0:
            raise RuntimeError("bsq_batch_compress failed")
        if self.lib.bsq_batch_decompress(self.handle, self.header_ptrs, self.count, 1, self.out_ptrs, self.n) != 0:
            raise RuntimeError("bsq_batch_decompress failed")

    def __del__(self):
        if getattr(self, "handle", None):
            self.lib.bsq_batch_destroy(self.handle)


def _settings(case):
    return (case["rows"], case["cols"], case["outlier"], case["error"], case["rank"], case["niters"], FORMATS[case["uv"]],
            FORMATS[case["s"]], FORMATS[case["q"]])


def _compressor(case):
    rows, cols, outlier, error, rank, niters, uv, s, q = _settings(case)
    return TORCH_API.Compressor(rows, cols, outlier=outlier, error=error, rank=rank, niters=niters, uv=uv, s=s, q=q)


def prepare(case, seed):
    if case["kind"] == "batch":
        return dict(case=case, batch=_Batch(case, [_matrix(case, seed * 100 + i) for i in range(case["count"])]))
    if case["kind"] == "dropin":
        settings, lib = _settings(case), PKG.lib()
        eff = min(case["rank"], case["rows"], case["cols"]) if case["rank"] > 0 else case["rank"]
        if lib.bsq_compress_initialize(*settings, PKG.INPUT_HOST) or lib.bsq_decompress_initialize(*settings[:4], eff, *settings[6:]):
            raise RuntimeError("initialize failed")
        x = np.ascontiguousarray(_matrix(case, seed).cpu().numpy())
        return dict(case=case, x=x, out=torch.empty(case["rows"], case["cols"], device="cuda"))
    state = dict(case=case, comp=_compressor(case))
    x = _matrix(case, seed)
    if case["kind"] == "decode":
        state["packed"] = state["comp"].compress(x)
        _section_fill(case, state["packed"], seed)
    else:
        state["x"] = x
    return state


def _lowrank_outputs(header, data, matrix):
    """S, the outlier section's bytes (exact) and the matrix that came back."""
    at = 200 + header.section_s.offset
    out = {"s": data[at: at + header.section_s.size].clone().view(torch.float32), "matrix": matrix}
    if header.flags & PKG.FLAG_OUTLIER:
        at = 200 + header.section_outlier_topk.offset
        out["outliers"] = data[at: at + header.section_outlier_topk.size]
    return out


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "encode":
        packed = state["comp"].compress(state["x"])
        return packed.data[200: packed.nbytes]                # the payload; the header in front holds an address
    if kind == "decode":
        return state["comp"].decompress(state["packed"])
    if kind == "roundtrip":
        packed = state["comp"].compress(state["x"])
        return _lowrank_outputs(packed.header, packed.data, state["comp"].decompress(packed))
    if kind == "dropin":
        got = PKG.compress_to_bytes(state["x"].ctypes.data)
        if got is None or PKG.decompress_packed(got[1], state["out"].data_ptr(), state["x"].size) != 0:
            raise RuntimeError("compress or decompress failed")
        if case["rank"] > 0:
            return _lowrank_outputs(got[0], torch.from_numpy(got[1]), state["out"])
        return {"payload": got[1][200:], "matrix": state["out"]}
    b = state["batch"]
    b.run()
    return [_lowrank_outputs(b.headers[i], b.packed[i], b.out[i]) for i in range(b.count)]


# ---- what a pass cannot do without -----------------------------------------------------------------------------------
def _packed_bytes(case):
    rows, cols = case["rows"], case["cols"]

    def quant(fmt, n):
        return 4 * n if fmt == "none" else (n + 1) // 2 + (n + 63) // 64 * (4 if fmt == "nf4" else 1) + 48

    rank = min(case["rank"], rows, cols)
    b = quant(case["uv"], rows * rank) + quant(case["uv"], cols * rank) + 4 * rank if rank > 0 else quant(case["q"], rows * cols)
    return b + 6 * rows * (_topk(cols, case["outlier"]) + _topk(cols, case["error"]))


def work(case):
    rows, cols, kind = case["rows"], case["cols"], case["kind"]
    n, packed, rank = rows * cols, _packed_bytes(case), max(0, min(case["rank"], rows, cols))
    back = 2 * n * rank
    # range finder: W Omega, W^T Q and W Q per iteration, the projection; one orthonormalisation of each panel (its Gram
    # matrix and the product with the inverse factor); the two products that turn the core's factors into U and V
    small, big = min(rows, cols), max(rows, cols)
    it = case["niters"]
    forth = 2 * n * rank * (2 + 2 * it) + 4 * rank * rank * (big * (1 + it) + small * (1 + it)) + 2 * rank * rank * (rows + cols)
    if case["error"] > 0:
        forth += back
    if rank == 0:
        forth = back = 0
    if kind == "encode":
        return {"bytes": 4 * n + packed, "flops": forth}
    if kind == "decode":
        return {"bytes": 4 * n + packed, "flops": back}
    return {"bytes": case["count"] * (8 * n + 2 * packed), "flops": case["count"] * (forth + back)}


def tolerance(case):
    if case["rank"] < 1:
        return "exact"                                        # codes, scales, lists and their sums are defined bit for bit
    if case["kind"] == "decode":
        return {"rel": 2e-6}                                  # FP32 sums of `rank` products; 3e-8 to 3e-7 against 64 bits
    if case["uv"] == "none":
        # FP32 factors.  Another solver for the core: up to 8e-5 in S and 3e-5 in the matrix (the orthonormalisation's shift
        # of 1e-5 allows that much); products in another order or operand split: 5e-6
        return {"rel": 3e-4}
    # Quantised factors: NF4's levels are not symmetric, so a singular pair of the other sign, or rotated within a flat
    # spectrum, is coded differently.  Another solver or another operand split of the products: 0.04 to 0.08 of the matrix
    return {"rel": 0.3}


# ---- the same in 64 bits ---------------------------------------------------------------------------------------------
LEVELS = [-1.0, -0.6961928009986877, -0.5250730514526367, -0.39491748809814453, -0.28444138169288635, -0.18477343022823334,
          -0.09105003625154495, 0.0, 0.07958029955625534, 0.16093020141124725, 0.24611230194568634, 0.33791524171829224,
          0.44070982933044434, 0.5626170039176941, 0.7229568362236023, 1.0]


def _exact_decode(case, state):
    data, hdr, rows, cols = state["packed"].data, state["packed"].header, case["rows"], case["cols"]
    rank = hdr.effective_rank

    def raw(at, count, dtype):
        size = torch.empty((), dtype=dtype).element_size()
        return data[200 + at: 200 + at + count * size].clone().view(dtype)

    def quant(sec, fmt, n):
        nb, at = (n + 63) // 64, sec.offset + 48
        if fmt == "nf4":
            scales, at = raw(at, nb, torch.float32).double(), at + nb * 4
        else:
            dq = raw(sec.offset + 40, 1, torch.float32).double()
            scales, at = raw(at, nb, torch.float8_e4m3fn).double() * dq, at + nb
        codes = raw(at, (n + 1) // 2, torch.uint8).long()
        codes = torch.stack([codes >> 4, codes & 15], 1).reshape(-1)[:n]
        return torch.tensor(LEVELS, dtype=torch.float64, device="cuda")[codes] * scales.repeat_interleave(64)[:n]

    if rank:
        u, v = ((raw(sec.offset, n * rank, torch.float32).double() if case["uv"] == "none" else quant(sec, case["uv"], n * rank)).view(n, rank)
                for sec, n in ((hdr.section_u, rows), (hdr.section_v, cols)))
        y = (u * raw(hdr.section_s.offset, rank, torch.float32).double()) @ v.T
    else:
        y = quant(hdr.section_direct, case["q"], rows * cols).view(rows, cols)
    for flag, sec, ratio in ((PKG.FLAG_ERROR, hdr.section_error_topk, case["error"]), (PKG.FLAG_OUTLIER, hdr.section_outlier_topk, case["outlier"])):
        if hdr.flags & flag:
            k = _topk(cols, ratio)
            idx = raw(sec.offset + 8, rows * k, torch.int16).long().view(rows, k) & 0xFFFF
            y.scatter_add_(1, idx, raw(sec.offset + 8 + rows * k * 2, rows * k, torch.float32).double().view(rows, k))
    return y


def _omega(n, k):
    """The range finder's random matrix: block 1 of cuRAND's default sequence for seed 1234, n x k, column-major."""
    found = glob.glob(os.path.join(os.path.dirname(torch.__file__), "..", "nvidia", "curand", "lib", "libcurand.so.10"))
    rand = ctypes.CDLL(found[0] if found else ctypes.util.find_library("curand") or "libcurand.so.10")
    gen, count = ctypes.c_void_p(), n * k + (n * k & 1)
    out = torch.empty(count, device="cuda")
    torch.cuda.synchronize()
    rcs = [rand.curandCreateGenerator(ctypes.byref(gen), 100), rand.curandSetPseudoRandomGeneratorSeed(gen, ctypes.c_ulonglong(1234)),
           rand.curandSetGeneratorOffset(gen, ctypes.c_ulonglong(n * k)),
           rand.curandGenerateNormal(gen, ctypes.c_void_p(out.data_ptr()), ctypes.c_size_t(count), ctypes.c_float(0.0), ctypes.c_float(1.0))]
    torch.cuda.synchronize()
    rand.curandDestroyGenerator(gen)
    if any(rcs):
        raise RuntimeError("cuRAND failed")
    return out[: n * k].view(k, n).T.double()


def _exact_lowrank(case, x):
    rows, cols = case["rows"], case["cols"]
    a, out = x.double(), {}
    ko = _topk(cols, case["outlier"])
    if ko:
        order = x.abs().sort(dim=1, descending=True, stable=True).indices[:, :ko]       # equal magnitudes: lower column first
        vals = x.gather(1, order)
        a.scatter_(1, order, 0.0)
        head = np.array([rows, cols, ko, 0], np.uint16).view(np.uint8)
        out["outliers"] = torch.cat([torch.from_numpy(head).cuda(), order.to(torch.int32).to(torch.int16).view(torch.uint8).reshape(-1),
                                     vals.contiguous().view(torch.uint8).reshape(-1)])
    w = a if rows >= cols else a.T
    rank = min(case["rank"], rows, cols)
    q = torch.linalg.qr(w @ _omega(w.shape[1], rank))[0]
    for _ in range(case["niters"]):
        q = torch.linalg.qr(w @ torch.linalg.qr(w.T @ q)[0])[0]
    b = w.T @ q                                               # N x rank
    out["s"] = torch.linalg.svdvals(torch.linalg.qr(b, mode="r")[1])
    out["matrix"] = None                                      # quantised factors: depends on the signs of the singular vectors
    if case["uv"] == "none":
        y = q @ b.T
        y = y if rows >= cols else y.T.contiguous()
        if ko:
            y.scatter_add_(1, order, vals.double())
        out["matrix"] = y
    return out


def exact(case, seed):
    if case["kind"] == "decode":
        return _exact_decode(case, prepare(case, seed))
    if case["rank"] < 1:
        return None                                           # bytes, compared as they are
    if case["kind"] == "batch":
        return [_exact_lowrank(case, _matrix(case, seed * 100 + i)) for i in range(case["count"])]
    got = _exact_lowrank(case, _matrix(case, seed))
    return got
