"""The work that users of the framework have it do, as timed passes through its public entry points.

Kinds of pass ("op"):

  zfp_enc, zfp_dec   one direction of the fixed-rate ZFP codec on the swap path's view of a flat tensor
                     (32 x 32 x numel/1024): what a program does that codes activations on the device by itself.
  zfp_field          compress and decompress of a field in its own extents (1-D, 2-D or 3-D, edges that are not
                     multiples of four, any bit budget): feature maps, token matrices, flat vectors.
  sparse_enc         the ordered sparse compressor: the packed buffer is the same in every run.
  sparse_dec         its scatter-back.
  sparse_trip        the single-read compressor and the scatter-back (what the swap manager runs).
  swap               a training step's use of the swap manager: tensors go out one after the other, everything
                     lands on the host, then they come back in the opposite order.
  host_trip          cuda_compress and cuda_decompress, the reference's own calls, on pinned host buffers.

Sizes: the sweep from 64 KiB up at 4, 8 and 16 bits per value, the convolution activations of VGG16 at batch
128, the hidden and feed-forward activations of a BERT-base-shaped encoder at batch 32 x 512, 50 / 75 / 90 % zeros.
"""
import ctypes as C
import math

import torch

import cswap_b200 as cs
from cswap_b200 import _lib

MIB = 1 << 20
POLICIES = {"raw": cs.POLICY_RAW, "sparse": cs.POLICY_SPARSE, "zfp": cs.POLICY_ZFP}


def listed():
    return [
        # the smallest tensor of the sweep: a call is launch latency
        {"name": "zfp_enc_64KiB_r8", "op": "zfp_enc", "numel": 64 * 256, "maxbits": 512, "values": "normal"},
        # a late VGG16 activation, [128, 512, 2, 2], at the finest rate
        {"name": "zfp_dec_1MiB_r16", "op": "zfp_dec", "numel": MIB // 4, "maxbits": 1024, "values": "normal"},
        # the first VGG16 activations, [128, 64, 32, 32]
        {"name": "zfp_enc_32MiB_r8", "op": "zfp_enc", "numel": 32 * MIB // 4, "maxbits": 512, "values": "tanh"},
        # the feed-forward activation of the encoder, [32, 512, 3072]
        {"name": "zfp_enc_192MiB_r16", "op": "zfp_enc", "numel": 192 * MIB // 4, "maxbits": 1024, "values": "normal"},
        # the benchmark's tensor
        {"name": "zfp_dec_256MiB_r8", "op": "zfp_dec", "numel": 256 * MIB // 4, "maxbits": 512, "values": "tanh"},
        # feature maps with ragged edges, in their own extents
        {"name": "zfp_field_3d_ragged", "op": "zfp_field", "nx": 31, "ny": 33, "nz": 4096, "maxbits": 512,
         "values": "tanh"},
        # a token matrix, [4096, 768]
        {"name": "zfp_field_2d", "op": "zfp_field", "nx": 768, "ny": 4096, "nz": 0, "maxbits": 128,
         "values": "normal"},
        # [128, 128, 16, 16] behind a ReLU
        {"name": "sparse_enc_16MiB_50", "op": "sparse_enc", "numel": 16 * MIB // 4, "zeros": 0.5},
        # a small ragged activation
        {"name": "sparse_trip_ragged_90", "op": "sparse_trip", "numel": 100003, "zeros": 0.9},
        # a large one
        {"name": "sparse_dec_256MiB_75", "op": "sparse_dec", "numel": 256 * MIB // 4, "zeros": 0.75},
        # eight VGG16 activations of [128, 256, 8, 8] in a step
        {"name": "swap_8x8MiB_zfp", "op": "swap", "numel": 8 * MIB // 4, "count": 8, "policy": "zfp",
         "maxbits": 512},
        # the reference's own calls from host memory
        {"name": "host_trip_64MiB_r8", "op": "host_trip", "numel": 64 * MIB // 4, "maxbits": 512, "values": "tanh"},
    ]


def _log_between(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["zfp_enc", "zfp_dec", "zfp_enc", "zfp_dec", "zfp_field", "sparse_enc", "sparse_dec",
                     "sparse_trip", "swap", "host_trip"])
    if op in ("zfp_enc", "zfp_dec"):
        slabs = _log_between(rng, 16, 65536)  # 64 KiB ... 256 MiB, any number of slabs
        return {"op": op, "numel": 1024 * slabs, "maxbits": 64 * rng.choice([4, 8, 16]),
                "values": rng.choice(["tanh", "normal", "uniform"])}
    if op == "zfp_field":
        dims = rng.choice([1, 2, 3])
        numel = _log_between(rng, 1 << 16, 1 << 22)
        rate = rng.choice([8, 16])
        values = rng.choice(["tanh", "normal", "uniform"])
        if dims == 1:
            return {"op": op, "nx": numel, "ny": 0, "nz": 0, "maxbits": 4 * rate, "values": values}
        if dims == 2:
            nx = _log_between(rng, 32, 4096)
            return {"op": op, "nx": nx, "ny": max(1, numel // nx), "nz": 0, "maxbits": 16 * rate, "values": values}
        nx, ny = _log_between(rng, 5, 128), _log_between(rng, 5, 128)
        budget = 300 if rng.random() < 0.2 else 64 * rate  # now and then one that is not whole words
        return {"op": op, "nx": nx, "ny": ny, "nz": max(1, numel // (nx * ny)), "maxbits": budget, "values": values}
    if op in ("sparse_enc", "sparse_dec", "sparse_trip"):
        zeros = round(rng.uniform(0.3, 0.95), 2)
        # no more bytes than the largest listed case
        most = int((1 << 26) * 5.0 / (8.0 - 4.0 * zeros)) // (2 if op == "sparse_trip" else 1)
        return {"op": op, "numel": _log_between(rng, 1 << 14, min(most, 1 << 26)), "zeros": zeros}
    if op == "swap":
        policy = rng.choice(["raw", "sparse", "zfp"])
        numel = _log_between(rng, 1 << 12, 1 << (21 if policy == "zfp" else 20))
        return {"op": op, "numel": numel, "count": rng.randint(1, 8), "policy": policy,
                "maxbits": 64 * rng.choice([8, 16])}
    slabs = _log_between(rng, 1024, 16384)  # 4 ... 64 MiB
    return {"op": op, "numel": 1024 * slabs, "maxbits": 64 * rng.choice([4, 8]), "values": "tanh"}


def _values(kind, numel, gen):
    if kind == "uniform":
        return torch.rand(numel, generator=gen, device="cuda").mul_(2.0).sub_(1.0)
    t = torch.randn(numel, generator=gen, device="cuda")
    return t.tanh_() if kind == "tanh" else t


def _relu_values(numel, zeros, gen):
    """max(0, N(mu, 1)) with the requested share of zeros."""
    mu = -math.sqrt(2.0) * torch.erfinv(torch.tensor(2.0 * zeros - 1.0, dtype=torch.float64)).item()
    return torch.randn(numel, generator=gen, device="cuda").add_(mu).clamp_(min=0.0)


def _numel(case):
    if case["op"] == "zfp_field":
        return case["nx"] * max(case["ny"], 1) * max(case["nz"], 1)
    return case["numel"]


class _HostTrip:
    """A field in host memory and the stream objects the reference's calls take."""

    def __init__(self, field, maxbits):
        n = field.numel()
        nx, ny, nz = cs.zfp_view(n)
        need = cs.zfp_max_bytes(nx, ny, nz, maxbits)
        self.field, self.back = (torch.empty(n, dtype=torch.float32, pin_memory=True) for _ in range(2))
        self.stream = torch.empty(need, dtype=torch.uint8, pin_memory=True)
        self.field.copy_(field)
        p = self.stream.data_ptr()
        self.bits = _lib.Bitstream(64, 0, p, p, p + need)
        self.zfp = _lib.ZfpStream(1, maxbits, 64, -1074, C.pointer(self.bits), _lib._Exec(0, _lib._Omp(0, 0)))
        self.src = _lib.ZfpField(3, nx, ny, nz, 0, 0, 0, 0, 0, self.field.data_ptr())
        self.dst = _lib.ZfpField(3, nx, ny, nz, 0, 0, 0, 0, 0, self.back.data_ptr())


def prepare(case, seed):
    op = case["op"]
    gen = torch.Generator(device="cuda").manual_seed(seed)
    s = {"case": case}
    if op == "swap":
        # activations of a step: dense ones for ZFP and raw copies, half zeros for the sparse codec
        if case["policy"] == "sparse":
            s["tensors"] = [_relu_values(case["numel"], 0.5, gen) for _ in range(case["count"])]
        else:
            s["tensors"] = [_values("tanh", case["numel"], gen) for _ in range(case["count"])]
        room = case["count"] * (cs.sparse_layout(case["numel"]).bound + 4096) + (1 << 20)
        s["mgr"] = cs.SwapManager(pinned_bytes=room, staging_bytes=room, zfp_maxbits=case["maxbits"])
        return s
    n = _numel(case)
    if op.startswith("sparse"):
        t = _relu_values(n, case["zeros"], gen)
        if op == "sparse_enc":
            s["out"] = torch.zeros(cs.sparse_layout(n).bound, dtype=torch.uint8, device="cuda")
        if op == "sparse_dec":
            s["packed"], _ = cs.sparse_compress(t)
        else:
            s["t"] = t
        return s
    t = _values(case["values"], n, gen)
    if op == "zfp_dec":
        s["stream"] = cs.zfp_compress(t, case["maxbits"])
    elif op == "host_trip":
        s["host"] = _HostTrip(t, case["maxbits"])
    else:
        s["t"] = t
    return s


def run(s):
    case = s["case"]
    op = case["op"]
    if op == "zfp_enc":
        return cs.zfp_compress(s["t"], case["maxbits"])
    if op == "zfp_dec":
        return cs.zfp_decompress(s["stream"], case["numel"], case["maxbits"])
    if op == "zfp_field":
        dims = (case["nx"], case["ny"], case["nz"])
        stream = cs.zfp_compress(s["t"], case["maxbits"], dims)
        return stream, cs.zfp_decompress(stream, s["t"].numel(), case["maxbits"], dims)
    if op == "sparse_enc":
        return cs.sparse_compress(s["t"], out=s["out"])
    if op == "sparse_dec":
        return cs.sparse_decompress(s["packed"], case["numel"])
    if op == "sparse_trip":
        packed, nnz = cs.sparse_compress(s["t"], onepass=True)
        return cs.sparse_decompress(packed, case["numel"]), nnz
    if op == "swap":
        mgr, policy = s["mgr"], POLICIES[case["policy"]]
        tickets = [mgr.swap_out(t, policy) for t in s["tensors"]]
        mgr.sync()
        back = []
        for tk in reversed(tickets):
            back.append(mgr.swap_in(tk))
            tk.release()
        return back
    h = s["host"]
    n = cs.lib().cuda_compress(C.byref(h.zfp), C.byref(h.src))
    cs.lib().cuda_decompress(C.byref(h.zfp), C.byref(h.dst))
    return n, h.stream, h.back


def _stream_bytes(case):
    if case["op"] != "zfp_field":
        return _numel(case) // 64 * case["maxbits"] // 8
    blocks = 1
    for e in (case["nx"], case["ny"], case["nz"]):
        blocks *= max(1, -(-e // 4))
    return -(-blocks * case["maxbits"] // 64) * 8


def work(case):
    """Bytes read and written once: tensors, streams, packed buffers.  The codecs are integer work: no flops."""
    op, n = case["op"], _numel(case)
    if op in ("zfp_enc", "zfp_dec"):
        b = 4 * n + _stream_bytes(case)
    elif op in ("zfp_field", "host_trip"):
        b = 2 * (4 * n + _stream_bytes(case))
    elif op == "swap":
        payload = {"raw": 4 * n, "sparse": 2 * n + n // 8, "zfp": _stream_bytes(case)}[case["policy"]]
        b = case["count"] * 2 * (4 * n + payload)
    else:
        packed = n // 8 + n // 1024 + int(4 * n * (1.0 - case["zeros"]))
        b = (2 if op == "sparse_trip" else 1) * (4 * n + packed)
    return {"bytes": b, "flops": 0}


def tolerance(case):
    """Streams, packed buffers and rebuilt tensors are integer and byte work: the same bits."""
    return "exact"
