"""The 2-D and 3-D decoders have a floating point path, a mixed one (3-D) and an integer one, and take a block's
planes in chunks of sixteen and eight: budgets on either side of where the kernels change, block exponents on either side of what the
floating point path takes, values that reach a block's full range, plane counts on either side of
what 24 bits hold, and bits that no encoder wrote.  All against the oracle, bit for bit."""
import numpy as np
import pytest

import util
from test_core_host import _check_decode, _run, core  # noqa: F401

BUDGETS = [256, 512, 800, 832, 864, 960, 1024, 1408, 1440]


def _inputs(n, seed):
    rng = np.random.default_rng(seed)
    t = util.tanh_normal(n, seed)
    full = np.where(rng.random(n) < 0.5, -1, 1) * (1 - 2.0 ** -rng.integers(2, 24, n))  # next to the top of the range
    yield full.astype(np.float32)
    yield util.normal(n, seed)
    yield (np.sin(0.01 * np.arange(n)) + 1e-4 * t).astype(np.float32)
    yield np.where(rng.random(n) < 0.02, t, 0).astype(np.float32)
    yield util.block_zoo(n, seed)
    for k in (-127, -100, -94, -93, -92, -88, -87, -86, 97, 98, 99, 127):  # taken: exponents from -93 (2-D: -87) to 98
        yield np.ldexp(t, k).astype(np.float32)


def _streams(words, seed):
    yield from util.arbitrary_streams(words, seed)
    rng = np.random.default_rng(seed)
    s = rng.integers(0, 2**32, words, dtype=np.uint64).astype(np.uint32)
    s[0::2] = (s[0::2] & 0xFFFFFE00) | ((int(rng.integers(34, 226)) << 1) | 1)  # exponents the path takes
    yield s
    s = s.copy()
    s[1::2] = 0xFFFFFFFF
    yield s


@pytest.mark.parametrize("dims,maxbits", [((32, 32, 8), b) for b in BUDGETS + [777, 833, 1025, 1409]] +
                         [((128, 64, 0), b) for b in (64, 128, 200, 256, 272, 384, 512)])
def test_core(core, oracle, dims, maxbits):  # noqa: F811
    for a in _inputs(8192, maxbits):
        _run(core, oracle, a, dims, maxbits)
    for s in _streams(oracle.zfp_stream_bytes(*dims, maxbits) // 4, maxbits):
        _check_decode(core, oracle, np.ascontiguousarray(s).view(np.uint64), dims, maxbits)


@pytest.mark.gpu
@pytest.mark.parametrize("dims,maxbits", [(d, b) for d in ((32, 32, 24), (31, 30, 9)) for b in BUDGETS + [777, 1025, 1409]] +
                         [((131, 63, 0), b) for b in (64, 128, 200, 256, 272, 384, 512)])
def test_kernels(oracle, dims, maxbits):
    import torch
    import cswap_b200 as cs
    n = dims[0] * dims[1] * max(dims[2], 1)
    streams = [oracle.zfp_encode(a[:n], *dims, maxbits) for a in _inputs((n + 63) // 64 * 64, maxbits)]
    streams += [np.ascontiguousarray(s).view(np.uint64)
                for s in _streams(oracle.zfp_stream_bytes(*dims, maxbits) // 4, maxbits)]
    for s in streams:
        got = cs.zfp_decompress(torch.from_numpy(s.view(np.uint8).copy()).cuda(), n, maxbits, dims).cpu().numpy()
        ref = oracle.zfp_decode(s, *dims, maxbits)
        assert np.array_equal(got.view(np.uint32), ref.view(np.uint32))
