"""The decoders as a warp runs them: 32 lanes with 32 different blocks, which vote on what all of them do next.  The lanes
are run on the CPU, one after the other from vote to vote, so that a vote which some of them do not reach shows - on a GPU
they would wait for each other - and the values are compared with the oracle's, bit for bit."""
import ctypes as C

import numpy as np
import pytest

import util
from test_core_host import core  # noqa: F401

FLOATS, INTS, AGAIN, PARTED = range(4)


def decode(core, oracle, stream, dims, maxbits):  # noqa: F811
    """Decodes warp by warp, compares, and returns how many warps went which way."""
    s = np.ascontiguousarray(stream).view(np.uint64)
    ref = oracle.zfp_decode(s, *dims, maxbits)
    got = np.zeros(ref.size, dtype=np.float32)
    ways = (C.c_int * 4)()
    core.core_decode_warps(s.ctypes.data_as(C.c_void_p), *(C.c_size_t(d) for d in dims), maxbits,
                           got.ctypes.data_as(C.c_void_p), ways)
    assert ways[PARTED] == 0
    assert np.array_equal(got.view(np.uint32), ref.view(np.uint32))
    return list(ways)


def mixed_field(seed, warps=8):
    """32 x 32 view in which every warp (half a tile of four slabs) holds blocks that decode in different ways by
    themselves: noise, offset noise, smooth values, constants, zeros, values near the smallest and the largest."""
    rng = np.random.default_rng(seed)
    nz = 4 * ((warps + 1) // 2)
    a = util.normal(1024 * nz, seed).reshape(nz // 4, 4, 8, 4, 8, 4)  # tile, z, by, y, bx, x
    z, y, x = np.meshgrid(np.arange(4), np.arange(4), np.arange(4), indexing="ij")
    for t in range(nz // 4):
        for by in range(8):
            for bx in range(8):
                k = rng.integers(10)
                b = a[t, :, by, :, bx, :]
                smooth = np.sin(0.1 * (x + 0.7 * y + 0.5 * z) + rng.random())
                if k == 1:
                    b += np.float32(rng.choice([3, 10, 30, 100]))
                elif k == 2:
                    b[:] = smooth
                elif k == 3:
                    b[:] = smooth + rng.choice([.001, .01, .03, .1]) * b
                elif k == 4:
                    b[:] = rng.standard_normal()
                elif k == 5:
                    b[:] = 0
                elif k == 6:
                    b *= np.float32(1e-36)
                elif k == 7:
                    b *= np.float32(1e36)
                elif k == 8:
                    b[:] = np.where(rng.random((4, 4, 4)) < 0.5, -1, 1) * (1 - 2.0 ** -rng.integers(2, 24, (4, 4, 4)))
    return a.reshape(-1).astype(np.float32), (32, 32, nz)


@pytest.mark.parametrize("maxbits", [9, 64, 256, 512, 768, 832, 864, 1024, 1216, 1280, 1408, 1440, 2048, 777, 1025])
def test_warps_of_blocks_that_differ(core, oracle, maxbits):  # noqa: F811
    for seed in range(4):
        a, dims = mixed_field(seed)
        decode(core, oracle, oracle.zfp_encode(a, *dims, maxbits), dims, maxbits)
    for s in util.arbitrary_streams(oracle.zfp_stream_bytes(*dims, maxbits) // 4, maxbits):
        decode(core, oracle, s, dims, maxbits)


@pytest.mark.parametrize("maxbits", [9, 64, 128, 200, 256, 272, 384, 512])
def test_2d_warps_of_blocks_that_differ(core, oracle, maxbits):  # noqa: F811
    dims = (128, 62, 0)
    for seed in range(4):
        a = mixed_field(seed)[0][:dims[0] * dims[1]]
        decode(core, oracle, oracle.zfp_encode(a, *dims, maxbits), dims, maxbits)
    for s in util.arbitrary_streams(oracle.zfp_stream_bytes(*dims, maxbits) // 4, maxbits):
        decode(core, oracle, s, dims, maxbits)
