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


def values_between_noise_and_smooth(n, seed):
    g = util.normal(n, seed)
    i = np.arange(n)
    smooth = 1.7 * np.sin(0.11 * (i % 32) + 0.07 * (i // 32 % 32) + 0.05 * (i // 1024) + 0.3)
    yield from ((f"normal+{k}", g + k) for k in (0, 3, 10, 30, 100))
    yield from ((f"smooth+{k}", smooth + k * g) for k in (0, 0.001, 0.01, 0.03, 0.1))
    yield from ((f"tanh*{k}", np.tanh(k * g)) for k in (1, 2, 3))
    yield "signs", 0.9999 * np.sign(g)
    yield "channels", (g.reshape(-1, 1024) + 4 * util.normal(n // 1024, seed + 1)[:, None]).reshape(-1)
    yield "relu", np.maximum(g - 1.28, 0)
    yield "constant in parts", np.maximum(0.05 * g + 0.5 + smooth, 0)


@pytest.mark.parametrize("maxbits", [64, 192, 256, 300, 512, 704, 832, 864, 1024, 1152, 1216, 1280, 1408, 2048])
def test_no_block_is_decoded_twice(core, oracle, maxbits):  # noqa: F811
    """Which decoder a warp's blocks get is told from their group tests: none of these values are tried by the floating point
    decoder and then decoded again, but for a few warps whose results come close to 2^31."""
    dims = (32, 32, 32)
    for name, a in values_between_noise_and_smooth(32 * 1024, maxbits):
        ways = decode(core, oracle, oracle.zfp_encode(np.ascontiguousarray(a, dtype=np.float32), *dims, maxbits), dims, maxbits)
        assert ways[AGAIN] <= sum(ways) // 8, (name, ways)


def test_each_way_is_taken(core, oracle):  # noqa: F811
    """Blocks whose planes and leading empty planes leave 24 bits enough go by floating point, what they do not
    fit and the smooth ones by integers; bits that no encoder wrote give results beyond 2^31, and are decoded twice."""
    dims = (32, 32, 32)
    values = {name: np.ascontiguousarray(a, dtype=np.float32) for name, a in values_between_noise_and_smooth(32 * 1024, 1)}
    way = {}
    for name, maxbits in (("normal+0", 512), ("normal+30", 512), ("smooth+0.03", 256), ("constant in parts", 512),
                          ("smooth+0", 512), ("normal+100", 832), ("normal+0", 1024), ("normal+0", 192)):
        way[name, maxbits] = decode(core, oracle, oracle.zfp_encode(values[name], *dims, maxbits), dims, maxbits)
    for key in (("normal+0", 512), ("normal+30", 512), ("smooth+0.03", 256), ("constant in parts", 512)):
        assert way[key][INTS] == way[key][AGAIN] == 0, (key, way)
    for key in (("smooth+0", 512), ("normal+100", 832), ("normal+0", 1024), ("normal+0", 192)):
        assert way[key][FLOATS] == way[key][AGAIN] == 0, (key, way)
    bits, more = (util.arbitrary_streams(oracle.zfp_stream_bytes(*dims, 288) // 4, seed)[0] for seed in (1, 10))
    bits |= more  # three ones in four
    bits[0::9] = (bits[0::9] & ~np.uint32(0x1FF)) | np.uint32((130 << 1) | 1)
    assert decode(core, oracle, bits, dims, 288)[AGAIN] > 0


@pytest.mark.gpu
@pytest.mark.parametrize("maxbits", [32, 64, 224, 255, 256, 288, 704, 832, 833, 864, 1024, 1440, 2048, 4096])
def test_kernels_on_warps_that_differ(oracle, maxbits):
    """Budgets on either side of where the kernel changes, warps that go different ways, in the swap path's view and with
    ragged edges."""
    import torch
    import cswap_b200 as cs
    for dims in ((32, 32, 32), (31, 30, 17)):
        n = dims[0] * dims[1] * dims[2]
        fields = [a for _, a in values_between_noise_and_smooth(32 * 1024, maxbits)] + [mixed_field(s, 16)[0] for s in range(2)]
        streams = [oracle.zfp_encode(np.ascontiguousarray(a[:n], dtype=np.float32), *dims, maxbits) for a in fields]
        streams += [np.ascontiguousarray(s).view(np.uint64)
                    for s in util.arbitrary_streams(oracle.zfp_stream_bytes(*dims, maxbits) // 4, maxbits)]
        for s in streams:
            got = cs.zfp_decompress(torch.from_numpy(s.view(np.uint8).copy()).cuda(), n, maxbits, dims).cpu().numpy()
            assert np.array_equal(got.view(np.uint32), oracle.zfp_decode(s, *dims, maxbits).view(np.uint32))
