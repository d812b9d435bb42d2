"""What the launchers do when the runtime refuses something, and which kernels they
choose, without a GPU: the library's object files linked against a stand-in for
the CUDA runtime (tests/fake_cudart.cpp) that records launches and copies.  No
kernel runs; what the kernels compute is tested on the GPU."""
import ctypes as C
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")
OBJECTS = ("sparse_kernels", "zfp_kernels", "cswap_abi", "sparse_static")


class Fake:
    def __init__(self, path):
        self.lib = C.CDLL(path)
        self.lib.fake_log.restype = C.c_char_p
        # stands for every device buffer: no kernel runs, so only the address is looked at
        self._mem = (C.c_char * (1 << 16))()
        self.buf = (C.addressof(self._mem) + 255) // 256 * 256

    def log(self):
        return self.lib.fake_log().decode().splitlines()

    def kernels(self):
        """Names of the kernels that were launched, in order."""
        names = ("sparse_small", "sparse_count", "block_exclusive_scan", "sparse_pack", "sparse_zero",
                 "sparse_onepass", "sparse_unpack", "zfp_encode_slab", "zfp_decode_slab", "zfp_encode_generic",
                 "zfp_decode_generic")
        return [next(n for n in names if n in line) for line in self.log() if line.startswith("launch")]

    def compress(self, n, onepass=False):
        fn = self.lib.csw_sparse_compress_onepass if onepass else self.lib.csw_sparse_compress
        p = C.c_void_p(self.buf)
        return fn(p, C.c_size_t(n), p, C.c_size_t(1 << 40), p, None)

    def zfp(self, dims, maxbits, decode=False):
        p, d = C.c_void_p(self.buf), [C.c_size_t(v) for v in dims]
        if decode:
            return self.lib.csw_zfp_decompress(p, C.c_size_t(1 << 40), *d, maxbits, p, None)
        return self.lib.csw_zfp_compress(p, *d, maxbits, p, C.c_size_t(1 << 40), None, None)


@pytest.fixture(scope="module")
def fake_path(tmp_path_factory):
    from cswap_b200 import build
    build.build()
    objs = [os.path.join(build.HERE, "build", o + ".o") for o in OBJECTS]
    if not all(os.path.exists(o) for o in objs):
        build.build(force=True)
    so = str(tmp_path_factory.mktemp("fake") / "libfake.so")
    subprocess.check_call(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-I", os.path.join(CUDA, "include"), "-o", so,
                           os.path.join(HERE, "fake_cudart.cpp")] + objs + ["-Wl,-Bsymbolic", "-Wl,-z,defs"])
    return so


@pytest.fixture(scope="module")
def fake_library(fake_path):
    return Fake(fake_path)


@pytest.fixture
def fake(fake_library):
    fake_library.lib.fake_reset()
    return fake_library


def test_a_refused_launch_leaves_no_error_behind(fake):
    """A call whose launch is refused says so itself; the runtime's last error, which the next caller of
    cudaGetLastError in the process would take for its own, is clear again."""
    calls = [lambda: fake.compress(1 << 20), lambda: fake.compress(1 << 20, onepass=True),
             lambda: fake.zfp((32, 32, 64), 512), lambda: fake.zfp((32, 32, 64), 512, decode=True),
             lambda: fake.zfp((33, 7, 0), 128), lambda: fake.zfp((33, 7, 0), 128, decode=True),
             lambda: fake.lib.csw_sparse_decompress(C.c_void_p(fake.buf), C.c_size_t(5000), C.c_void_p(fake.buf), None)]
    for call in calls:
        fake.lib.fake_reset()
        fake.lib.fake_fail_launches(100)
        assert call() == 3 and fake.lib.fake_pending_error() == 0
        assert fake.lib.csw_last_cuda_error() == 701  # cudaErrorLaunchOutOfResources
    for decode in (False, True):  # more shared memory than a kernel may use without opting in
        fake.lib.fake_reset()
        fake.lib.fake_fail_attributes(100)
        assert fake.zfp((32, 32, 64), 2048, decode) == 3 and fake.lib.fake_pending_error() == 0


@pytest.mark.parametrize("most", [0, 8])  # CTAs of the largest cluster that can be placed
@pytest.mark.parametrize("n", [0, 1, 4096, 9 * 4096, 16 * 4096, 100003, 64 * 4096])
def test_a_cluster_that_cannot_be_placed_is_replaced(fake, n, most):
    """Where a process has only part of a GPC a cluster launch is refused: the call then makes the ordinary
    launches, which need nothing of the sort, and succeeds."""
    tiles = -(-n // 4096)
    for onepass, ordinary in ((False, ["sparse_count", "block_exclusive_scan", "sparse_pack"]),
                              (True, ["sparse_zero", "sparse_onepass"])):
        if not tiles:  # nothing to count or pack, only the total to write
            ordinary = [k for k in ordinary if k in ("block_exclusive_scan", "sparse_zero")]
        fake.lib.fake_reset()
        fake.lib.fake_max_cluster(most)
        assert fake.compress(n, onepass) == 0
        assert fake.kernels() == (["sparse_small"] if max(tiles, 1) <= most else ordinary)
        assert fake.lib.fake_pending_error() == 0


def test_the_single_pass_compressor_leaves_its_cluster_at_512_kib(fake):
    """Above, the cluster's blocks want an SM each, and two launches are shorter; the ordered compressor, whose
    alternative is three dependent launches, keeps it up to 1 MiB."""
    for n in (1, 4096, 65536, 65537, 131072, 131073, 180000, 262144, 262145):
        for onepass, most, ordinary in ((False, 262144, ["sparse_count", "block_exclusive_scan", "sparse_pack"]),
                                        (True, 131072, ["sparse_zero", "sparse_onepass"])):
            fake.lib.fake_reset()
            assert fake.compress(n, onepass) == 0
            assert fake.kernels() == (["sparse_small"] if n <= most else ordinary)


@pytest.mark.parametrize("decode", [False, True])
@pytest.mark.parametrize("where", ["apart", "touching", "in place", "at the field's end", "at the stream's end"])
def test_host_calls_on_overlapping_buffers_are_not_cut(fake, decode, where):
    """Large host-to-host calls run in chunks whose results are written while later chunks are still to be read.
    Where the host's field and stream share memory everything is read first, as the reference reads it."""
    from cswap_b200._lib import Bitstream, ZfpField, ZfpStream
    nz, maxbits = 4096, 512
    field_bytes, stream_bytes = 4096 * nz, nz // 4 * 64 * maxbits // 8
    mem = (C.c_char * (2 * field_bytes))()
    field = C.addressof(mem) + stream_bytes
    begin = field + {"apart": field_bytes + 4096, "touching": field_bytes, "in place": 0,
                     "at the field's end": field_bytes - 8, "at the stream's end": 8 - stream_bytes}[where]
    bs = Bitstream(64, 0, begin, begin, begin + stream_bytes)
    zs, f = ZfpStream(maxbits, maxbits, 32, -1074, C.pointer(bs)), ZfpField(3, 32, 32, nz, 0, 0, 0, 0, 0, field)
    fake.lib.fake_host_pointers()
    fake.lib.cuda_compress.restype = C.c_size_t
    if decode:
        fake.lib.cuda_decompress(C.byref(zs), C.byref(f))
    else:
        assert fake.lib.cuda_compress(C.byref(zs), C.byref(f)) == stream_bytes
    read, written = (stream_bytes, field_bytes) if decode else (field_bytes, stream_bytes)
    copies = [line.split()[1:] for line in fake.log() if line.startswith("copy")]
    assert sum(int(n) for k, n in copies if k == "h2d") == read and sum(int(n) for k, n in copies if k == "d2h") == written
    assert (len(copies) == 2) == (where not in ("apart", "touching"))
    assert len(copies) != 2 or [k for k, _ in copies] == ["h2d", "d2h"]
    assert bs.bits == 64 and bs.ptr == begin + stream_bytes


@pytest.mark.parametrize("sms", [148, 74, 18])
def test_grids_follow_the_devices_own_sms(fake_path, tmp_path, sms):
    """Blocks are spread over warps until there is one for each scheduler of the device at hand, and 2-D decoders
    take several rounds from twice as many CTAs as it holds: a partition has fewer SMs than the whole chip."""
    import shutil
    so = str(tmp_path / "libfake.so")  # a library of its own: the count of a device is asked for once
    shutil.copy(fake_path, so)
    fake = Fake(so)
    fake.lib.fake_reset()
    fake.lib.fake_sms(sms)
    for dims in ((32, 32, 148), (31, 30, 148), (32, 32, 8192)):
        blocks = -(-dims[0] // 4) * -(-dims[1] // 4) * -(-dims[2] // 4)
        per_warp = next((1 << k for k in range(5) if blocks >> k <= 4 * sms), 32)
        for decode in (False, True):
            assert fake.zfp(dims, 512, decode) == 0
            assert int(fake.log()[-1].split("grid ")[1].split()[0]) == -(-blocks // (4 * per_warp))
    ctas = 768 * 4096 // 16 // 128
    rounds = 1 if ctas < 16 * sms else min(ctas // (8 * sms), 8)
    assert fake.zfp((768, 4096, 0), 128, decode=True) == 0
    assert int(fake.log()[-1].split("grid ")[1].split()[0]) == -(-ctas // rounds)
