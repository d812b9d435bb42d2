"""Codec calls in the company of other work on their stream.  The kernels are
launched programmatically (they may start while the kernel in front still runs,
and two of the sparse ones read their input that early), so: a long kernel that
rewrites the tensor directly in front of a call, one that overwrites it directly
behind, and calls captured into a graph, where programmatic launches become a
different kind of edge."""
import numpy as np
import pytest

import util

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def cs():
    import torch
    import cswap_b200
    assert torch.cuda.is_available()
    cswap_b200.lib()
    return cswap_b200


# name -> (values, call); every call returns tensors that do not depend on the schedule
def _calls(cs):
    def trip(t, onepass):
        packed, nnz = cs.sparse_compress(t, onepass=onepass)
        return cs.sparse_decompress(packed, t.numel()), nnz

    def zfp(t, maxbits, dims=None):
        s = cs.zfp_compress(t, maxbits, dims)
        return s, cs.zfp_decompress(s, t.numel(), maxbits, dims)

    return {
        "ordered_cluster": (100003, lambda t: trip(t, False)), "ordered": (300001, lambda t: trip(t, False)),
        "ordered_16MiB": (1 << 22, lambda t: trip(t, False)),
        "onepass_cluster": (100003, lambda t: trip(t, True)), "onepass": (300001, lambda t: trip(t, True)),
        "onepass_16MiB": (1 << 22, lambda t: trip(t, True)),
        "zfp_64KiB": (1 << 14, lambda t: zfp(t, 512)), "zfp_8MiB": (1 << 21, lambda t: zfp(t, 1024)),
        "zfp_3d": (31 * 33 * 500, lambda t: zfp(t, 300, (31, 33, 500))),
        "zfp_2d": (770 * 1001, lambda t: zfp(t, 128, (770, 1001, 0))), "zfp_1d": (100003, lambda t: zfp(t, 37, (100003, 0, 0))),
    }


NAMES = list(_calls(None))


def _same(got, want):
    import torch
    return all(torch.equal(a if a.dtype != torch.float32 else a.view(torch.int32),
                           b if b.dtype != torch.float32 else b.view(torch.int32)) for a, b in zip(got, want))


@pytest.mark.parametrize("name", NAMES)
def test_between_kernels_that_rewrite_the_tensor(cs, name):
    """The tensor is the end of a 256 MiB buffer that one kernel fills from front to back right before the call
    and another overwrites right after it; the outputs are those of the call on its own."""
    import torch
    n, call = _calls(cs)[name]
    src = torch.relu(torch.randn(1 << 26, device="cuda", generator=torch.Generator(device="cuda").manual_seed(n)))
    start = ((1 << 26) - n) // 4 * 4  # on a 16-byte boundary, as allocations are
    want = call(src[start:start + n].clone())
    big = torch.empty_like(src)
    tensor = big[start:start + n]
    torch.cuda.synchronize()
    for stream in (torch.cuda.current_stream(), torch.cuda.Stream()):
        with torch.cuda.stream(stream):
            for _ in range(4):
                big.fill_(7.0)
                torch.mul(src, 1.0, out=big)
                got = call(tensor)
                big.fill_(-3.0)
                torch.cuda.synchronize()
                assert _same(got, want)


@pytest.mark.parametrize("name", NAMES)
def test_captured_into_a_graph(cs, name):
    """Producer, call and a kernel that overwrites the tensor, captured and replayed on other inputs."""
    import torch
    n, call = _calls(cs)[name]
    feed, tensor = torch.empty(n, device="cuda"), torch.empty(n, device="cuda")
    feed.copy_(torch.from_numpy(util.relu_normal(n, 0.5, seed=1)))
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        call(feed)  # as a program would: once before the capture
    torch.cuda.current_stream().wait_stream(side)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        torch.mul(feed, 1.0, out=tensor)
        got = call(tensor)
        tensor.fill_(-3.0)
    for seed in range(2, 6):
        feed.copy_(torch.from_numpy(util.relu_normal(n, 0.5 if seed % 2 else 0.9, seed=seed)))
        want = call(feed.clone())
        graph.replay()
        graph.replay()
        torch.cuda.synchronize()
        assert _same(got, want)
