"""qs_invert_batched_noalloc keeps no scratch: calls on different matrices may overlap on two streams, and a
call of a size that has run before can be captured into a graph. Equal bits to the call on its own."""
import ctypes

import numpy as np
import pytest

import quichotte_b200 as qb

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def matrices(N, batch, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    A = torch.randn(batch, N, N, dtype=torch.complex128, device="cuda", generator=g)
    return A + 3 * np.sqrt(N) * torch.eye(N, device="cuda")


def invert(A, info, stream):
    rc = qb._lib.qs_invert_batched_noalloc(A.shape[1], A.shape[0], ctypes.c_void_p(A.data_ptr()), ctypes.c_void_p(info.data_ptr()),
                                           ctypes.c_void_p(stream.cuda_stream))
    assert rc == 0


@pytest.mark.parametrize("N, batch", [(24, 400), (120, 40), (120, 300), (192, 300), (260, 20)])
def test_overlapping_calls_and_capture(N, batch):
    A = [matrices(N, batch, s) for s in (1, 2)]
    info = [torch.full((batch,), -1, dtype=torch.int32, device="cuda") for _ in A]
    alone = [a.clone() for a in A]
    for a, i in zip(alone, info):
        invert(a, i, torch.cuda.current_stream())
    torch.cuda.synchronize()
    both = [a.clone() for a in A]
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    torch.cuda.synchronize()
    for _ in range(3):
        for a, b, i, s in zip(A, both, info, streams):
            with torch.cuda.stream(s):
                b.copy_(a)
            invert(b, i, s)
    torch.cuda.synchronize()
    captured = A[0].clone()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        invert(captured, info[0], torch.cuda.current_stream())
    graph.replay()
    torch.cuda.synchronize()
    bits = lambda t: torch.view_as_real(t)
    assert all(torch.equal(bits(a), bits(b)) for a, b in zip(alone, both))
    assert torch.equal(bits(alone[0]), bits(captured)) and not info[0].any() and not info[1].any()
