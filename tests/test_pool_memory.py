"""The FP64 multiplies' planes: a buffer of their own in the stream's pools, which no other call's memory and no capture
is disturbed by, and without which the multiply still runs."""
import numpy as np
import pytest

from oracle import psmma_oracle as O

pytestmark = pytest.mark.gpu


def _operands(n, k, seed=1):
    import torch
    from psmma_git_gb300 import fortran_empty
    A = fortran_empty(n, k)
    A.copy_(torch.from_numpy(O.cfg_matrix(n, k, seed=seed)))
    return A, torch.from_numpy(O.cfg_vector(2 * k - 1, seed=seed + 1)).cuda(), fortran_empty(n, k)


def _toeplitz(n, k, A, g, Q, prec, stream, **kw):
    from psmma_git_gb300 import psmma_toeplitz
    psmma_toeplitz(n, k, 1.0, A, g, 0.0, Q, precision=prec, stream=stream, **kw)
    stream.synchronize()
    return Q.cpu().numpy().copy()


def test_captured_split_call_outlives_fp64_growth(cuda):
    # a captured split call keeps the address of the stream's pool: an FP64 call needing more must leave that buffer
    import torch
    from psmma_git_gb300 import psmma_toeplitz
    stream = torch.cuda.Stream()
    A, g, Q = _operands(500, 600)
    torch.cuda.synchronize()
    want = _toeplitz(500, 600, A, g, Q, "split", stream)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        psmma_toeplitz(500, 600, 1.0, A, g, 0.0, Q, precision="split", stream=stream)
    _toeplitz(1500, 1600, *_operands(1500, 1600), "fp64", stream)
    other = torch.full((64 << 20,), 0xA5, dtype=torch.uint8, device=cuda)  # would reuse memory that was freed
    Q.zero_()
    torch.cuda.synchronize()
    graph.replay()
    torch.cuda.synchronize()
    np.testing.assert_array_equal(want, Q.cpu().numpy())
    assert int(other.min()) == int(other.max()) == 0xA5


def test_fp64_call_beside_a_capture(cuda):
    # its first call allocates on a stream that is not captured; K below the kernel's split-K sizes
    import torch
    from psmma_git_gb300 import load, psmma_toeplitz
    n, k = 300, 200
    A, g, Q = _operands(n, k)
    side, stream = torch.cuda.Stream(), torch.cuda.Stream()
    x = torch.zeros(8, device=cuda)
    want = _toeplitz(n, k, A, g, Q, "fp64", stream)
    load().psmma_release_workspace()
    Q.zero_()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=side):
        x += 1.0
        psmma_toeplitz(n, k, 1.0, A, g, 0.0, Q, stream=stream)
    graph.replay()
    torch.cuda.synchronize()
    np.testing.assert_array_equal(want, Q.cpu().numpy())
    assert x.cpu().numpy().tolist() == [1.0] * 8


def test_planes_yield_to_other_calls(cuda):
    import torch
    from psmma_git_gb300 import KIND_TOEPLITZ, load, workspace_size
    n = 2048  # planes 0.7 GB, split workspace 0.3 GB
    lib = load()
    streams = [torch.cuda.Stream() for _ in range(4)]
    A, g, Q = _operands(n, n)
    torch.cuda.synchronize()
    exact = _toeplitz(n, n, A, g, Q, "fp64", streams[0])
    parts = max(256, workspace_size(KIND_TOEPLITZ, n, n))  # the kernel's partial sums
    kernel = _toeplitz(n, n, A, g, Q, "fp64", streams[0], work=torch.empty(parts, dtype=torch.uint8, device=cuda))
    split = _toeplitz(n, n, A, g, Q, "split", streams[0])
    assert (exact != kernel).any()
    lib.psmma_release_workspace()

    def leave(gib):
        torch.cuda.empty_cache()
        return torch.empty(torch.cuda.mem_get_info()[0] - int(gib * 2 ** 30), dtype=torch.uint8, device=cuda)

    most = leave(4.0)
    try:
        for s in streams[:2]:
            np.testing.assert_array_equal(_toeplitz(n, n, A, g, Q, "fp64", s), exact)
        rest = leave(1.0)  # the planes would take more than half of it: the kernel, and no buffer
        left = torch.cuda.mem_get_info()[0]
        np.testing.assert_array_equal(_toeplitz(n, n, A, g, Q, "fp64", streams[2]), kernel)
        assert torch.cuda.mem_get_info()[0] >= left - parts - (8 << 20)
        np.testing.assert_array_equal(_toeplitz(n, n, A, g, Q, "fp64", streams[1]), exact)  # the buffer it has
        del rest
        rest = leave(0.1)  # less than a split call needs: the planes of the other streams go
        np.testing.assert_array_equal(_toeplitz(n, n, A, g, Q, "split", streams[3]), split)
        del rest
    finally:
        del most
        torch.cuda.empty_cache()
    left = torch.cuda.mem_get_info()[0]
    np.testing.assert_array_equal(_toeplitz(n, n, A, g, Q, "fp64", streams[2]), exact)
    assert torch.cuda.mem_get_info()[0] < left - (512 << 20)
    assert lib.psmma_stream_release(streams[2].cuda_stream) == 0
    assert torch.cuda.mem_get_info()[0] > left - (64 << 20)
