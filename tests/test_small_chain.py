"""Small products launch their kernels behind one another without waiting for each to drain: back-to-back calls on shared
operands, on several streams, and inside a graph give what single, synchronised calls give."""
import numpy as np
import pytest

from oracle import psmma_oracle as O

SIZES = [(1, 1), (33, 64), (250, 262), (251, 262), (700, 836), (700, 837), (2047, 2048)]


def _operands(n, k):
    import torch
    from psmma_git_gb300 import fortran_empty
    A = fortran_empty(n, k)
    A.copy_(torch.from_numpy(O.cfg_matrix(n, k, seed=n)))
    return A, torch.from_numpy(O.cfg_vector(2 * k - 1, seed=k)).cuda(), fortran_empty(n, k)


def _call(n, k, A, g, Q, prec, **kw):
    from psmma_git_gb300 import psmma_toeplitz
    psmma_toeplitz(n, k, 1.0, A, g, 0.0, Q, precision=prec, **kw)


@pytest.mark.gpu
@pytest.mark.parametrize("prec", ["fp64", "split"])
@pytest.mark.parametrize("n,k", SIZES)
def test_back_to_back_calls_chain(prec, n, k):
    # each call's result is the next one's A (n x k in, n x k out): a kernel that started before its predecessor
    # had finished would read the wrong one
    import torch
    A, g, Q = _operands(n, k)
    g /= 4.0 * k ** 0.5
    X, want = A.clone(memory_format=torch.preserve_format), []
    Y = torch.empty_like(Q)
    for _ in range(6):
        _call(n, k, X, g, Y, prec)
        torch.cuda.synchronize()
        want.append(Y.cpu().numpy().copy())
        X, Y = Y, X
    for _ in range(3):
        X, Y = A.clone(memory_format=torch.preserve_format), torch.empty_like(Q)
        torch.cuda.synchronize()
        got = []
        for _ in range(6):
            _call(n, k, X, g, Y, prec)
            got.append(Y.clone())
            X, Y = Y, X
        torch.cuda.synchronize()
        for a, b in zip(want, got):
            np.testing.assert_array_equal(a, b.cpu().numpy())


@pytest.mark.gpu
@pytest.mark.parametrize("prec", ["fp64", "split"])
def test_streams_and_graph(prec):
    import torch
    from psmma_git_gb300 import KIND_TOEPLITZ, workspace_size
    probs = [_operands(n, k) for n, k in SIZES]
    want = []
    for (n, k), (A, g, Q) in zip(SIZES, probs):
        _call(n, k, A, g, Q, prec)
        torch.cuda.synchronize()
        want.append(Q.cpu().numpy().copy())
        Q.zero_()
    streams = [torch.cuda.Stream() for _ in range(3)]
    torch.cuda.synchronize()
    for r in range(12):
        for p, ((n, k), (A, g, Q)) in enumerate(zip(SIZES, probs)):
            _call(n, k, A, g, Q, prec, stream=streams[p % 3])
    torch.cuda.synchronize()
    for w, (_, _, Q) in zip(want, probs):
        np.testing.assert_array_equal(w, Q.cpu().numpy())
    if prec == "split":  # the FP64 precision keeps its kernel in a graph; a stream whose status word exists
        n, k = SIZES[2]
        A, g, Q = probs[2]
        work = torch.empty(workspace_size(KIND_TOEPLITZ, n, k, precision=prec), dtype=torch.uint8, device="cuda")
        Q.zero_()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=streams[2]):
            _call(n, k, A, g, Q, prec, work=work, stream=streams[2])
        graph.replay()
        torch.cuda.synchronize()
        np.testing.assert_array_equal(want[2], Q.cpu().numpy())
