"""Requests at the limits of a server's memory budget, and FP64 requests of every kind alone and in the mix."""
import numpy as np
import pytest

from oracle import psmma_oracle as O

pytestmark = pytest.mark.gpu


def test_fp64_dft_in_an_arena_of_the_dense_size(cuda):
    # the dense product needs 16 n bytes, the transform of a prime order some six times that
    import torch
    import psmma_git_gb300 as P
    from psmma_git_gb300.server import Server
    n, k = 997, 3
    B = O.cfg_matrix(n, k, seed=2, complex_=True)
    dB = P.fortran_empty(n, k, torch.complex128)
    dB.copy_(torch.from_numpy(B))
    for budget in (20480, 1 << 20):
        dC = P.fortran_empty(n, k, torch.complex128)
        with Server(budget, max_inflight=2) as srv:
            assert srv.wait(srv.submit("dft", n, k, 1.0, dB, None, 0.0, dC, precision="fp64"))["status"] == 0
        assert O.rel_fro(dC.cpu().numpy(), O.dft_product(1.0, B, 0.0, None)) < 1e-13


def test_request_of_the_whole_budget_runs(cuda):
    # the workspace is no whole number of the arena's pages
    import torch
    import psmma_git_gb300 as P
    from psmma_git_gb300.server import Server
    n, k = 70, 60
    need = P.workspace_size(P.KIND_HANKEL, n, k, "split")
    assert need % 4096
    A, g = O.cfg_matrix(n, k, seed=1), O.cfg_vector(2 * k - 1, seed=2)
    dA, dQ, dg = P.fortran_empty(n, k), P.fortran_empty(n, k), torch.from_numpy(g).to(cuda)
    dA.copy_(torch.from_numpy(A))
    with Server(need, max_inflight=2) as srv:
        for t in [srv.submit("hankel", n, k, 1.0, dA, dg, 0.0, dQ) for _ in range(3)]:
            assert srv.wait(t, timeout_s=10.0)["status"] == 0
    assert O.rel_fro(dQ.cpu().numpy(), O.dense_product("hankel", 1.0, A, g, 0.0, None, k)) < 1e-12
