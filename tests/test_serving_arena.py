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
