"""FP64 products of many rows with a small H: the DMMA kernel, whose few steps are faster there than the exact route's
passes over padded planes; with fewer rows or a larger H the exact route."""
import numpy as np
import pytest

from oracle import psmma_oracle as O


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["toeplitz", "cauchy"])
@pytest.mark.parametrize("n,k,kernel", [(5000, 8, False), (9000, 1, True), (50000, 5, True), (60000, 16, True), (10000, 32, False),
                                        (19456, 32, True), (30000, 32, False), (30000, 33, False)])
def test_route_of_tall_products(kind, n, k, kernel, cuda):
    import torch
    import psmma_git_gb300 as P
    A = O.cfg_matrix(n, k, seed=k)
    gen = O.cfg_cauchy_generators(k, seed=2) if kind == "cauchy" else O.cfg_vector(2 * k - 1, seed=2)
    dA, out = P.fortran_empty(n, k), []
    dA.copy_(torch.from_numpy(A))
    dg = P.fortran_empty(k, 4) if kind == "cauchy" else torch.empty(2 * k - 1, dtype=torch.float64, device=cuda)
    dg.copy_(torch.from_numpy(gen))
    for work in (None, torch.empty(256, dtype=torch.uint8, device=cuda)):  # with a workspace: the kernel
        Q = P.fortran_empty(n, k)
        getattr(P, "psmma_" + kind)(n, k, 1.0, dA, dg, 0.0, Q, work=work)
        out.append(Q.cpu().numpy())
    if kernel or k > 1:  # k = 1: one product, the same either way
        assert (out[0] == out[1]).all() == kernel
    H = O.dense_h(kind, gen, k)
    assert (np.abs(out[0] - A @ H) <= 2.0 ** -45 * (k + 2) * (np.abs(A) @ np.abs(H))).all()
