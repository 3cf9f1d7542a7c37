"""FP64 products that the exact route hands over: the partial sums of the DMMA kernel are added in split order by the few
blocks of a gated launch, to the bits of the kernel called alone with a workspace for its partial sums."""
import numpy as np
import pytest

from oracle import psmma_oracle as O


# element counts around multiples of the gated launch's 152 x 256 threads x 4 elements, odd sizes, one column
@pytest.mark.gpu
@pytest.mark.parametrize("n,k", [(1, 256), (129, 300), (152, 256), (608, 256), (609, 257), (777, 777), (1031, 509)])
@pytest.mark.parametrize("beta", [0.0, -0.5])
def test_partial_sums_in_split_order(n, k, beta, cuda):
    import torch
    from psmma_git_gb300 import KIND_TOEPLITZ, fortran_empty, psmma_toeplitz, workspace_size
    A = O.cfg_matrix(n, k, seed=n)
    A[n // 2, k // 3] = 2.0 ** 120  # a row of more bits than the route takes
    dA, Q0 = fortran_empty(n, k, ld=n + 3), torch.from_numpy(O.cfg_matrix(n, k, seed=k)).to(cuda)
    dA.copy_(torch.from_numpy(A))
    g = torch.from_numpy(O.cfg_vector(2 * k - 1, seed=5)).to(cuda)
    need = workspace_size(KIND_TOEPLITZ, n, k)
    assert need >= 2 * 8 * n * k  # split K
    out = []
    for work in (None, torch.empty(need, dtype=torch.uint8, device=cuda)):
        Q = fortran_empty(n, k, ld=n + 1)
        Q.copy_(Q0)
        psmma_toeplitz(n, k, 1.0, dA, g, beta, Q, work=work)
        torch.cuda.synchronize()
        out.append(Q.cpu().numpy())
    np.testing.assert_array_equal(out[0], out[1])
