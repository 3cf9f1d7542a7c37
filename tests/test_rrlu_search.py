"""The RRLU's pivot searches order the quotients |u / (d - f)| by exponents and FP32 mantissas and divide only
the leading ones in FP64.  Where that order has to step aside -- equal quotients, weights over hundreds of
decades, zero rows, blocks of one to a few more than a warp's or a block's threads -- the merge level has to give the
exact product, and the oracle's ranks."""
import numpy as np
import pytest

from oracle import psmma_oracle as O

SIZES = [2, 3, 9, 64, 65, 130, 515, 2050]


def _generators(n, weights):
    g = O.cfg_cauchy_generators(n, seed=n)
    rng = np.random.default_rng(n)
    if weights == "ties":  # integer distances, two weights: equal quotients everywhere
        return np.stack([2.0 * np.arange(n), 2.0 * np.arange(n) + 1, np.ones(n), 1.0 + (np.arange(n) % 3 == 0)], 1)
    if weights == "wide":
        g[:, 2] *= 10.0 ** rng.uniform(-60, 60, n)
        g[:, 3] *= 10.0 ** rng.uniform(-60, 60, n)
    if weights == "zeros":
        g[rng.integers(0, n, n // 4), 2] = 0.0
        g[rng.integers(0, n, n // 4), 3] = 0.0
    return g


@pytest.mark.gpu
@pytest.mark.parametrize("weights", ["ties", "wide", "zeros"])
def test_rrlu_search_on_awkward_quotients(weights):
    import torch
    from psmma_git_gb300 import cauchy_batch_lowrank, fortran_empty
    probs, dev = [], []
    for n in SIZES:
        A, g = O.cfg_matrix(n, n, seed=n + 1), _generators(n, weights)
        Ad, Qd = fortran_empty(n, n), fortran_empty(n, n)
        Ad.copy_(torch.from_numpy(A))
        probs.append((A, g))
        dev.append((Ad, torch.from_numpy(g).cuda().t().contiguous().t(), Qd))
    ranks, _ = cauchy_batch_lowrank(dev, 1.0, 0.0, compressor="rrlu", tol=1e-14, precision="fp64")
    torch.cuda.synchronize()
    for i, ((A, g), (_, _, Qd)) in enumerate(zip(probs, dev)):
        n = A.shape[0]
        H = O.dense_h("cauchy", g, n)
        _, ro = O.merge_level_product(A, g, np.zeros((n, n)), 1.0, 0.0, "rrlu", 1e-14)
        for a, b in zip(ranks[2 * i:2 * i + 2], ro):
            assert abs(a - b) <= 1, (n, ranks[2 * i:2 * i + 2], ro)
        # 1e-14 of the largest pivot is left out of each block, and FP64 sums of n terms are in the rest
        assert np.linalg.norm(Qd.cpu().numpy() - A @ H) <= 1e-13 * np.linalg.norm(A) * np.linalg.norm(H), n
