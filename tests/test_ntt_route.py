"""Toeplitz and Hankel multiplies of the split precision by number-theoretic transforms: the same
integer product as the modular GEMMs, so the same result bit for bit where that path scales every
column alike; generators the route leaves go to the single product."""
import numpy as np
import pytest

from oracle import psmma_oracle as O

PRIMES = [1073479681, 1072496641, 1071513601, 1070727169, 1068564481]


def test_primes_and_limb_crt():
    # transforms of 2^15 points need 2^15 | p - 1; the CRT's quotient estimate and its 32-bit limbs,
    # restated with the kernel's word sizes, recover any |Z| < 2^115 (four primes) or 2^126 (five)
    rng = np.random.default_rng(0)
    for np_, bits in ((4, 115), (5, 126)):
        ps = PRIMES[:np_]
        M = int(np.prod([1], dtype=object))
        for p in ps:
            assert p < 2 ** 30 and (p - 1) % 2 ** 15 == 0 and pow(2, p - 1, p) == 1
            M *= p
        for Z in [0, 1, -1, 2 ** bits - 1, 1 - 2 ** bits] + [int.from_bytes(rng.bytes(16), "little") % 2 ** (bits + 1)
                                                              - 2 ** bits for _ in range(300)]:
            X = [Z * pow(M // p, -1, p) % p for p in ps]
            q = (sum(x * ((1 << 52) // p) >> 32 for x, p in zip(X, ps)) + (1 << 19)) >> 20
            assert sum(x * (M // p) for x, p in zip(X, ps)) - q * M == Z
            for l in range(np_):
                assert sum(x * ((M // p >> (32 * l)) & 0xFFFFFFFF) for x, p in zip(X, ps)) < 2 ** 64


def _run(kind, n, k, alpha, A, g, beta, Q0, cuda, pad=0, **kw):
    import torch
    import psmma_git_gb300 as P
    col = lambda x: torch.from_numpy(np.ascontiguousarray(x.T)).to(cuda).t()  # noqa: E731
    dA, dQ = (P.fortran_empty(n, k, torch.float64, cuda, ld=n + pad) for _ in range(2))
    dA.copy_(col(A))
    dQ.copy_(col(Q0))
    getattr(P, "psmma_" + kind)(n, k, alpha, dA, torch.from_numpy(g).to(cuda), beta, dQ, precision="split", **kw)
    torch.cuda.synchronize()
    return dQ.cpu().numpy()


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["toeplitz", "hankel"])
@pytest.mark.parametrize("n,k,nmod,alpha,beta,pad", [(70, 4096, 0, 1.0, 0.0, 0), (1, 4096, 13, -0.5, 2.0, 3),
                                                     (65, 3500, 15, 1.0, 0.5, 1), (33, 4097, 14, 1.0, 0.0, 0),
                                                     (129, 8192, 8, 0.75, -1.5, 2), (31, 8193, 0, 1.0, 0.0, 1),
                                                     (17, 16384, 13, 1.0, 0.0, 0)])
def test_same_result_as_the_gemms(kind, n, k, nmod, alpha, beta, pad, cuda):
    # lengths 2^13 (k to 4096), 2^14, 2^15, filled and just begun; four and five primes; the single
    # product (block_levels = -1) gives the same bits on a generator whose columns share a binade
    A, Q0 = O.cfg_matrix(n, k, seed=n + k), O.cfg_matrix(n, k, seed=n)
    A[n // 2, : k // 3] = 0.0
    g = O.cfg_vector(2 * k - 1, seed=k)
    args = (kind, n, k, alpha, A, g, beta, Q0, cuda, pad)
    np.testing.assert_array_equal(_run(*args, n_moduli=nmod), _run(*args, n_moduli=nmod, block_levels=-1))


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["toeplitz", "hankel"])
@pytest.mark.parametrize("spread", [6, 40])
def test_graded_generators_keep_column_accuracy(kind, spread, cuda):
    # columns whose largest entries differ by 6 binades (within the primes' spare bits) and by 40 (the
    # single product): every column keeps the split path's relative accuracy
    n, k = 64, 4096
    A = O.cfg_matrix(n, k, seed=5)
    g = O.cfg_vector(2 * k - 1, seed=6) * 2.0 ** (-spread * np.arange(2 * k - 1) / (2 * k - 1) * 2)
    got = _run(kind, n, k, 1.0, A, g, 0.0, np.zeros((n, k)), cuda)
    assert O.col_max_rel(got, O.dense_product(kind, 1.0, A, g, 0.0, None, k)) < 1e-12


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["toeplitz", "hankel"])
def test_nonfinite_inputs(kind, cuda):
    # an Inf row of A: a NaN row; a NaN in the generator: the single product's NaN columns
    n, k = 40, 4096
    A, g = O.cfg_matrix(n, k, seed=7), O.cfg_vector(2 * k - 1, seed=8)
    A[3, 9], A[11] = np.inf, 0.0
    z = np.zeros((n, k))
    got, ref = (_run(kind, n, k, 1.0, A, g, 0.0, z, cuda, block_levels=lv) for lv in (0, -1))
    assert np.isnan(got[3]).all() and (got[11] == 0.0).all()
    np.testing.assert_array_equal(got, ref)
    g[100] = np.nan
    got, ref = (_run(kind, n, k, 1.0, A, g, 0.0, z, cuda, block_levels=lv) for lv in (0, -1))
    assert np.isnan(got[:, :k // 2]).any()
    np.testing.assert_array_equal(got, ref)


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["toeplitz", "hankel"])
def test_zero_generator_and_wide_scales(kind, cuda):
    n, k = 20, 4096
    A = O.cfg_matrix(n, k, seed=9) * 2.0 ** np.linspace(-300, 300, n).round()[:, None]
    z = np.zeros((n, k))
    assert (_run(kind, n, k, 1.0, A, np.zeros(2 * k - 1), 0.0, z, cuda) == 0.0).all()
    g = O.cfg_vector(2 * k - 1, seed=10) * 2.0 ** -200
    got, ref = (_run(kind, n, k, 1.0, A, g, 0.0, z, cuda, block_levels=lv) for lv in (0, -1))
    np.testing.assert_array_equal(got, ref)
