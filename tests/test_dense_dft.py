"""DFT orders that no form of the fixed-point transform covers (n / R above 7200 and not a product of 2, 3 and 5 for every
R up to 16) keep the dense products: the plain 3M product (odd n), and the radix-2, 4 and 8 first step, on the split path
with the recombination of at most and of more than 96 bits, and on the FP64 tensor cores."""
import numpy as np
import pytest

from oracle import psmma_oracle as O


def _uncovered(n):
    def smooth(m):
        for f in (2, 3, 5):
            while m % f == 0:
                m //= f
        return m == 1
    return not any(n % R == 0 and (n // R <= 7200 or (n // R <= 14400 and smooth(n // R)))
                   for R in (1, 2, 3, 4, 5, 6, 8, 9, 10, 12, 15, 16))


@pytest.mark.gpu
@pytest.mark.parametrize("n,k,radix", [(7207, 5, 1), (9973, 2, 1), (14414, 3, 2), (28828, 2, 4), (57656, 1, 8),
                                       (57656, 5, 8)])
@pytest.mark.parametrize("prec,moduli,tol", [("split", 0, 1e-12), ("split", 16, 1e-12), ("fp64", 0, 1e-13)])
def test_orders_left_to_the_dense_products(n, k, radix, prec, moduli, tol, cuda):
    import torch
    import psmma_git_gb300 as P
    assert _uncovered(n) and P.load().psmma_split_dft_radix(n) == radix
    B, C0 = O.cfg_matrix(n, k, seed=n, complex_=True), O.cfg_matrix(n, k, seed=k, complex_=True)
    dB, dC = P.fortran_empty(n, k, torch.complex128, ld=n + 2), P.fortran_empty(n, k, torch.complex128, ld=n + 1)
    for alpha, beta in ((1.0, 0.0), (-0.75, 0.5)):
        dB.copy_(torch.from_numpy(B))
        dC.copy_(torch.from_numpy(C0 if beta else np.full((n, k), np.nan + 0j)))
        P.pzmdftl(n, k, alpha, dB, beta, dC, precision=prec, n_moduli=moduli)
        ref = alpha * np.fft.fft(B.astype(np.clongdouble), axis=0) + beta * C0
        err = np.sqrt((np.abs(dC.cpu().numpy() - ref) ** 2).sum(axis=0) / (np.abs(ref) ** 2).sum(axis=0))
        assert (err <= tol).all()


@pytest.mark.gpu
@pytest.mark.parametrize("prec", ["split", "fp64"])
@pytest.mark.parametrize("n", [7207, 14414])
def test_dense_columns_that_are_not_finite(n, prec, cuda):
    import torch
    import psmma_git_gb300 as P
    B = O.cfg_matrix(n, 3, seed=n, complex_=True)
    B.imag[n // 7, 1] = np.nan
    dB, dC = P.fortran_empty(n, 3, torch.complex128), P.fortran_empty(n, 3, torch.complex128)
    dB.copy_(torch.from_numpy(B))
    P.pzmdftl(n, 3, 1.0, dB, 0.0, dC, precision=prec)
    got = dC.cpu().numpy()
    assert np.isnan(got[:, 1].real).all() and np.isnan(got[:, 1].imag).all()
    assert O.rel_fro(got[:, [0, 2]], np.fft.fft(B[:, [0, 2]], axis=0)) < 1e-12


@pytest.mark.parametrize("n,prec", [(7207, "split"), (14414, "split"), (14414, "fp64")])
@pytest.mark.parametrize("off", [(8, 0), (0, 8)])
def test_bases_off_16_bytes_are_refused_before_any_launch(n, prec, off, lib):
    # the dense products' passes would fault on them; the addresses are never read
    import ctypes as C
    import psmma_git_gb300 as P
    opts = P.make_opts(prec)
    opts.work, opts.lwork = C.c_void_p(1 << 40), P.workspace_size(P.KIND_DFT, n, 2, prec)
    st = lib.pzmdftl(n, 2, 1.0, C.c_void_p((1 << 41) + off[0]), n, 0.0, C.c_void_p((1 << 42) + off[1]), n, C.byref(opts), None)
    assert st == -114
