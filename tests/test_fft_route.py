"""The DFT multiply as a fixed-point fast Fourier transform: every output is the exact transform
to about 2^-57 of its column's norm, rounded to FP64 once, so that the relative error of a column
stays below 2^-53 (the rounding) times 1.25, for both precisions and all three forms of the
transform (direct, Bluestein's convolution, two levels), against an extended-precision FFT."""
import numpy as np
import pytest

from oracle import psmma_oracle as O

pytestmark = pytest.mark.gpu

BOUND = 1.25 * 2.0 ** -53


def _run(n, k, alpha, B, beta, C0, cuda, prec, pad=0, odd=False):
    """B and C as n x k blocks of larger arrays; odd: 8-byte aligned bases (not 16)."""
    import torch
    import psmma_git_gb300 as P

    def place(x):
        flat = torch.full((2 * (n + pad) * k + 1,), 7.0, dtype=torch.float64, device=cuda)
        base = flat[1:] if odd else flat[:-1]
        m = base.view(k, n + pad, 2)
        m[:, :n].copy_(torch.view_as_real(torch.from_numpy(np.ascontiguousarray(x.T))).to(cuda))
        return flat, m

    import ctypes as C
    _, b = place(B)
    _, c = place(C0)
    opts = P.make_opts(prec)
    st = P.load().pzmdftl(n, k, alpha, C.c_void_p(b.data_ptr()), n + pad, beta, C.c_void_p(c.data_ptr()), n + pad,
                          C.byref(opts), C.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert st == 0
    torch.cuda.synchronize()
    out = c.cpu().numpy()
    assert (out[:, n:] == 7.0).all()  # rows past n untouched
    return (out[:, :n, 0] + 1j * out[:, :n, 1]).T


def _ref(alpha, B, beta, C0):
    return alpha * np.fft.fft(B.astype(np.clongdouble), axis=0) + beta * C0.astype(np.clongdouble)


def _check(got, ref):
    err = np.sqrt((np.abs(got.astype(np.clongdouble) - ref) ** 2).sum(axis=0))
    assert (err <= BOUND * np.sqrt((np.abs(ref) ** 2).sum(axis=0))).all()


@pytest.mark.parametrize("prec", ["fp64", "split"])
@pytest.mark.parametrize("n,k", [(1, 2), (2, 3), (3, 1), (4, 2), (5, 2), (6, 2), (8, 2), (9, 2), (10, 2), (12, 2),
                                 (15, 2), (16, 5), (25, 3), (125, 2), (2187, 2), (3125, 2), (512, 40), (4800, 3),
                                 (8192, 3), (14336 // 7 * 6, 2), (13824, 2),         # direct
                                 (7, 3), (11, 2), (97, 5), (513, 4), (2046, 3), (4801, 2), (7151, 2),  # Bluestein
                                 (14400, 2), (16384, 2), (32768, 1), (8190, 2), (14337, 2), (7162, 2)])  # two levels
def test_columns_are_rounded_once(n, k, prec, cuda):
    B = O.cfg_matrix(n, k, seed=n + k, complex_=True)
    _check(_run(n, k, 1.0, B, 0.0, np.full((n, k), np.nan + 0j), cuda, prec, pad=n % 3, odd=bool(n & 1)),
           _ref(1.0, B, 0.0, np.zeros((n, k))))


@pytest.mark.parametrize("n", [300, 1021, 8190])
def test_alpha_beta_and_column_scales(n, cuda):
    # columns 2^600 apart, one of a single entry, one zero, one subnormal; alpha and beta add one
    # rounding each
    B = O.cfg_matrix(n, 6, seed=n, complex_=True)
    B[:, 1] *= 2.0 ** 600
    B[:, 2] *= 2.0 ** -600
    B[:, 3] = 0.0
    B[n // 3, 3] = 1.0 - 2.0j
    B[:, 4] = 0.0
    z = np.zeros((n, 6), complex)
    _check(_run(n, 6, 1.0, B, 0.0, z, cuda, "fp64"), _ref(1.0, B, 0.0, z))
    C0 = O.cfg_matrix(n, 6, seed=n + 1, complex_=True)
    got, ref = _run(n, 6, 0.75, B, -0.5, C0, cuda, "fp64"), _ref(0.75, B, -0.5, C0)
    size = np.sqrt((np.abs(0.75 * _ref(1.0, B, 0.0, z)) ** 2).sum(axis=0)) + np.linalg.norm(C0, axis=0)
    assert (np.sqrt((np.abs(got - ref) ** 2).sum(axis=0)) <= 3 * BOUND * size).all()
    B[:, 5] *= 2.0 ** -1050
    got, ref = _run(n, 6, 1.0, B, 0.0, z, cuda, "fp64")[:, 5], _ref(1.0, B, 0.0, z)[:, 5]
    assert (np.abs(got - ref) <= 2.0 ** -1074 + BOUND * np.abs(ref)).all()


@pytest.mark.parametrize("n", [64, 97, 14400])
def test_nonfinite_columns(n, cuda):
    # split: NaN throughout the column; FP64: the infinities and NaN of the FP64 sums
    B = O.cfg_matrix(n, 3, seed=n, complex_=True)
    B[n // 5, 1] = np.inf
    z = np.zeros((n, 3), complex)
    for prec in ("split", "fp64"):
        got = _run(n, 3, 1.0, B, 0.0, z, cuda, prec)
        assert not np.isfinite(got[:, 1]).any()
        assert prec == "fp64" or np.isnan(got[:, 1]).all()
        _check(got[:, [0, 2]], _ref(1.0, B[:, [0, 2]], 0.0, z[:, [0, 2]]))
