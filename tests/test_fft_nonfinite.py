"""DFT columns that are not finite: the FP64 precision gives the classes (infinities, NaN) of the FP64 sums over the
column, in time that depends on the infinities alone."""
import numpy as np
import pytest

from oracle import psmma_oracle as O


def _classes(B):
    """Of each output's parts, by the FP64 sums' rules: 1 +inf, 2 -inf, 3 NaN (an infinity times a zero cosine or sine,
    infinities of both signs, a NaN); every output of a column that is not finite is one of them."""
    n, k = B.shape
    out = np.zeros((2, n, k), np.uint8)
    bit = np.array([2, 3, 1], np.uint8)  # sign -1, 0, 1
    for c in range(k):
        j = np.arange(n, dtype=np.int64)  # outputs that further terms can change
        for l in np.nonzero(~(np.isfinite(B.real[:, c]) & np.isfinite(B.imag[:, c])))[0]:
            t = j * int(l) % n
            cs = np.where((4 * t < n) | (4 * t > 3 * n), 1, np.where((4 * t > n) & (4 * t < 3 * n), -1, 0))
            sn = np.where((t == 0) | (2 * t == n), 0, np.where(2 * t < n, 1, -1))
            for v, re, im in ((B[l, c].real, cs, -sn), (B[l, c].imag, sn, cs)):
                if np.isnan(v):
                    out[:, :, c] = 3
                elif np.isinf(v):
                    out[0, j, c] |= bit[1 + int(np.sign(v)) * re]
                    out[1, j, c] |= bit[1 + int(np.sign(v)) * im]
            j = j[(out[:, j, c] != 3).any(axis=0)]
    return out


# direct, from registers, Bluestein, two levels (whose 14337 = 3 * 4779 and 32768 read the column in one part, 65280 =
# 16 * 4080 in five)
@pytest.mark.gpu
@pytest.mark.parametrize("n,k", [(12, 8), (360, 8), (1024, 8), (997, 8), (4800, 64), (14337, 8), (32768, 8), (65280, 8)])
def test_infinities_in_every_column(n, k, cuda):
    import torch
    import psmma_git_gb300 as P
    rng = np.random.default_rng(n)
    B = O.cfg_matrix(n, k, seed=n, complex_=True)
    for c in range(k):
        l = int(rng.integers(n))
        if c % 8 == 0:
            B.real[l, c] = np.inf
        elif c % 8 == 1:
            B.imag[l, c] = -np.inf
        elif c % 8 == 2:
            B[0, c] = complex(np.inf, -np.inf)
        elif c % 8 == 3:
            B.real[[0, n // 3, n // 2], c] = -np.inf
        elif c % 8 == 4:
            B.imag[l, c] = np.nan
            B.real[0, c] = np.inf
        elif c % 8 == 5:
            B.imag[:, c] = np.inf
        elif c % 8 == 6:
            B.real[-1, c] = -np.inf
            B.imag[-1, c] = np.inf
        else:
            B.real[rng.integers(n, size=5), c] = np.inf
    dB, dC = P.fortran_empty(n, k, torch.complex128), P.fortran_empty(n, k, torch.complex128)
    dB.copy_(torch.from_numpy(B))
    dC.fill_(1.0 + 1.0j)
    P.pzmdftl(n, k, 1.0, dB, 0.0, torch.empty_like(dC))
    a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    torch.cuda.synchronize()
    a.record()
    P.pzmdftl(n, k, -2.0, dB, 0.5, dC)
    b.record()
    torch.cuda.synchronize()
    got = dC.cpu().numpy()
    re, im = _classes(B)
    value = np.array([0.5, -np.inf, np.inf, np.nan])  # times alpha < 0
    np.testing.assert_array_equal(got.real, value[re])
    np.testing.assert_array_equal(got.imag, value[im])
    assert a.elapsed_time(b) < 20.0  # n^2 sums a column took 265 ms at n = 4800
