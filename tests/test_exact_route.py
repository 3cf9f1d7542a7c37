"""The FP64 precision's exact modular route: every entry is the exact product of the stored
operands rounded once, and operands it does not take give the DMMA kernel's result bit for bit.

A caller workspace too small for the route keeps the DMMA kernel alone, which is what the
route is compared with where it must hand the product over."""
import math
from fractions import Fraction

import numpy as np
import pytest

from oracle import psmma_oracle as O

MODULI = [256, 255, 253, 251, 247, 241, 239, 233, 229, 227, 223, 211, 199, 197, 193, 191,
          217, 181, 179, 173, 167, 163, 157, 151, 149, 139, 137, 131, 127, 113, 109, 107]


def _parts(G):
    sizes = [3, 3, 2] if G == 2 else [3] * ((4 * G - 4 * (4 * G % 3)) // 3) + [4] * (4 * G % 3)
    first = [sum(sizes[:i]) for i in range(len(sizes))]
    return [MODULI[f:f + n] for f, n in zip(first, sizes)]


@pytest.mark.parametrize("G", range(2, 9))
def test_grouped_crt_recovers_the_integer(G):
    # the kernel's 32-bit part step, quotient estimates and sums of 32-bit limbs restated in Python
    # integers with its word sizes, at both ends of the range and at random Z, from any
    # representatives of the residues in [-128, 127]
    M, shift = math.prod(MODULI[:4 * G]), 47 if G == 2 else 52
    assert all(math.gcd(a, b) == 1 for i, a in enumerate(MODULI) for b in MODULI[:i])
    assert sum(map(len, _parts(G))) == 4 * G and M < 1 << (32 * G)
    rng = np.random.default_rng(G)
    top = int(0.497 * M)
    cases = [0, 1, -1, top, -top, M // 3] + [int.from_bytes(rng.bytes(32), "little") % (2 * top) - top
                                             for _ in range(200)]
    for Z in cases:
        acc, qs = [0] * G, 1 << (shift - 33)
        for ms in _parts(G):
            P = math.prod(ms)
            W = M // P
            c = [(P // m) * (pow(W % m, -1, m) * pow(P // m % m, -1, m) % m) for m in ms]
            b = -sum(128 * x for x in c) % P
            u = []
            for m in ms:
                r = Z % m
                r = r - m if r > 127 or (r - m >= -128 and rng.random() < 0.5) else r
                assert -128 <= r <= 127
                u.append(r + 128)
            t = (b + sum(x * y for x, y in zip(u, c))) % (1 << 32)
            est = (b << 20) // P + sum(x * ((y << 20) // P) for x, y in zip(u, c))
            assert est < 1 << 32 and (1 << shift) // P < 1 << 32
            X = (t - (est >> 20) * P) % (1 << 32)
            assert X < 1.002 * P and (X - b - sum(x * y for x, y in zip(u, c))) % P == 0
            qs += (X * ((1 << shift) // P)) >> 32
            for s in range(G):
                acc[s] += X * ((W >> (32 * s)) & 0xFFFFFFFF)
            assert G < 7 or W < 1 << (32 * (G - 1))
        assert max(acc[:G - 1]) < 1 << 63
        q, carry, out = qs >> (shift - 32), 0, 0
        for s in range(G):
            v = acc[s] + q * ((((1 << 256) - M) >> (32 * s)) & 0xFFFFFFFF) + carry
            assert s == G - 1 or v < 1 << 64
            out |= (v & 0xFFFFFFFF) << (32 * s)
            carry = v >> 32
        assert out - ((1 << (32 * G)) if out >> (32 * G - 1) else 0) == Z


def test_residue_chunks_stay_exact_in_fp32():
    # sum_t g_t c_t of eight 14-bit chunks is below 2^24, where FP32 integers are exact
    for m in MODULI:
        g = [pow(2, 14 * t, m) for t in range(8)]
        g = [x - m if x > m // 2 else x for x in g]
        assert sum(abs(x) for x in g) * (2 ** 14 - 1) < 2 ** 24


def _col(x, cuda):
    import torch
    return torch.from_numpy(np.ascontiguousarray(np.asarray(x).T)).to(cuda).t()


def _call(kind, n, k, A, gen, cuda, alpha=1.0, beta=0.0, Q0=None, pad=0, dmma=False):
    import torch
    import psmma_git_gb300 as P
    dA = P.fortran_empty(n, k, torch.float64, cuda, ld=n + pad)
    dA.copy_(_col(A, cuda))
    dQ = P.fortran_empty(n, k, torch.float64, cuda, ld=n + pad)
    dQ.copy_(_col(np.full((n, k), np.nan) if Q0 is None else Q0, cuda))
    work = torch.empty(256, dtype=torch.uint8, device=cuda) if dmma else None
    if kind == "eig":
        P.psmma_cauchyeig(n, k, alpha, dA, *[torch.from_numpy(x).to(cuda) for x in gen], beta, dQ, work=work)
    else:
        dg = _col(gen, cuda) if kind == "cauchy" else torch.from_numpy(gen).to(cuda)
        getattr(P, "psmma_" + kind)(n, k, alpha, dA, dg, beta, dQ, work=work)
    torch.cuda.synchronize()
    return dQ.cpu().numpy()


def _data(name, n, k, rng):
    A = rng.standard_normal((n, k)) if name != "uniform" else rng.uniform(-1, 1, (n, k))
    if name == "wide":
        A *= 2.0 ** rng.integers(-15, 16, (n, k))
    if name == "zeros":
        A[rng.random((n, k)) < 0.6] = 0.0
        A[n // 2] = 0.0
    if name == "tiny":
        A *= 2.0 ** -900
    if name == "rows":
        A *= 2.0 ** rng.integers(-300, 301, (n, 1))
    return A


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["toeplitz", "hankel"])
@pytest.mark.parametrize("n,k", [(1, 1), (3, 63), (33, 64), (128, 65), (257, 300), (65, 1100), (520, 129)])
@pytest.mark.parametrize("data", ["uniform", "wide", "zeros", "tiny", "rows"])
def test_products_are_rounded_once(kind, n, k, data, cuda):
    rng = np.random.default_rng(n * 31 + k)
    A = _data(data, n, k, rng)
    g = rng.uniform(-1, 1, 2 * k - 1)
    got = _call(kind, n, k, A, g, cuda, pad=n % 3)
    for _ in range(12):
        i, j = int(rng.integers(n)), int(rng.integers(k))
        h = g[np.arange(k) + j] if kind == "hankel" else g[(k - 1) + j - np.arange(k)]
        s = sum((Fraction(float(a)) * Fraction(float(b)) for a, b in zip(A[i], h)), Fraction(0))
        assert got[i, j] == float(s)


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["cauchy", "eig"])
@pytest.mark.parametrize("n,k,alpha,beta", [(1, 1, 1.0, 0.0), (100, 65, -0.75, 0.5), (300, 520, 2.0, -1.0)])
def test_generated_kinds_match_the_kernel(kind, n, k, alpha, beta, cuda):
    # the entries are those of the DMMA kernel, whose k FP64 additions then differ from the one
    # rounding by at most k half units of the sum of |a||h| (and alpha, beta once more)
    rng = np.random.default_rng(k)
    A, Q0 = _data("normal", n, k, rng), rng.uniform(-1, 1, (n, k))
    gen = O.cfg_cauchy_generators(k, seed=3) if kind == "cauchy" else \
        [np.ascontiguousarray(x) for x in O.eig_generators(k, seed=4)]
    H = O.dense_h("cauchy", gen, k) if kind == "cauchy" else O.cauchy_like_eig(*gen)
    got = _call(kind, n, k, A, gen, cuda, alpha, beta, Q0, pad=2)
    ref = _call(kind, n, k, A, gen, cuda, alpha, beta, Q0, pad=2, dmma=True)
    bound = 2.0 ** -52 * (abs(alpha) * (k + 2) * (np.abs(A) @ np.abs(H)) * (1 + 1e-9) + 2 * abs(beta) * np.abs(Q0))
    assert (np.abs(got - ref) <= bound).all()


@pytest.mark.gpu
@pytest.mark.parametrize("what", ["inf_a", "nan_gen", "wide_row", "wide_gen"])
def test_operands_left_to_the_kernel(what, cuda):
    # a non-finite entry, a row of A and a generator spanning more bits than the route takes: the
    # DMMA kernel's result bit for bit (its NaN and Inf pattern among it)
    n, k = 150, 200  # below the kernel's split-K sizes, whose partial sums need a workspace
    rng = np.random.default_rng(7)
    A, g = rng.standard_normal((n, k)), rng.uniform(-1, 1, 2 * k - 1)
    if what == "inf_a":
        A[5, 7] = np.inf
    if what == "nan_gen":
        g[100] = np.nan
    if what == "wide_row":
        A[3, 4] = 2.0 ** 90
    if what == "wide_gen":
        g[11] = 2.0 ** -80
        g[300] = 2.0 ** 60
    for beta in (0.0, 0.5):
        Q0 = rng.uniform(-1, 1, (n, k))
        np.testing.assert_array_equal(_call("toeplitz", n, k, A, g, cuda, 1.5, beta, Q0),
                                      _call("toeplitz", n, k, A, g, cuda, 1.5, beta, Q0, dmma=True))


@pytest.mark.gpu
def test_capture_keeps_the_kernel(cuda):
    # a captured call takes the DMMA kernel (a graph must not keep the route's workspace)
    import torch
    import psmma_git_gb300 as P
    n = k = 96
    rng = np.random.default_rng(1)
    A, g = rng.standard_normal((n, k)), rng.uniform(-1, 1, 2 * k - 1)
    dA, dg, dQ = _col(A, cuda), torch.from_numpy(g).to(cuda), P.fortran_empty(n, k, torch.float64, cuda)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        P.psmma_toeplitz(n, k, 1.0, dA, dg, 0.0, dQ)
    P.load().psmma_release_workspace()
    graph.replay()
    torch.cuda.synchronize()
    np.testing.assert_array_equal(dQ.cpu().numpy(), _call("toeplitz", n, k, A, g, cuda, dmma=True))
