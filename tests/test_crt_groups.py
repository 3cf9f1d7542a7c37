"""The split recombination in groups of two to four moduli (crt_row4): the kernel's arithmetic in Python integers for
every number of moduli, and products of integer operands on the GPU, which have to be exact."""
import numpy as np
import pytest

MODULI = [256, 255, 253, 251, 247, 241, 239, 233, 229, 227, 223, 211, 199, 197, 193, 191]
U32, U64 = (1 << 32) - 1, (1 << 64) - 1


def _recombine(z, nmod):
    ms = MODULI[:nmod]
    M = int(np.prod([int(m) for m in ms], dtype=object))
    limbs = lambda v: [(v >> (32 * t)) & U32 for t in range(4)]
    groups, first = (nmod + 1) // 3, 0
    acc, qs = [0] * 4, 1 << 14
    for g in range(groups):
        size = 4 if g == 0 and nmod % 3 == 1 else min(3, nmod - first)
        mg = ms[first:first + size]
        first += size
        P = int(np.prod([int(m) for m in mg], dtype=object))
        W = M // P
        assert P <= U32 and (1 << 47) // P <= U32
        t = f = bias = 0
        for m in mg:
            c = (P // m) * (pow(W, -1, m) * pow(P // m, -1, m) % m)
            r = z % m
            r = r - m if r > m // 2 or r > 127 else r  # the int8 planes
            u = r + 128
            assert 0 <= u <= 255
            t, f = t + u * c, f + u * ((c << 20) // P)
            bias += 128 * c
        b = -bias % P
        t, f = t + b, f + (b << 20) // P
        assert f <= U32
        X = (t - (f >> 20) * P) & U32
        assert X < 1.002 * P and (X - t) % P == 0
        qs += X * ((1 << 47) // P) >> 32
        acc = [a + X * w for a, w in zip(acc, limbs(W))]
    assert first == nmod
    q, carry, out = qs >> 15, 0, 0
    for s, ml in enumerate(limbs((1 << 128) - M)):
        v = acc[s] + q * ml + carry
        assert s == 3 or v <= U64
        out |= (v & U32) << (32 * s)
        carry = v >> 32
    return out - (1 << 128) if out >> 127 else out


@pytest.mark.parametrize("nmod", range(8, 17))
def test_grouped_recombination_is_exact(nmod):
    rng = np.random.default_rng(nmod)
    M = int(np.prod([int(m) for m in MODULI[:nmod]], dtype=object))
    top = 497 * M // 1000  # the operands' bits keep |Z| below
    zs = [0, 1, -1, 127, -128, top, -top, top - 1]
    zs += [int(rng.integers(-1 << 62, 1 << 62)) * (top >> 62) + int(rng.integers(0, 1 << 30)) for _ in range(200)]
    zs += [int(rng.integers(-1 << 40, 1 << 40)) for _ in range(50)]
    for z in zs:
        z = max(-top, min(top, z))
        assert _recombine(z, nmod) == z


@pytest.mark.gpu
@pytest.mark.parametrize("nmod", range(8, 17))
@pytest.mark.parametrize("n,k", [(7, 5), (130, 200)])
def test_integer_products_are_exact(nmod, n, k):
    import torch
    from psmma_git_gb300 import fortran_empty, psmma_toeplitz
    bits = 9 + (nmod - 8)  # both operands fit the digits that nmod moduli leave them
    rng = np.random.default_rng(100 * nmod + n)
    A = rng.integers(-(1 << bits), 1 << bits, (n, k)).astype(np.float64)
    G = rng.integers(-(1 << bits), 1 << bits, 2 * k - 1).astype(np.float64)
    Ad, Qd = fortran_empty(n, k), fortran_empty(n, k)
    Ad.copy_(torch.from_numpy(A))
    psmma_toeplitz(n, k, 1.0, Ad, torch.from_numpy(G).cuda(), 0.0, Qd, precision="split", n_moduli=nmod)
    torch.cuda.synchronize()
    from oracle import psmma_oracle as O
    exact = A.astype(object).dot(O.dense_h("toeplitz", G, k).astype(object)).astype(np.float64)
    assert np.array_equal(Qd.cpu().numpy(), exact)
