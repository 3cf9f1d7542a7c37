"""Performance cases of the structured multiply: what a program that uses this library runs.

A case is a dict of plain values.  ``op`` is the entry point ("cauchy", "toeplitz", "hankel",
"dft", "eig", "merge_cauchy", "merge_toeplitz"), ``prec`` the precision option, ``n`` x ``k``
the operand, ``host`` whether the operands are (pinned) host arrays as the Fortran callers
have them.  Operands are column-major with an optional padded leading dimension (``pad``).
"""
import math

import numpy as np
import torch

import psmma_git_gb300 as P

DEV = "cuda:0"


def _case(name, op, prec, n, k, alpha=1.0, beta=0.0, **more):
    c = {"op": op, "prec": prec, "n": n, "k": k, "alpha": alpha, "beta": beta, "moduli": 0, "pad": 0,
         "data": "uniform", "clustered": 0.0, "host": False, "count": 0, "compressor": ""}
    c.update(more)
    return {"name": name, **c} if name else c


def listed():
    return [
        # one small multiply through the default (FP64) path: a leaf of the divide-and-conquer
        # tree, where the call's latency counts
        _case("cauchy_fp64_256", "cauchy", "fp64", 256, 256),
        # the FP64 Cauchy multiply of one mid-size merge
        _case("cauchy_fp64_2048", "cauchy", "fp64", 2048, 2048),
        # the Toeplitz test program's size, FP64
        _case("toeplitz_fp64_1024", "toeplitz", "fp64", 1024, 1024, data="unit"),
        # the DFT test program's size, FP64
        _case("dft_fp64_4800", "dft", "fp64", 4800, 4800),
        # the headline: the split Cauchy multiply at the largest size, clustered poles
        _case("cauchy_split_16384", "cauchy", "split", 16384, 16384, moduli=13, data="normal", clustered=0.1),
        # the eigensolver's multiply on an odd, rectangular, padded operand, accumulating into Q
        _case("eig_split_1000x777", "eig", "split", 1000, 777, alpha=-0.75, beta=0.5, pad=3, data="normal"),
        # the Toeplitz and DFT multiplies of the benchmark
        _case("toeplitz_split_8192", "toeplitz", "split", 8192, 8192, moduli=13),
        _case("dft_split_8192", "dft", "split", 8192, 8192, moduli=13),
        # a tall Hankel multiply of odd sizes with the default options
        _case("hankel_split_5000x3003", "hankel", "split", 5000, 3003, beta=0.25, pad=5),
        # a merge level of the divide-and-conquer tree with compressed off-diagonal blocks,
        # by column-pivoted QR and by the structured LU
        _case("merge_rrqr_16", "merge_cauchy", "split", 2900, 0, count=16, compressor="rrqr", moduli=13),
        _case("merge_rrlu_32", "merge_cauchy", "split", 4096, 0, count=32, compressor="rrlu", moduli=13),
        # host arrays in and out, as the Fortran callers have them
        _case("cauchy_host_split_4096", "cauchy", "split", 4096, 4096, data="normal", host=True),
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    prec = rng.choice(["fp64", "split", "split"])
    what = rng.choice(["product"] * 6 + ["merge", "host"])
    alpha = rng.choice([1.0, 1.0, -0.75, 2.5])
    beta = rng.choice([0.0, 0.0, 0.5])
    data = rng.choice(["uniform", "normal", "unit"])
    moduli = rng.choice([0, 13, 14])
    if what == "merge":
        op = rng.choice(["merge_cauchy", "merge_cauchy", "merge_toeplitz"])
        comp = "rrqr" if op == "merge_toeplitz" else rng.choice(["rrqr", "rrlu"])
        return _case("", op, "split", _logint(rng, 300, 2900), 0, alpha, beta, count=rng.randint(3, 16),
                     compressor=comp, moduli=moduli, data=data)
    op = rng.choice(["cauchy", "toeplitz", "hankel", "dft", "eig"])
    hi = {"host": 4096, "product": 14000}[what] if prec == "split" else (2900 if op == "dft" else 4000)
    n = _logint(rng, 128, hi)
    # mostly square, as the eigensolver's; else tall (or, for the DFT, fewer columns)
    k = n if rng.random() < 0.6 else max(64, int(n * rng.uniform(0.25, 1.0)))
    return _case("", op, prec, n, k, alpha, beta, moduli=moduli, data=data, pad=rng.choice([0, 0, 1, 7]),
                 clustered=rng.choice([0.0, 0.1]) if op == "cauchy" else 0.0, host=what == "host")


# ---- inputs --------------------------------------------------------------------------------
def _rng(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(1000003 * seed + 17)
    return g


def _values(g, data, *shape):
    if data == "normal":
        return torch.randn(*shape, dtype=torch.float64, device=DEV, generator=g)
    x = torch.rand(*shape, dtype=torch.float64, device=DEV, generator=g)
    return x if data == "unit" else 2.0 * x - 1.0


def _matrix(g, data, n, k, pad, cplx=False):
    """Column-major n x k with leading dimension n + pad."""
    if cplx:
        base = torch.complex(_values(g, data, k, n + pad), _values(g, data, k, n + pad))
    else:
        base = _values(g, data, k, n + pad)
    return base.t()[:n, :]


def _poles(g, k, clustered):
    d = torch.sort(torch.rand(k, dtype=torch.float64, device=DEV, generator=g)).values
    if clustered > 0.0 and k > 2:
        m = max(1, int(round(clustered * k)))
        idx = 1 + torch.randperm(k - 1, device=DEV, generator=g)[:m]
        gap = 1e-10 * (0.5 + 0.5 * torch.rand(k, dtype=torch.float64, device=DEV, generator=g))
        hit = torch.zeros(k, dtype=torch.bool, device=DEV)
        hit[idx] = True
        # a clustered pole sits one small gap above its left neighbour
        step = torch.where(hit, gap, torch.diff(d, prepend=torch.zeros(1, dtype=torch.float64, device=DEV)) + 1e-12)
        d = torch.cumsum(step, 0)
    return d


def _generator(g, op, k, clustered):
    if op in ("toeplitz", "hankel"):
        return _values(g, "uniform", 2 * k - 1)
    if op == "cauchy":
        d = _poles(g, k, clustered)
        gap = torch.cat([torch.diff(d), torch.ones(1, dtype=torch.float64, device=DEV)])
        w = d + (0.05 + 0.9 * torch.rand(k, dtype=torch.float64, device=DEV, generator=g)) * gap
        return torch.stack([d, w, _values(g, "normal", k), _values(g, "normal", k)]).t()
    f = _poles(g, k, 0.0)
    gap = torch.cat([torch.diff(f), torch.ones(1, dtype=torch.float64, device=DEV)])
    dl = (0.05 + 0.9 * torch.rand(k, dtype=torch.float64, device=DEV, generator=g)) * gap
    dr = dl - gap
    return [f, _values(g, "normal", k), _values(g, "normal", k), dl, dr]


def _sizes(case):
    """The sizes of a merge level: spread over their logarithm from n / 10 to n."""
    c = case["count"]
    return [max(16, int(round(case["n"] * 10.0 ** (-(c - 1 - i) / max(1, c - 1))))) - i % 3 for i in range(c)]


def _pinned(x):
    """A column-major numpy array on pinned host memory."""
    t = torch.empty(tuple(reversed(x.shape)), dtype=x.dtype, pin_memory=True)
    t.copy_(x.t())
    return t, t.numpy().T


def prepare(case, seed):
    g = _rng(seed)
    op, n, k, pad = case["op"], case["n"], case["k"], case["pad"]
    s = {"case": case, "keep": []}
    if op.startswith("merge"):
        kind = op.split("_")[1]
        s["problems"] = []
        for m in _sizes(case):
            if kind == "toeplitz":  # smooth off the diagonal: blocks of low rank
                x = torch.arange(-(m - 1), m, dtype=torch.float64, device=DEV)
                gen = _values(g, "unit", 1) / (x + 0.5 + 0.1 * _values(g, "uniform", 1))
            else:
                gen = _generator(g, "cauchy", m, 0.0)
            s["problems"].append((_matrix(g, case["data"], m, m, 0), gen, _matrix(g, "uniform", m, m, 0)))
        return s
    cplx = op == "dft"
    s["A"] = _matrix(g, case["data"], n, k, pad, cplx)
    s["gen"] = None if cplx else _generator(g, op, k, case["clustered"])
    s["Q"] = _matrix(g, "uniform", n, k, pad, cplx)
    if case["host"]:
        for key in ("A", "gen", "Q"):
            if isinstance(s[key], list):
                s[key] = [x.cpu().numpy() for x in s[key]]
            elif s[key] is not None and s[key].dim() == 1:
                s[key] = s[key].cpu().numpy()
            elif s[key] is not None:
                t, s[key] = _pinned(s[key])
                s["keep"].append(t)
    return s


def run(s):
    c = s["case"]
    op, n, k = c["op"], c["n"], c["k"]
    kw = {"precision": c["prec"], "n_moduli": c["moduli"]}
    if op == "merge_toeplitz":
        ranks, _ = P.toeplitz_batch_lowrank(s["problems"], c["alpha"], c["beta"], **kw)
        return [[q for _, _, q in s["problems"]], np.asarray(ranks)]
    if op == "merge_cauchy":
        ranks, _ = P.cauchy_batch_lowrank(s["problems"], c["alpha"], c["beta"], compressor=c["compressor"], **kw)
        return [[q for _, _, q in s["problems"]], np.asarray(ranks)]
    if op == "dft":
        return P.pzmdftl(n, k, c["alpha"], s["A"], c["beta"], s["Q"], **kw)
    if op == "eig":
        f, u, v, dl, dr = s["gen"]
        return P.psmma_cauchyeig(n, k, c["alpha"], s["A"], f, u, v, dl, dr, c["beta"], s["Q"], **kw)
    fn = {"cauchy": P.psmma_cauchy, "toeplitz": P.psmma_toeplitz, "hankel": P.psmma_hankel}[op]
    return fn(n, k, c["alpha"], s["A"], s["gen"], c["beta"], s["Q"], **kw)


# ---- what a pass cannot do without -----------------------------------------------------------
def _product_work(op, n, k, beta):
    touch = 3 if beta != 0.0 else 2
    if op == "dft":
        return 16.0 * n * k * touch, 5.0 * n * math.log2(max(2, n)) * k
    if op in ("toeplitz", "hankel"):  # two real transforms of 2 k points a row
        return 8.0 * n * k * touch + 16.0 * k, n * (10.0 * k * math.log2(max(2, 2 * k)) + 6.0 * k)
    return 8.0 * n * k * touch + 32.0 * k, 2.0 * n * k * k


def work(case):
    if case["op"].startswith("merge"):
        # two dense diagonal blocks and two blocks of rank about 25 a problem
        b = f = 0.0
        for m in _sizes(case):
            b += 8.0 * m * m * (3 if case["beta"] != 0.0 else 2)
            f += 1.0 * m ** 3 + 4.0 * 25 * m * m
        return {"bytes": b, "flops": f}
    b, f = _product_work(case["op"], case["n"], case["k"], case["beta"])
    return {"bytes": b, "flops": f}


# ---- the same in 64 bits ---------------------------------------------------------------------
def _dense(op, gen, k):
    if op in ("toeplitz", "hankel"):
        i = torch.arange(k, device=DEV)
        idx = i[:, None] + i[None, :] if op == "hankel" else (k - 1) + i[None, :] - i[:, None]
        return gen[idx]
    if op == "cauchy":
        d, f, u, v = gen[:, 0], gen[:, 1], gen[:, 2], gen[:, 3]
        return u[:, None] * v[None, :] / (d[:, None] - f[None, :])
    f, u, v, dl, dr = gen
    i = torch.arange(k, device=DEV)
    f1 = torch.cat([f[1:], f[-1:]])
    low = (f[:, None] - f[None, :]) - dl[None, :]
    high = (f[:, None] - f1[None, :]) - dr[None, :]
    return u[:, None] * v[None, :] / torch.where(i[:, None] <= i[None, :], low, high)


def _on_device(x):
    if isinstance(x, list):
        return [_on_device(y) for y in x]
    return torch.from_numpy(np.ascontiguousarray(x.T)).to(DEV).t() if isinstance(x, np.ndarray) else x


def exact(case, seed):
    s = prepare(case, seed)
    op, k, a, b = case["op"], case["k"], case["alpha"], case["beta"]
    if op.startswith("merge"):
        kind = op.split("_")[1]
        out = []
        for A, gen, Q in s["problems"]:
            r = a * (A @ _dense(kind, gen, A.shape[0]))
            out.append(r + b * Q if b != 0.0 else r)
        return [out, None]
    A, gen, Q = _on_device(s["A"]), _on_device(s["gen"]), _on_device(s["Q"])
    r = a * (torch.fft.fft(A, dim=0) if op == "dft" else A @ _dense(op, gen, k))
    if b != 0.0:
        r = r + b * Q
    return r
