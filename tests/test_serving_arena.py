"""Requests at the limits of a server's memory budget, and FP64 requests of the real kinds alone and in the mix."""
import numpy as np
import pytest

from oracle import psmma_oracle as O

pytestmark = pytest.mark.gpu


def test_fp64_dft_in_an_arena_of_the_dense_size(cuda):
    # the dense product needs 16 n bytes, the transform of a prime order some six times that
    import torch
    import psmma_git_gb300 as P
    from psmma_git_gb300.server import Server
    n, k = 997, 3
    B = O.cfg_matrix(n, k, seed=2, complex_=True)
    dB = P.fortran_empty(n, k, torch.complex128)
    dB.copy_(torch.from_numpy(B))
    for budget in (20480, 1 << 20):
        dC = P.fortran_empty(n, k, torch.complex128)
        with Server(budget, max_inflight=2) as srv:
            assert srv.wait(srv.submit("dft", n, k, 1.0, dB, None, 0.0, dC, precision="fp64"))["status"] == 0
        assert O.rel_fro(dC.cpu().numpy(), O.dft_product(1.0, B, 0.0, None)) < 1e-13


def test_request_of_the_whole_budget_runs(cuda):
    # the workspace is no whole number of the arena's pages
    import torch
    import psmma_git_gb300 as P
    from psmma_git_gb300.server import Server
    n, k = 70, 60
    need = P.workspace_size(P.KIND_HANKEL, n, k, "split")
    assert need % 4096
    A, g = O.cfg_matrix(n, k, seed=1), O.cfg_vector(2 * k - 1, seed=2)
    dA, dQ, dg = P.fortran_empty(n, k), P.fortran_empty(n, k), torch.from_numpy(g).to(cuda)
    dA.copy_(torch.from_numpy(A))
    with Server(need, max_inflight=2) as srv:
        for t in [srv.submit("hankel", n, k, 1.0, dA, dg, 0.0, dQ) for _ in range(3)]:
            assert srv.wait(t, timeout_s=10.0)["status"] == 0
    assert O.rel_fro(dQ.cpu().numpy(), O.dense_product("hankel", 1.0, A, g, 0.0, None, k)) < 1e-12


def test_fp64_requests_alone_and_in_the_mix(cuda):
    # the server runs the FP64 tensor-core kernel for the real kinds, which have no workspace: the same bits alone, in the
    # mix and by a direct call with a workspace too small for split K; a direct call without one differs by the
    # k FP64 roundings of the kernel's sums at most
    import torch
    import psmma_git_gb300 as P
    from psmma_git_gb300.server import Server
    reqs = []
    for i, (kind, n) in enumerate([("cauchy", 300), ("toeplitz", 900), ("hankel", 513), ("toeplitz", 130),
                                   ("cauchy", 1100), ("hankel", 64)]):
        A = O.cfg_matrix(n, n, seed=40 + i)
        gen = O.cfg_cauchy_generators(n, seed=60 + i) if kind == "cauchy" else O.cfg_vector(2 * n - 1, seed=60 + i)
        dA = P.fortran_empty(n, n)
        dA.copy_(torch.from_numpy(A))
        dg = P.fortran_empty(n, 4) if kind == "cauchy" else torch.empty(2 * n - 1, dtype=torch.float64, device=cuda)
        dg.copy_(torch.from_numpy(gen))
        bound = 2.0 ** -52 * (n + 2) * (np.abs(A) @ np.abs(O.dense_h(kind, gen, n))) * (1 + 1e-9)
        reqs.append((kind, n, dA, dg, bound))
    outs = lambda: [P.fortran_empty(n, n) for _, n, *_ in reqs]
    torch.cuda.synchronize()
    alone, mix = outs(), outs()
    with Server(1 << 20, max_inflight=4) as srv:
        for (kind, n, dA, dg, _), Q in zip(reqs, alone):
            assert srv.wait(srv.submit(kind, n, n, 1.0, dA, dg, 0.0, Q, precision="fp64"))["status"] == 0
        for t in [srv.submit(kind, n, n, 1.0, dA, dg, 0.0, Q, precision="fp64")
                  for (kind, n, dA, dg, _), Q in zip(reqs, mix)]:
            assert srv.wait(t)["status"] == 0
    work = torch.empty(256, dtype=torch.uint8, device=cuda)
    for (kind, n, dA, dg, bound), a, m in zip(reqs, alone, mix):
        assert torch.equal(a, m), (kind, n)
        Q = P.fortran_empty(n, n)
        getattr(P, "psmma_" + kind)(n, n, 1.0, dA, dg, 0.0, Q, work=work)
        assert torch.equal(a, Q), (kind, n)
        getattr(P, "psmma_" + kind)(n, n, 1.0, dA, dg, 0.0, Q)
        assert (np.abs(Q.cpu().numpy() - a.cpu().numpy()) <= bound).all(), (kind, n)


def test_burst_overlaps_on_the_device(cuda):
    # by the requests' own times: those submitted behind a product of some ten milliseconds start before it ends, all in one
    # admission (none waits for the launches, let alone the end, of the one before)
    import torch
    import psmma_git_gb300 as P
    from psmma_git_gb300.server import Server
    big, reqs = 12000, []
    for i, n in enumerate([big, 300, 257, 400]):
        dA, dg = P.fortran_empty(n, n), torch.from_numpy(O.cfg_vector(2 * n - 1, seed=i)).to(cuda)
        dA.copy_(torch.rand(n, n, dtype=torch.float64, device=cuda))
        reqs.append((n, dA, dg, P.fortran_empty(n, n)))
    need = sum(P.workspace_size(P.KIND_TOEPLITZ, n, n, "split") for n, *_ in reqs)
    torch.cuda.synchronize()
    with Server(need + (1 << 20), max_inflight=4) as srv:
        for _ in range(2):  # the first burst pays for the first use of every kernel and stream
            infos = [srv.wait(t) for t in [srv.submit("toeplitz", n, n, 1.0, A, g, 0.0, Q) for n, A, g, Q in reqs]]
    starts = [i["submit_s"] + i["queue_s"] for i in infos]
    assert all(i["status"] == 0 for i in infos)
    assert max(starts) < infos[0]["end_s"]
