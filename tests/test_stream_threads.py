"""Host threads that share one stream: each call's chain of launches works in the stream's pool, so that a call holds
the pool from taking it to its last launch; results are those of the same calls one after the other."""
import threading

import numpy as np
import pytest

from oracle import psmma_oracle as O

# (kind, n, k, precision): the chains of small and of ordinary products, a product that grows the pool, a DFT
JOBS = [("toeplitz", 256, 200, "fp64"), ("hankel", 900, 1100, "fp64"), ("toeplitz", 2100, 2200, "fp64"),
        ("toeplitz", 300, 300, "split"), ("dft", 480, 7, "fp64")]


def _operands(kind, n, k, seed):
    import torch
    from psmma_git_gb300 import fortran_empty
    dt = torch.complex128 if kind == "dft" else torch.float64
    A, Q = fortran_empty(n, k, dt), fortran_empty(n, k, dt)
    A.copy_(torch.from_numpy(O.cfg_matrix(n, k, seed=seed, complex_=kind == "dft")))
    return A, None if kind == "dft" else torch.from_numpy(O.cfg_vector(2 * k - 1, seed=seed + 1)).cuda(), Q


def _call(job, A, g, Q, stream):
    import psmma_git_gb300 as P
    kind, n, k, prec = job
    if kind == "dft":
        P.pzmdftl(n, k, 1.0, A, 0.0, Q, precision=prec, stream=stream)
    else:
        getattr(P, "psmma_" + kind)(n, k, 1.0, A, g, 0.0, Q, precision=prec, stream=stream)


@pytest.mark.gpu
def test_threads_on_one_stream(cuda):
    import torch
    import psmma_git_gb300 as P
    stream = torch.cuda.Stream()
    ops = [_operands(*job[:3], seed=10 * i + 1) for i, job in enumerate(JOBS)]
    torch.cuda.synchronize()
    want = []
    for job, (A, g, Q) in zip(JOBS, ops):
        _call(job, A, g, Q, stream)
        torch.cuda.synchronize()
        want.append(Q.cpu().numpy().copy())
        Q.zero_()
    torch.cuda.synchronize()
    P.load().psmma_release_workspace()  # the pool grows again while the threads run
    errors, start = [], threading.Barrier(len(JOBS) + 1)

    def worker(job, A, g, Q):
        try:
            torch.cuda.set_device(0)
            start.wait()
            for _ in range(25):
                _call(job, A, g, Q, stream)
        except Exception as e:  # noqa: BLE001
            errors.append(e)

    def releaser():
        torch.cuda.set_device(0)
        start.wait()
        for _ in range(5):
            P.load().psmma_release_workspace()

    threads = [threading.Thread(target=worker, args=(job, *op)) for job, op in zip(JOBS, ops)]
    threads.append(threading.Thread(target=releaser))
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    assert not errors
    for w, (_, _, Q) in zip(want, ops):
        np.testing.assert_array_equal(w, Q.cpu().numpy())
