"""Contexts of different sizes in host threads of their own (a context is not re-entrant, two contexts are
independent).  The kernels that keep a system in shared memory are the same functions for every context, and the most
dynamic shared memory that a launch may ask for is an attribute of the function: it has to stay at what the largest
system needs while a smaller one is solved beside it."""

import ctypes
import threading

import numpy as np
import pytest
import torch

from cases import build_gpu_solver, j2_box_spec

pytestmark = pytest.mark.gpu


def _system(dims, **kw):
    from edelweissfe_gb300.solver import TimeStep

    s = build_gpu_solver(j2_box_spec(*dims, *[0.1 * k for k in dims]), **kw)
    d, P, F = s._vec(), s._vec(), s._vec()
    s.computeElements(d, d, P, F, TimeStep(1, 0.1, 0.1, 0.1, 0.1, 0.1))
    s.assembleStiffnessCSR()
    b = torch.as_tensor(np.random.default_rng(sum(dims)).normal(size=s.nDof), device="cuda")
    b[s.dirIdx] = 0.0
    return s, b


# FP64: a cluster of 16 CTAs of 8 lanes per row (50 and 63 rows a CTA); the grid form (25 and 31 rows)
@pytest.mark.parametrize("small,large", [((15, 6, 6), (17, 7, 6)), ((26, 10, 11), (30, 11, 11))], ids=["cluster", "grid"])
def test_solves_of_two_sizes_side_by_side(gpu_lib, small, large):
    """Two threads a size, some hundreds of solves of a few iterations each: every call is accepted and
    returns the bits of the same call made alone."""
    from edelweissfe_gb300 import _lib
    from edelweissfe_gb300.solver import LinSolverOptions

    systems = [_system(d, keFp64=True, linsolver=LinSolverOptions(mixed=False)) for d in (small, large, small, large)]
    opts = _lib.EfSolveOpts(_lib.EF_SOLVE_PCG, 0, 1e-10, 1e-10, 2, 30, 1, 0)
    accepted = (_lib.EF_OK, _lib.EF_NOT_CONVERGED)  # two iterations

    def solve(s, b, x, stream):
        info = _lib.EfSolveInfo()
        st = gpu_lib.ef_solve(s.ctx, ctypes.byref(opts), b.data_ptr(), x.data_ptr(), ctypes.byref(info), stream)
        return st, gpu_lib.ef_last_error()

    alone = []
    for s, b in systems:
        x = s._vec()
        torch.cuda.synchronize()
        assert solve(s, b, x, s._stream())[0] in accepted
        alone.append(x)
    refused, different = [], []
    start = threading.Barrier(len(systems))

    def work(s, b, expected):
        x = s._vec()
        stream = torch.cuda.Stream()
        torch.cuda.synchronize()
        start.wait()
        for _ in range(400):
            st, message = solve(s, b, x, stream.cuda_stream)
            if st not in accepted:
                refused.append((st, message))
        if not torch.equal(x, expected):
            different.append(s.nDof)

    threads = [threading.Thread(target=work, args=(s, b, x)) for (s, b), x in zip(systems, alone)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not refused, (len(refused), refused[0])
    assert not different
