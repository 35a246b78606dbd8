"""The persistent PCG at the edges of its dispatch: one cluster of 1, 2, ... 16 CTAs (FP32 systems of up to
128 rows a CTA, more where they still fit into shared memory; FP64 of 16 rows a CTA), the grid form with its
slots, and the streaming kernel where a system does not fit into the SMs' shared memory.

Solves with rtol 1e-10 are checked against the FP64 system's own product (ef_bsr_matvec): the residual
of both the all-FP64 and the mixed solution, whose refinement sees the same tangent matrix-free, stays
below 1e-9, ten times the tolerance, which covers the rounding of either operator (about 1e-14
of |K| |x|, with |K| |x| / |b| below 1e4 on these systems)."""

import numpy as np
import pytest
import torch

from cases import build_gpu_solver, j2_box_spec

pytestmark = pytest.mark.gpu

# nodes: 8, 36 | 126, 130 (one CTA in FP32, then two) | 2040, 2057 (128 rows a CTA on 16 CTAs, then more)
# | 3564, 4092 (grid) | 17955 (FP64: streams)
DIMS = [(1, 1, 1), (3, 2, 2), (6, 2, 5), (12, 1, 4), (16, 9, 11), (16, 10, 10), (26, 10, 11), (30, 11, 10), (44, 20, 18)]


@pytest.mark.parametrize("dims", DIMS, ids=lambda d: "x".join(map(str, d)))
def test_pcg_solution_satisfies_the_fp64_system(gpu_lib, dims):
    from edelweissfe_gb300 import _lib
    from edelweissfe_gb300.solver import LinSolverOptions, TimeStep

    spec = j2_box_spec(*dims, *[0.1 * k for k in dims])
    ts = TimeStep(1, 0.1, 0.1, 0.1, 0.1, 0.1)
    solvers = [build_gpu_solver(spec, keFp64=fp64, linsolver=LinSolverOptions(mixed=not fp64, rtol=1e-10))
               for fp64 in (True, False)]  # fmt: skip
    b = torch.as_tensor(np.random.default_rng(3).normal(size=solvers[0].nDof), device="cuda")
    b[solvers[0].dirIdx] = 0.0
    for s in solvers:
        d, P, F = s._vec(), s._vec(), s._vec()
        s.computeElements(d, d, P, F, ts)
        s.assembleStiffnessCSR()
    for s in solvers:
        for _ in range(2):  # a second solve finds the first one's slots and vectors
            x = s.linearSolve(b)
            y = s._vec()
            f = solvers[0]
            _lib.check(f.lib.ef_bsr_matvec(f.ctx, x.data_ptr(), y.data_ptr(), f._stream()), "ef_bsr_matvec")
            assert float((b - y).norm() / b.norm()) <= 1e-9
            assert s.lastSolveInfo.relResidual <= 1e-10 and float(x[s.dirIdx].abs().max()) == 0.0
