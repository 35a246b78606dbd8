"""The streaming form of the persistent PCG, in both precisions: at small systems, which would run in shared memory
(EF_PCG_RESIDENT=0, which is also what a context does that finds no memory for the resident plan), and at one whose
FP32 blocks are too large for it; and both forms on rows of 81 blocks, on a tied mesh and on uneven rows.

The residual against the FP64 system's own product is checked as in test_pcg_shapes.py: below ten times the
solve's tolerance.  Total-Lagrange systems are taken in the undeformed state."""

import numpy as np
import pytest
import torch

from cases import build_gpu_solver, build_gpu_tied, j2_box_spec, tied_tl_spec

pytestmark = pytest.mark.gpu

SYSTEMS = {
    "hex8-8": lambda **kw: build_gpu_solver(j2_box_spec(1, 1, 1, 0.1, 0.1, 0.1), **kw),
    "hex8-130": lambda **kw: build_gpu_solver(j2_box_spec(12, 1, 4, 1.2, 0.1, 0.4), **kw),
    "hex8-4092": lambda **kw: build_gpu_solver(j2_box_spec(30, 11, 10, 3.0, 1.1, 1.0), **kw),
    "hex20-111": lambda **kw: build_gpu_solver(j2_box_spec(3, 2, 2, 0.3, 0.2, 0.2, elType="C3D20"), **kw),
    "hex20-2241": lambda **kw: build_gpu_solver(j2_box_spec(8, 7, 7, 0.8, 0.7, 0.7, elType="C3D20"), **kw),
    "tied-328": lambda **kw: build_gpu_tied(tied_tl_spec(4, 4, 3, 3), **kw),
    "tied-1981": lambda **kw: build_gpu_tied(tied_tl_spec(8, 8, 6, 6), **kw),
    "hex8-38125": lambda **kw: build_gpu_solver(j2_box_spec(60, 24, 24, 6.0, 2.4, 2.4), **kw),  # FP32: streams anyway
}


@pytest.mark.parametrize("resident", [True, False], ids=["resident", "streaming"])
@pytest.mark.parametrize("name", SYSTEMS)
def test_pcg_solution_satisfies_the_fp64_system(gpu_lib, monkeypatch, name, resident):
    from edelweissfe_gb300 import _lib
    from edelweissfe_gb300.solver import LinSolverOptions, TimeStep

    if not resident:
        monkeypatch.setenv("EF_PCG_RESIDENT", "0")
    solvers = [SYSTEMS[name](keFp64=fp64, linsolver=LinSolverOptions(mixed=not fp64, rtol=1e-9)) for fp64 in (True, False)]
    f = solvers[0]
    b = torch.as_tensor(np.random.default_rng(3).normal(size=f.nDof), device="cuda")
    b[f.dirIdx] = 0.0
    if f.model.ties is not None:
        b.view(-1, 3)[torch.as_tensor(f.model.ties[0], device="cuda")] = 0.0  # eliminated
    for s in solvers:
        d, P, F = s._vec(), s._vec(), s._vec()
        s.computeElements(d, d, P, F, TimeStep(1, 0.1, 0.1, 0.1, 0.1, 0.1))
        s.assembleStiffnessCSR()
    for s in solvers:
        x = s.linearSolve(b)
        y = f._vec()
        _lib.check(f.lib.ef_bsr_matvec(f.ctx, x.data_ptr(), y.data_ptr(), f._stream()), "ef_bsr_matvec")
        free = torch.ones_like(b)
        if f.model.ties is not None:
            free.view(-1, 3)[torch.as_tensor(f.model.ties[0], device="cuda")] = 0.0
        assert float(((b - y) * free).norm() / b.norm()) <= 1e-8
        assert s.lastSolveInfo.relResidual <= 1e-9 and float(x[s.dirIdx].abs().max()) == 0.0
