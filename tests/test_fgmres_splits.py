"""The fine kernels of the FGMRES solve with every number of warps per slice (the rule takes 4 to 32 by the
number of slices; 1 and 2 are options), on packed and diagonal slices whose last one is part filled and
whose warps get no step at all, and the coarse kernels on both sides of their rules (a warp or a CTA per
coarse node of the restriction).  The refined solution, whatever the preconditioner rounds, satisfies the FP64
system: the residual against the FP64 context's own product stays below 1e-7, ten times the solve's rtol."""

import numpy as np
import pytest
import torch

from cases import build_gpu_solver, j2_box_spec

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("warps", [1, 2, 4, 8, 16, 32])
@pytest.mark.parametrize("elType,dims", [("C3D8", (9, 4, 6)), ("C3D20", (5, 3, 2)), ("C3D8", (30, 13, 9))])
def test_fgmres_with_every_split_solves_the_fp64_system(gpu_lib, monkeypatch, elType, dims, warps):
    from edelweissfe_gb300 import _lib
    from edelweissfe_gb300.solver import LinSolverOptions, TimeStep

    monkeypatch.setenv("EF_SELL_SPLIT", str(warps))
    monkeypatch.setenv("EF_SELL_SPLIT_PRODUCT", str(warps))
    monkeypatch.setenv("EF_SA_RESTRICT_WARP", str(warps & 1))
    spec = j2_box_spec(*dims, *[0.1 * k for k in dims], elType=elType)
    ts = TimeStep(1, 0.1, 0.1, 0.1, 0.1, 0.1)
    s = build_gpu_solver(spec, linsolver=LinSolverOptions(method="fgmres", rtol=1e-8))
    f = build_gpu_solver(spec, keFp64=True, linsolver=LinSolverOptions(mixed=False))
    b = torch.as_tensor(np.random.default_rng(7).normal(size=s.nDof), device="cuda")
    b[s.dirIdx] = 0.0
    for g in (s, f):
        d, P, F = g._vec(), g._vec(), g._vec()
        g.computeElements(d, d, P, F, ts)
        g.assembleStiffnessCSR()
    x, y = s.linearSolve(b), s._vec()
    _lib.check(f.lib.ef_bsr_matvec(f.ctx, x.data_ptr(), y.data_ptr(), f._stream()), "ef_bsr_matvec")
    assert float((b - y).norm() / b.norm()) <= 1e-7
    assert s.lastSolveInfo.relResidual <= 1e-8


@pytest.mark.parametrize("dims", [(4, 2, 2), (50, 16, 16), (60, 20, 20)], ids=lambda d: "x".join(map(str, d)))
def test_fgmres_gram_schmidt_of_every_vector_length(gpu_lib, dims):
    """Vectors of 135, 44,217 and 80,703 elements: the basis dealt out over four, two and one set of threads
    (13,000 elements above: four); more columns than are loaded ahead.  The same check."""
    from edelweissfe_gb300 import _lib
    from edelweissfe_gb300.solver import LinSolverOptions, TimeStep

    spec = j2_box_spec(*dims, *[0.1 * k for k in dims])
    ts = TimeStep(1, 0.1, 0.1, 0.1, 0.1, 0.1)
    s = build_gpu_solver(spec, linsolver=LinSolverOptions(method="fgmres", rtol=1e-8, innerRtol=1e-7, restart=100))
    f = build_gpu_solver(spec, keFp64=True, linsolver=LinSolverOptions(mixed=False))
    b = torch.as_tensor(np.random.default_rng(9).normal(size=s.nDof), device="cuda")
    b[s.dirIdx] = 0.0
    for g in (s, f):
        d, P, F = g._vec(), g._vec(), g._vec()
        g.computeElements(d, d, P, F, ts)
        g.assembleStiffnessCSR()
    x, y = s.linearSolve(b), s._vec()
    _lib.check(f.lib.ef_bsr_matvec(f.ctx, x.data_ptr(), y.data_ptr(), f._stream()), "ef_bsr_matvec")
    assert float((b - y).norm() / b.norm()) <= 1e-7


@pytest.mark.parametrize("dims", [(24, 49, 47), (24, 49, 48)], ids=["60000-nodes", "61250-nodes"])
def test_fgmres_product_on_both_sides_of_its_streaming_rule(gpu_lib, dims):
    """The product in the diagonal form reads cached lines up to 60,000 nodes and streams above.  The same check."""
    from edelweissfe_gb300 import _lib
    from edelweissfe_gb300.solver import LinSolverOptions, TimeStep

    spec = j2_box_spec(*dims, *[0.1 * k for k in dims])
    ts = TimeStep(1, 0.1, 0.1, 0.1, 0.1, 0.1)
    s = build_gpu_solver(spec, linsolver=LinSolverOptions(method="fgmres", rtol=1e-8))
    f = build_gpu_solver(spec, keFp64=True, linsolver=LinSolverOptions(mixed=False))
    b = torch.as_tensor(np.random.default_rng(11).normal(size=s.nDof), device="cuda")
    b[s.dirIdx] = 0.0
    for g in (s, f):
        d, P, F = g._vec(), g._vec(), g._vec()
        g.computeElements(d, d, P, F, ts)
        g.assembleStiffnessCSR()
    x, y = s.linearSolve(b), s._vec()
    _lib.check(f.lib.ef_bsr_matvec(f.ctx, x.data_ptr(), y.data_ptr(), f._stream()), "ef_bsr_matvec")
    assert float((b - y).norm() / b.norm()) <= 1e-7
