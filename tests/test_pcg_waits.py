"""The bounded waits of the persistent PCG: a CTA that gives up waiting for the others leaves its rows of the solution
unwritten, so the solve fails with EF_ERR_DEVICE whichever CTA it was, and the context stays usable.  EF_PCG_POLLS is the
number of polls after which a wait gives up; with none every wait does, with few some do."""

import os
import shutil
import subprocess

import numpy as np
import pytest
import torch

from cases import build_gpu_solver, j2_box_spec


def test_any_cta_that_gave_up_fails_the_solve(tmp_path):
    """The host's reading of a launch's record: CTA 0 may have written the end of the solve while another gave up."""
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("no C++ compiler")
    plan = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "edelweissfe_gb300", "csrc", "pcg_plan.h")
    source, exe = tmp_path / "check.cpp", str(tmp_path / "check")
    source.write_text(f"""#include "{plan}"
int main() {{
    PcgResult r = {{7, 0, 1, 1.0, 1.0}};
    pcg_result_clear(r);
    if (!pcg_result_timed_out(r)) return 1;  // nobody wrote the record
    r.status = 0;
    if (pcg_result_timed_out(r)) return 2;
    r.gaveUp = 1;
    return pcg_result_timed_out(r) ? 0 : 3;
}}
""")
    subprocess.run([gxx, "-std=c++17", "-o", exe, str(source)], check=True)
    assert subprocess.run([exe]).returncode == 0


# the resident grid form and the streaming kernel
@pytest.mark.gpu
@pytest.mark.parametrize("dims", [(26, 10, 11), (44, 20, 18)], ids=["resident", "streaming"])
@pytest.mark.parametrize("polls", [0, 1, 3, 10, 30])
def test_wait_that_runs_out_is_reported(gpu_lib, monkeypatch, dims, polls):
    import ctypes

    from edelweissfe_gb300 import _lib
    from edelweissfe_gb300.solver import LinSolverOptions, TimeStep

    s = build_gpu_solver(j2_box_spec(*dims, *[0.1 * k for k in dims]), keFp64=True, linsolver=LinSolverOptions(mixed=False, rtol=1e-10))
    d, P, F = s._vec(), s._vec(), s._vec()
    s.computeElements(d, d, P, F, TimeStep(1, 0.1, 0.1, 0.1, 0.1, 0.1))
    s.assembleStiffnessCSR()
    b = torch.as_tensor(np.random.default_rng(6).normal(size=s.nDof), device="cuda")
    b[s.dirIdx] = 0.0
    before = s.linearSolve(b)
    opts = _lib.EfSolveOpts(_lib.EF_SOLVE_PCG, 0, 1e-10, 1e-10, 20000, 30, 1, 0)
    monkeypatch.setenv("EF_PCG_POLLS", str(polls))
    for _ in range(5):
        x, info = s._vec(), _lib.EfSolveInfo()
        st = gpu_lib.ef_solve(s.ctx, ctypes.byref(opts), b.data_ptr(), x.data_ptr(), ctypes.byref(info), s._stream())
        assert st == _lib.EF_ERR_DEVICE or (polls > 0 and st == _lib.EF_OK and torch.equal(x, before)), (st, info.relResidual)
        if st == _lib.EF_ERR_DEVICE:  # the element status reports and clears it, as other device failures
            assert gpu_lib.ef_element_status(s.ctx, s._stream(), None) == _lib.EF_ERR_DEVICE
        assert gpu_lib.ef_element_status(s.ctx, s._stream(), None) == _lib.EF_OK
    monkeypatch.delenv("EF_PCG_POLLS")
    assert torch.equal(s.linearSolve(b), before)
