"""The batched PCG at the edges of its dispatch: every tile shape on batches that get clusters of 1, 2, 4
and 8 CTAs, with problems from one element (fewer rows than a cluster has CTAs) upwards.  Every problem's
solution is checked against the FP64 system's own product (ef_bsr_matvec): each stops at its own relative
residual of 1e-10, so that 1e-9 leaves the two operators' rounding (about 1e-14 of |K| |x|) ample room."""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

# cubes' edge counts: a lone cube, few uneven ones, one large among small ones, and more than one per SM
BATCHES = {"lone": [5], "few": [1, 2, 9, 3, 6], "uneven": [14] + [2] * 30, "many": [3, 4, 5, 6] * 100}


@pytest.mark.parametrize("name", sorted(BATCHES))
def test_every_tile_solves_every_problem(gpu_lib, name):
    from edelweissfe_gb300 import _lib
    from edelweissfe_gb300.batch import BatchNISTGPU
    from edelweissfe_gb300.solver import TimeStep

    spec = [dict(n=n, props=[210000.0, 0.2 + 0.01 * (k % 20), 250.0, 1000.0, 0.0, 0.0]) for k, n in enumerate(BATCHES[name])]
    s = BatchNISTGPU(spec, graph=False)
    s._elements()
    _lib.check(s.lib.ef_assemble_bsr(s.ctx, s._stream()), "ef_assemble_bsr")
    b = torch.as_tensor(np.random.default_rng(5).normal(size=s.nDof), device="cuda") * s.freeDof
    if len(spec) > 1:
        b[s.problem_dofs(1)] = 0.0  # a problem that is already solved
    for tile in range(s.lib.ef_batch_tile_count()):
        _lib.check(s.lib.ef_batch_set_tile(s.ctx, tile), "ef_batch_set_tile")
        x, y = s._vec(), s._vec()
        _lib.check(s.lib.ef_batch_solve(s.ctx, 1e-10, 20000, b.data_ptr(), x.data_ptr(), s.kIters.data_ptr(),
                                        s.kRel.data_ptr(), s._stream()), "ef_batch_solve")  # fmt: skip
        _lib.check(s.lib.ef_bsr_matvec(s.ctx, x.data_ptr(), y.data_ptr(), s._stream()), "ef_bsr_matvec")
        r = (b - y).cpu().numpy()
        bh, its, rel = b.cpu().numpy(), s.kIters.cpu().numpy(), s.kRel.cpu().numpy()
        assert (rel <= 1e-10).all()
        for p in range(len(spec)):
            d = s.problem_dofs(p)
            if p == 1:
                assert its[p] == 0 and not x[d].any()
            else:
                assert its[p] > 0 and np.linalg.norm(r[d]) <= 1e-9 * np.linalg.norm(bh[d]), (tile, p)
