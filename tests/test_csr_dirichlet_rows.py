"""ef_csr_dirichlet_rows keeps the rows in buffers of its context between calls."""

import numpy as np
import pytest
import torch

from cases import build_gpu_solver, j2_box_spec

pytestmark = pytest.mark.gpu


def _system():
    from edelweissfe_gb300 import _lib
    from edelweissfe_gb300.solver import LinSolverOptions, TimeStep

    s = build_gpu_solver(j2_box_spec(4, 3, 3, 0.4, 0.3, 0.3), keFp64=True, scalarCSR=True, linsolver=LinSolverOptions(mixed=False))
    d, P, F = s._vec(), s._vec(), s._vec()
    s.computeElements(d, d, P, F, TimeStep(1, 0.1, 0.1, 0.1, 0.1, 0.1))
    indptr, indices = np.zeros(s.nDof + 1, np.int32), np.zeros(s.info.nnz, np.int32)
    _lib.check(s.lib.ef_csr_pattern(s.ctx, indptr.ctypes.data, indices.ctypes.data), "ef_csr_pattern")
    data = torch.zeros(s.info.nnz, dtype=torch.float64, device="cuda")
    _lib.check(s.lib.ef_update_csr(s.ctx, None, data.data_ptr(), s._stream()), "ef_update_csr")
    return s, indptr, indices, data


def _apply(s, data, rows):
    return s.lib.ef_csr_dirichlet_rows(s.ctx, data.data_ptr(), rows.ctypes.data, rows.size, s._stream())


def _expected(data, indptr, indices, rows):
    out = data.cpu().numpy().copy()
    for r in rows:
        k = np.arange(indptr[r], indptr[r + 1])
        out[k] = indices[k] == r
    return out


def test_refused_under_capture_and_usable_after(gpu_lib):
    from edelweissfe_gb300 import _lib

    s, indptr, indices, K = _system()
    rows = np.array([0, 5, 17], np.int64)
    data = K.clone()
    assert _apply(s, data, rows) == _lib.EF_OK  # the buffers are there
    assert np.array_equal(data.cpu().numpy(), _expected(K, indptr, indices, rows))
    captured = K.clone()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        captured.mul_(1.0)
        st = _apply(s, captured, rows)
    assert st == _lib.EF_ERR_STATE
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(captured, K)
    data = K.clone()
    assert _apply(s, data, rows) == _lib.EF_OK
    assert np.array_equal(data.cpu().numpy(), _expected(K, indptr, indices, rows))


def test_calls_in_a_row_keep_their_own_rows(gpu_lib):
    """Calls back to back on two streams, fewer and more rows than before, the caller's array reused at once."""
    from edelweissfe_gb300 import _lib

    s, indptr, indices, K = _system()
    rng = np.random.default_rng(1)
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    torch.cuda.synchronize()
    results = []
    rows = np.zeros(40, np.int64)
    for k in range(40):
        n = int(rng.integers(1, 41))
        rows[:n] = rng.choice(s.nDof, n, replace=False)
        with torch.cuda.stream(streams[k % 2]):
            data = K.clone()
            assert _apply(s, data, rows[:n]) == _lib.EF_OK
        results.append((data, rows[:n].copy()))
        rows[:] = 0
    torch.cuda.synchronize()
    for data, r in results:
        assert np.array_equal(data.cpu().numpy(), _expected(K, indptr, indices, r))
