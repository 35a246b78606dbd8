"""What ef_batch_setup chooses for a batch before any tuning."""

import os
import shutil
import subprocess

import numpy as np
import pytest
import torch


def test_default_tile_by_the_mean_problem_size(tmp_path):
    """128 threads a CTA (tile 1) for problems of up to 64 nodes on average, else 512 (tile 6)."""
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("no C++ compiler")
    plan = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "edelweissfe_gb300", "csrc", "pcg_plan.h")
    cases = {(1, 8): 1, (1, 64): 1, (1, 65): 6, (3, 192): 1, (3, 193): 6, (2000, 16000): 1, (1 << 26, 1 << 30): 1, (160, 200000): 6}
    checks = " && ".join(f"ef_batch_default_tile({p}, {n}) == {t}" for (p, n), t in cases.items())
    source, exe = tmp_path / "check.cpp", str(tmp_path / "check")
    source.write_text(f'#include "{plan}"\nint main() {{ return {checks} ? 0 : 1; }}\n')
    subprocess.run([gxx, "-std=c++17", "-o", exe, str(source)], check=True)
    assert subprocess.run([exe]).returncode == 0


def _batch(sizes):
    from edelweissfe_gb300.batch import BatchNISTGPU
    from edelweissfe_gb300.solver import TimeStep

    s = BatchNISTGPU([dict(n=n, props=[210000.0, 0.3, 250.0, 1000.0, 0.0, 0.0]) for n in sizes])
    d, P, F = s._vec(), s._vec(), s._vec()
    s.computeElements(d, d, P, F, TimeStep(1, 0.1, 0.1, 0.1, 0.1, 0.1))
    s.assembleStiffnessCSR()
    b = torch.as_tensor(np.random.default_rng(8).normal(size=s.nDof), device="cuda") * s.freeDof
    return s, b


def _solve(s, b):
    from edelweissfe_gb300 import _lib

    x = s._vec()
    _lib.check(s.lib.ef_batch_solve(s.ctx, 1e-10, 20000, b.data_ptr(), x.data_ptr(), s.kIters.data_ptr(),
                                    s.kRel.data_ptr(), s._stream()), "ef_batch_solve")  # fmt: skip
    assert float(s.kRel.max()) <= 1e-10
    return x


@pytest.mark.gpu
@pytest.mark.parametrize("sizes,tile", [([1, 2, 3] * 9, 1), ([3] * 5, 1), ([3, 3, 4], 6), ([4] * 6, 6)])
def test_untuned_tile_follows_the_problem_size(gpu_lib, sizes, tile):
    """An untuned solve has the bits of one with that tile set, and a tile that was set outlives another set-up."""
    from edelweissfe_gb300 import _lib

    s, b = _batch(sizes)
    x = _solve(s, b)
    assert [s.tile_shapes()[t] for t in (1, 6)] == [(128, 4), (512, 4)]
    _lib.check(s.lib.ef_batch_set_tile(s.ctx, tile), "ef_batch_set_tile")
    assert torch.equal(x, _solve(s, b))
    _lib.check(s.lib.ef_batch_set_tile(s.ctx, 7 - tile), "ef_batch_set_tile")
    y = _solve(s, b)
    _lib.check(s.lib.ef_batch_setup(s.ctx, s.nProb, s.nodePtr.ctypes.data), "ef_batch_setup")
    assert torch.equal(y, _solve(s, b))


@pytest.mark.gpu
@pytest.mark.parametrize("sizes", [[5], [1, 2, 9, 3, 6], [14] + [2] * 30, [3, 4, 5, 6] * 100], ids=["lone", "few", "uneven", "many"])
def test_solves_without_the_sliced_copy(gpu_lib, monkeypatch, sizes):
    """A batch whose sliced copy finds no room (EF_BATCH_SLICED=0 stands in for it) is solved from the block rows, with every
    tile and cluster size, by the same sums."""
    from edelweissfe_gb300 import _lib

    s, b = _batch(sizes)
    for tile in range(gpu_lib.ef_batch_tile_count()):
        _lib.check(s.lib.ef_batch_set_tile(s.ctx, tile), "ef_batch_set_tile")
        with monkeypatch.context() as env:
            x = _solve(s, b)
            env.setenv("EF_BATCH_SLICED", "0")
            free = torch.cuda.mem_get_info()[0]
            _lib.check(s.lib.ef_batch_setup(s.ctx, s.nProb, s.nodePtr.ctypes.data), "ef_batch_setup")
            assert torch.cuda.mem_get_info()[0] >= free
            assert torch.equal(x, _solve(s, b))
        _lib.check(s.lib.ef_batch_setup(s.ctx, s.nProb, s.nodePtr.ctypes.data), "ef_batch_setup")


@pytest.mark.gpu
@pytest.mark.parametrize("tile", [0, 1, 2, 3, 4, 5, 6])
def test_problems_without_nodes(gpu_lib, tile):
    """Empty node ranges among the others, and enough of them that clusters take only such problems."""
    from edelweissfe_gb300 import _lib

    s, b = _batch([2, 5, 1])
    _lib.check(s.lib.ef_batch_set_tile(s.ctx, tile), "ef_batch_set_tile")
    x = _solve(s, b)
    ptr = np.concatenate([[0], s.nodePtr, np.full(400, s.nodePtr[-1])]).astype(np.int32)  # 401 empty ones
    n = len(ptr) - 1
    its = torch.full((n,), -1, dtype=torch.int32, device="cuda")
    rel = torch.full((n,), -1.0, dtype=torch.float64, device="cuda")
    out = torch.full((n, 3), -1.0, dtype=torch.float64, device="cuda")
    y = s._vec()
    _lib.check(s.lib.ef_batch_setup(s.ctx, n, ptr.ctypes.data), "ef_batch_setup")
    _lib.check(s.lib.ef_batch_solve(s.ctx, 1e-10, 20000, b.data_ptr(), y.data_ptr(), its.data_ptr(), rel.data_ptr(),
                                    s._stream()), "ef_batch_solve")  # fmt: skip
    _lib.check(s.lib.ef_batch_norms(s.ctx, b.data_ptr(), b.data_ptr(), None, out.data_ptr(), s._stream()), "ef_batch_norms")
    its, rel, out = its.cpu().numpy(), rel.cpu().numpy(), out.cpu().numpy()
    some = np.diff(ptr) > 0
    assert (its[some] > 0).all() and (rel[some] <= 1e-10).all() and (out[some, 0] > 0).all()
    assert not its[~some].any() and not rel[~some].any() and not out[~some].any()
    assert float((x - y).norm() / x.norm()) <= 1e-6  # (another cluster size may sum in another order)
