"""The scalar CSR from a VIJ vector and from the context's own element blocks, bit for bit the reference's serial loop
data[x[k]] += V[k] (numerics/csrgenerator.pyx:100-115): elements of 24 and 60 degrees of freedom and groups of
both, FP64 and FP32 stiffness, few and many values per slot (dealt out over a CTA above 1.7), last CTAs part filled."""

import ctypes

import numpy as np
import pytest
import torch

from cases import J2_PROPS

pytestmark = pytest.mark.gpu

# (elements, box): 1, 1.5 and 1.95 values per slot of 8-node elements, 1, 1.2 and 1.4 of 20-node ones, and both in one model
MODELS = {
    "hex8-1": [("C3D8", (1, 1, 1))],
    "hex8-8": [("C3D8", (2, 2, 2))],
    "hex8-125": [("C3D8", (5, 5, 5))],
    "hex20-1": [("C3D20", (1, 1, 1))],
    "hex20-4": [("C3D20", (2, 2, 1))],
    "hex20-27": [("C3D20", (3, 3, 3))],
    "hex20-hex8": [("C3D20", (2, 2, 1)), ("C3D8", (3, 2, 2))],
    "hex8-hex20-hex8": [("C3D8", (1, 2, 1)), ("C3D20R", (2, 1, 1)), ("C3D8R", (2, 2, 3))],
}


@pytest.mark.parametrize("keFp64", [True, False], ids=["fp64", "fp32K"])
@pytest.mark.parametrize("name", MODELS)
def test_csr_of_both_routes_is_the_serial_loop(gpu_lib, name, keFp64):
    from edelweissfe_gb300 import _lib
    from edelweissfe_gb300.mesh import box_mesh
    from edelweissfe_gb300.model import ElementGroup, Model
    from edelweissfe_gb300.solver import LinSolverOptions, NISTGPU, TimeStep

    coords, groups, dofs = [], [], []
    for i, (el, n) in enumerate(MODELS[name]):  # boxes side by side, without common nodes
        m = box_mesh(*n, *[0.1 * k for k in n], x0=float(i), nNodesPerElement=20 if "20" in el else 8)
        elements = m["elements"] + sum(len(c) for c in coords)
        coords.append(m["coords"])
        groups.append(ElementGroup(el, elements, "vonmises", np.array(J2_PROPS)))
        dofs += [(3 * e[:, None] + np.arange(3)).ravel() for e in elements]
    s = NISTGPU(Model(np.concatenate(coords), groups), keFp64=keFp64, linsolver=LinSolverOptions(mixed=not keFp64),
                scalarCSR=True)  # fmt: skip
    rng = np.random.default_rng(5)
    d = torch.as_tensor(2e-4 * rng.normal(size=s.nDof), device="cuda")  # partly plastic: no two blocks alike
    P, F = s._vec(), s._vec()
    s.computeElements(d, d, P, F, TimeStep(1, 0.1, 0.1, 0.1, 0.1, 0.1))
    info = _lib.EfInfo()
    gpu_lib.ef_get_info(s.ctx, ctypes.byref(info))
    V = torch.full((info.nVIJ,), float("nan"), dtype=torch.float64, device="cuda")
    _lib.check(gpu_lib.ef_export_vij(s.ctx, V.data_ptr(), None), "ef_export_vij")
    indptr, indices = np.zeros(s.nDof + 1, np.int32), np.zeros(info.nnz, np.int32)
    _lib.check(gpu_lib.ef_csr_pattern(s.ctx, indptr.ctypes.data, indices.ctypes.data), "ef_csr_pattern")
    key = np.repeat(np.arange(s.nDof), np.diff(indptr)) * s.nDof + indices
    # value i + j n of an element's slice: row i, column j
    vij = np.concatenate([(e[None, :] * s.nDof + e[:, None]).ravel() for e in dofs])
    expected = np.zeros(info.nnz)
    np.add.at(expected, np.searchsorted(key, vij), V.cpu().numpy())
    for K in (None, V):
        data = torch.full((info.nnz,), float("nan"), dtype=torch.float64, device="cuda")
        _lib.check(gpu_lib.ef_update_csr(s.ctx, None if K is None else K.data_ptr(), data.data_ptr(), None), "ef_update_csr")
        assert np.array_equal(data.cpu().numpy(), expected)
