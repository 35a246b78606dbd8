"""The element kernels with element counts around their CTAs' (hex8: 8 elements in FP64, 16 in FP32; hex20: 2 and 4): the
stiffness is dealt out over the pairs of nodes of a CTA's elements, the last CTA of which is part filled.  The
elements of a reference fixture, some of them plastic, are repeated on degrees of freedom of their own; every
copy has the fixture's stiffness and forces, to the tolerances of the fixture's own test."""

import ctypes

import numpy as np
import pytest
import torch

from test_gpu_parity import _ctx_for_elements, golden

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("keFp64", [True, False], ids=["fp64", "fp32K"])
@pytest.mark.parametrize("elType,nEl", [("C3D8", n) for n in (1, 7, 8, 9, 15, 17, 33)] + [("C3D20", n) for n in (1, 2, 3, 5)])
def test_every_element_count_gives_the_reference_stiffness(gpu_lib, elType, nEl, keFp64):
    from edelweissfe_gb300 import _lib

    g = golden(f"elem_{elType}_vonmises.npz")
    nn = g["coords"].shape[1]
    idx = np.arange(nEl) % g["coords"].shape[0]
    ctx, nDof = _ctx_for_elements(gpu_lib, elType, "vonmises", g["props"], np.ascontiguousarray(g["coords"][idx]), keFp64)
    try:
        state0 = np.ascontiguousarray(g["state0"][idx])
        _lib.check(gpu_lib.ef_set_state(ctx, 0, state0.ctypes.data), "ef_set_state")
        U = torch.as_tensor(g["U"].reshape(g["coords"].shape[0], -1)[idx].reshape(-1), device="cuda")
        dU = torch.as_tensor(g["dU"].reshape(g["coords"].shape[0], -1)[idx].reshape(-1), device="cuda")
        P = torch.zeros(nDof, dtype=torch.float64, device="cuda")
        F = torch.zeros_like(P)
        t = np.array([0.5, 0.5])
        _lib.check(gpu_lib.ef_compute_elements(ctx, U.data_ptr(), dU.data_ptr(), t.ctypes.data, 0.1, P.data_ptr(),
                                               F.data_ptr(), None), "ef_compute_elements")  # fmt: skip
        assert gpu_lib.ef_element_status(ctx, None, None) == _lib.EF_OK
        info = _lib.EfInfo()
        gpu_lib.ef_get_info(ctx, ctypes.byref(info))
        K = torch.zeros(info.nVIJ, dtype=torch.float64, device="cuda")
        _lib.check(gpu_lib.ef_export_vij(ctx, K.data_ptr(), None), "ef_export_vij")
        Kref = g["Kvij"].reshape(-1, 3 * nn, 3 * nn)
        Pref = g["Pe"].reshape(len(Kref), -1)
        tolK = 1e-11 if keFp64 else 2e-6
        assert np.max(np.abs(K.cpu().numpy().reshape(nEl, 3 * nn, 3 * nn) - Kref[idx])) <= tolK * np.max(np.abs(Kref))
        assert np.max(np.abs(P.cpu().numpy().reshape(nEl, -1) - Pref[idx])) <= 1e-11 * np.max(np.abs(Pref))
    finally:
        gpu_lib.ef_destroy(ctx)
