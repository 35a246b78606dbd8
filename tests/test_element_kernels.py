"""The element kernels where their partition has an edge: element counts around a CTA's for the reduced and the
total-Lagrange elements (1, 2 or 8 elements a CTA in FP64, 1, 8 or 16 in FP32, by the Gauss points), and the signs that the
FP64 stiffness takes out of its factors: w detJ < 0 in an inverted element, c1 < 0 under softening."""

import ctypes

import numpy as np
import pytest
import torch

from test_gpu_parity import _ctx_for_elements, golden

pytestmark = pytest.mark.gpu


def _stiffness(lib, elType, material, props, coords, state0, U, dU, keFp64, status=True):
    """(Ke [e, n, n], Pe [e, n]) of elements on degrees of freedom of their own."""
    from edelweissfe_gb300 import _lib

    nEl, nd = coords.shape[0], 3 * coords.shape[1]
    ctx, nDof = _ctx_for_elements(lib, elType, material, props, np.ascontiguousarray(coords), keFp64)
    try:
        if state0 is not None:
            state0 = np.ascontiguousarray(state0)
            _lib.check(lib.ef_set_state(ctx, 0, state0.ctypes.data), "ef_set_state")
        U, dU = (torch.as_tensor(np.ascontiguousarray(v).reshape(-1), device="cuda") for v in (U, dU))
        P = torch.zeros(nDof, dtype=torch.float64, device="cuda")
        F = torch.zeros_like(P)
        t = np.array([0.5, 0.5])
        _lib.check(lib.ef_compute_elements(ctx, U.data_ptr(), dU.data_ptr(), t.ctypes.data, 0.1, P.data_ptr(), F.data_ptr(),
                                           None), "ef_compute_elements")  # fmt: skip
        st = lib.ef_element_status(ctx, None, None)
        assert st == _lib.EF_OK or not status
        info = _lib.EfInfo()
        lib.ef_get_info(ctx, ctypes.byref(info))
        K = torch.zeros(info.nVIJ, dtype=torch.float64, device="cuda")
        _lib.check(lib.ef_export_vij(ctx, K.data_ptr(), None), "ef_export_vij")
        return K.cpu().numpy().reshape(nEl, nd, nd), P.cpu().numpy().reshape(nEl, nd)
    finally:
        lib.ef_destroy(ctx)


COUNTS = {
    ("C3D8R", "vonmises"): (1, 7, 8, 9, 15, 17, 33),
    ("C3D8E", "vonmises"): (1, 2, 3, 5),
    ("C3D20R", "vonmises"): (1, 7, 9, 17),
    ("C3D8TL", "neohookewa"): (1, 7, 8, 9, 17),
    ("C3D8RTL", "neohookewa"): (1, 7, 8, 9, 17),
    ("C3D8ETL", "neohookewa"): (1, 2, 3, 5),
    ("C3D20TL", "neohookewa"): (1, 2, 3, 5),
    ("C3D20RTL", "neohookewa"): (1, 7, 8, 9, 17),
}


@pytest.mark.parametrize("keFp64", [True, False], ids=["fp64", "fp32K"])
@pytest.mark.parametrize("elType,material,nEl", [(e, m, n) for (e, m), counts in COUNTS.items() for n in counts])
def test_every_element_count_gives_the_reference_stiffness(gpu_lib, elType, material, nEl, keFp64):
    """The reference fixture's elements repeated nEl times around, to the tolerances of the fixture's own test."""
    g = golden(f"elem_{elType}_{material}.npz")
    n0, nn = g["coords"].shape[:2]
    idx = np.arange(nEl) % n0
    K, P = _stiffness(gpu_lib, elType, material, g["props"], g["coords"][idx], g["state0"][idx],
                      g["U"].reshape(n0, -1)[idx], g["dU"].reshape(n0, -1)[idx], keFp64)  # fmt: skip
    Kref = g["Kvij"].reshape(n0, 3 * nn, 3 * nn)
    Pref = g["Pe"].reshape(n0, -1)
    tolK = 1e-11 if keFp64 else 2e-6
    assert np.max(np.abs(K - Kref[idx])) <= tolK * np.max(np.abs(Kref))
    assert np.max(np.abs(P - Pref[idx])) <= 1e-11 * np.max(np.abs(Pref))


@pytest.mark.parametrize("elType", ["C3D8", "C3D8R", "C3D8E"])
def test_inverted_element_has_the_negative_weight_in_its_stiffness(gpu_lib, elType):
    """Element and displacements mirrored through the node order: detJ changes its sign and nothing else, so Ke and
    Pe are those of the element itself with the nodes exchanged and all signs turned.  Elastic and plastic increments."""
    from edelweissfe_gb300.mesh import box_mesh

    m = box_mesh(1, 1, 1, 0.1, 0.1, 0.1)
    X = m["coords"][m["elements"][0]]
    nn = len(X)
    # the node that takes a node's place when the first axis turns round
    mirror = np.array([np.argmin(np.linalg.norm(X - np.where([True, False, False], 0.1 - x, x), axis=1)) for x in X])
    props = np.array([210000.0, 0.3, 250.0, 1000.0, 0.0, 0.0])
    rng = np.random.default_rng(2)
    amplitude = np.array([1e-6, 4e-4])[:, None, None]  # strains of 1e-5 and of several yield strains
    u = amplitude * rng.uniform(-1, 1, (2, nn, 3))
    coords = np.stack([X, X])
    K, P = _stiffness(gpu_lib, elType, "vonmises", props, coords, None, u, u, True)
    Km, Pm = _stiffness(gpu_lib, elType, "vonmises", props, coords[:, mirror], None, u[:, mirror], u[:, mirror], True, status=False)
    d = (3 * mirror[:, None] + np.arange(3)).ravel()
    for e in range(2):
        assert np.max(np.abs(Km[e] + K[e][np.ix_(d, d)])) <= 1e-12 * np.max(np.abs(K[e]))
        assert np.max(np.abs(Pm[e] + P[e][d])) <= 1e-12 * np.max(np.abs(P[e]))


@pytest.mark.parametrize("elType", ["C3D8", "C3D8R"])
@pytest.mark.parametrize("fy0,H", [(250.0, 1000.0), (250.0, -20000.0), (-50.0, 1000.0)], ids=["hardening", "softening", "c1<0"])
def test_fp64_stiffness_of_either_sign_of_the_plastic_term(gpu_lib, elType, fy0, H):
    """c1 is negative where the yield stress has fallen below zero.  Ke is symmetric and the derivative of -Pe: against central differences, whose error with steps of 1e-7 of the strains
    in question is below 1e-5 of max |Ke| (rounding 1e-16 / 1e-7 of the forces, and the curvature of the return map over a step)."""
    from edelweissfe_gb300.mesh import box_mesh

    m = box_mesh(1, 1, 1, 0.1, 0.1, 0.1)
    X = m["coords"][m["elements"][0]]
    nn = len(X)
    props = np.array([210000.0, 0.3, fy0, H, 0.0, 0.0])
    u0 = 4e-4 * np.random.default_rng(4).uniform(-1, 1, (nn, 3)) + 0.004 * X * np.array([1.0, -0.4, -0.4])
    h = 1e-10
    steps = np.eye(3 * nn).reshape(3 * nn, nn, 3) * h
    u = np.concatenate([u0[None], u0[None] + steps, u0[None] - steps])
    K, P = _stiffness(gpu_lib, elType, "vonmises", props, np.repeat(X[None], len(u), 0), None, u, u, True)
    fd = -(P[1 : 1 + 3 * nn] - P[1 + 3 * nn :]).T / (2 * h)
    scale = np.max(np.abs(K[0]))
    assert np.max(np.abs(K[0] - K[0].T)) <= 1e-12 * scale
    assert np.max(np.abs(K[0] - fd)) <= 1e-5 * scale
