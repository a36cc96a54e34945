"""The task calls (no tables) on both sides of the sizes at which the FP64 kernels
change form, against the oracle bit for bit."""
import ctypes as C

import numpy as np
import pytest

import flecsale_gb300.hydro as H
from tests import _util as U

pytestmark = pytest.mark.gpu


def _state(dim, x):
    w = 0.05 * np.sin(2 * np.pi * (2 * x + np.arange(dim)[:, None]))
    return H.state_from_dvp(dim, 1 + w.sum(0) + (x[0] < 0.5), w, 1 + 1.4 * w.sum(0) + (x[0] < 0.5))


# 15,360 and 15,376 cells, 6,400 and 6,480; 8,000 and 8,400
@pytest.mark.parametrize("dim,n", [(2, (128, 120)), (2, (124, 124)), (2, (80, 80)), (2, (81, 80)),
                                   (3, (20, 20, 20)), (3, (20, 20, 21))])
@pytest.mark.parametrize("limiter", ["barth_jespersen", "none"])
@pytest.mark.parametrize("jitter", [0.0, 0.15])
def test_gradients(cuda, oracle_lib, dim, n, limiter, jitter):
    mesh = H.HostMesh.box(dim, n, [0] * dim, [1] * dim, jitter, 5)
    p = H.make_params(dim, limiter=limiter, cfl=0.3)
    state = _state(dim, mesh.arrays()["cell_centroid"])
    dmesh = H.DeviceMesh(mesh)
    ds = cuda.tensor(state, device="cuda")
    dg = cuda.zeros((U.grad_rows(dim), mesh.num_cells), dtype=cuda.float64, device="cuda")
    sv, gv = U.device_state_view(ds, dim), U.device_gradient_view(dg, dim)
    cuda.cuda.synchronize()
    H.check(H.lib().fvh_evaluate_gradients(C.byref(dmesh.view), C.byref(sv), C.byref(gv),
                                           C.byref(p), None))
    cuda.cuda.synchronize()
    assert np.array_equal(dg.cpu().numpy(), U.oracle_gradients(oracle_lib, mesh, state, p))


# 9,940 faces and 10,081; 6,072 and 10,095
@pytest.mark.parametrize("dim,n", [(2, (70, 70)), (2, (71, 70)), (3, (12, 12, 13)), (3, (15, 15, 14))])
@pytest.mark.parametrize("flux", ["hlle", "hllc", "rusanov"])
@pytest.mark.parametrize("order", [1, 2])
def test_fluxes(cuda, oracle_lib, dim, n, flux, order):
    mesh = H.HostMesh.box(dim, n, [0] * dim, [1] * dim, 0.15, 5)
    p = H.make_params(dim, flux=flux, order=order, cfl=0.3)
    state = _state(dim, mesh.arrays()["cell_centroid"])
    grads = U.oracle_gradients(oracle_lib, mesh, state, p)
    dmesh = H.DeviceMesh(mesh)
    ds, dg = (cuda.tensor(a, device="cuda") for a in (state, grads))
    df = cuda.zeros((dim + 2, mesh.num_faces), dtype=cuda.float64, device="cuda")
    sv, gv = U.device_state_view(ds, dim), U.device_gradient_view(dg, dim)
    fv = U.device_flux_view(df, dim)
    cuda.cuda.synchronize()
    H.check(H.lib().fvh_evaluate_fluxes(C.byref(dmesh.view), C.byref(sv), C.byref(gv), C.byref(fv),
                                        C.byref(p), None))
    cuda.cuda.synchronize()
    assert np.array_equal(df.cpu().numpy(), U.oracle_fluxes(oracle_lib, mesh, state, grads, p))
