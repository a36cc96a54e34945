"""The FP64 gradients' limiter, which FP32 bounds decide where they can, against
the oracle: fields at the edges of what the bounds decide (rounding noise, large
offsets, exact ties, values beyond the FP32 range), bit for bit, through the
task entry point and through a solver step (per-mesh tables)."""
import ctypes as C

import numpy as np
import pytest

import flecsale_gb300.hydro as H
from tests import _util as U

pytestmark = pytest.mark.gpu

KINDS = ["smooth", "noise", "offset", "linear", "rough", "huge", "tiny", "mixed"]


def _state(kind, mesh, rng):
    """Positive planes d, v.., e, p, T, a with the field `kind` in each."""
    D, nc = mesh.dim, mesh.num_cells
    x = mesh.arrays()["cell_centroid"]
    s = np.empty((5 + D, nc))
    for k in range(5 + D):
        w = sum(np.sin(2 * np.pi * rng.integers(1, 4) * x[i] + rng.uniform(0, 6)) for i in range(D))
        noise = rng.uniform(-1, 1, nc)
        s[k] = {"smooth": 2 + 0.1 * w, "noise": 1 + 1e-15 * noise, "offset": 1e7 + w + 1e-9 * noise,
                "linear": 2 + x[k % D] + 0.25 * x[(k + 1) % D], "rough": 2 + noise,
                "huge": 1e25 * (2 + 0.1 * w), "tiny": 1e-25 * (2 + 0.1 * w),
                # magnitudes from 2^-100 to 2^100 side by side
                "mixed": np.exp2(100 * noise)}[kind]
    return s


@pytest.mark.parametrize("dim,n,jitter", [(2, (1, 1), 0.0), (2, (3, 2), 0.0), (2, (33, 21), 0.0),
                                          (2, (45, 31), 0.2), (3, (5, 4, 3), 0.0),
                                          (3, (9, 8, 7), 0.15)])
@pytest.mark.parametrize("kind", KINDS)
def test_gradients_bitwise(cuda, oracle_lib, dim, n, jitter, kind):
    torch = cuda
    mesh = H.HostMesh.box(dim, n, [0] * dim, [1] * dim, jitter, 3)
    p = H.make_params(dim, flux="hllc", cfl=0.3, final_time=1e30)
    state = _state(kind, mesh, np.random.default_rng(KINDS.index(kind)))
    dmesh = H.DeviceMesh(mesh)
    ds = torch.tensor(state, device="cuda")
    dg = torch.zeros((U.grad_rows(dim), mesh.num_cells), dtype=torch.float64, device="cuda")
    sv, gv = U.device_state_view(ds, dim), U.device_gradient_view(dg, dim)
    torch.cuda.synchronize()
    H.check(H.lib().fvh_evaluate_gradients(C.byref(dmesh.view), C.byref(sv), C.byref(gv),
                                           C.byref(p), None))
    torch.cuda.synchronize()
    want = U.oracle_gradients(oracle_lib, mesh, state, p)
    assert np.array_equal(dg.cpu().numpy(), want, equal_nan=True)
    # a step with the solver's tables
    dstate = H.DeviceState(dim, mesh.num_cells)
    solver = H.Solver(dmesh, p)
    dstate.upload(state)
    solver.reset(0.0)
    solver.step(dstate)
    out = dstate.download()
    torch.cuda.synchronize()
    st, _, _ = U.oracle_run(oracle_lib, mesh, state, p, 1)
    if st == 0:  # (the oracle stops half-way where the state goes negative)
        assert np.array_equal(out, state, equal_nan=True)


def test_offsets_beyond_the_integer_pipe_range(cuda, oracle_lib):
    """x_nbr - x_c below 2^-500: such a mesh computes its offsets on the fly."""
    mesh = H.HostMesh.box(2, (24, 17), [0, 0], [1e-155, 1e100], 0.0, 3)
    p = H.make_params(2, flux="hllc", cfl=0.3, final_time=1e30)
    state = _state("smooth", mesh, np.random.default_rng(1))
    dmesh, dstate = H.DeviceMesh(mesh), H.DeviceState(2, mesh.num_cells)
    solver = H.Solver(dmesh, p)
    dstate.upload(state)
    solver.reset(0.0)
    solver.step(dstate)
    out = dstate.download()
    cuda.cuda.synchronize()
    st, _, _ = U.oracle_run(oracle_lib, mesh, state, p, 1)
    assert st == 0 and np.array_equal(out, state, equal_nan=True)
