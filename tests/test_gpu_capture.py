"""Calls in a stream under capture: a step or run is refused and leaves the capture
and the solver as they were; the tasks are captured."""
import ctypes as C

import numpy as np
import pytest

import flecsale_gb300.hydro as H
from tests import _util as U

pytestmark = pytest.mark.gpu


def _setup(precision, order=2):
    mesh = H.HostMesh.box(2, (24, 17), [0, 0], [1, 1], 0.15, 5)
    p = H.make_params(2, flux="hllc", order=order, cfl=0.3, final_time=1e9, precision=precision)
    x = mesh.arrays()["cell_centroid"]
    return mesh, p, H.state_from_dvp(2, 1 + (x[0] < 0.5), 0.1 * x, 1 + (x[0] < 0.5))


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("calls_before", [0, 1, 2])
@pytest.mark.parametrize("call", ["step", "run", "step on another state"])
def test_step_and_run_are_refused(cuda, precision, calls_before, call):
    mesh, p, s0 = _setup(precision)
    solver = H.Solver(H.DeviceMesh(mesh), p)
    dstate, other = (H.DeviceState(2, mesh.num_cells) for _ in range(2))
    stream = cuda.cuda.Stream()
    dstate.upload(s0, stream)
    other.upload(s0, stream)
    solver.reset(0.0, stream)
    for _ in range(calls_before):
        solver.step(dstate, stream)
    x = cuda.zeros(4, device="cuda")
    cuda.cuda.synchronize()
    graph = cuda.cuda.CUDAGraph()
    with cuda.cuda.stream(stream):
        graph.capture_begin()
        x += 1
        with pytest.raises(H.FvhError) as e:
            if call == "run":
                solver.run(dstate, 3, stream=stream)
            else:
                solver.step(dstate if call == "step" else other, stream)
        x += 1
        graph.capture_end()
    assert e.value.code == H.ERR_CUDA
    graph.replay()
    cuda.cuda.synchronize()
    assert x.tolist() == [2.0] * 4
    # the solver goes on as if nothing had been asked
    for _ in range(2):
        solver.step(dstate, stream)
    out, t = dstate.download(stream), solver.soln_time(stream)
    fresh = H.Solver(H.DeviceMesh(mesh), p)
    other.upload(s0, stream)
    fresh.reset(0.0, stream)
    for _ in range(calls_before + 2):
        fresh.step(other, stream)
    assert fresh.soln_time(stream) == t and np.array_equal(other.download(stream), out)


def test_tasks_are_captured(cuda, oracle_lib):
    mesh, p, s0 = _setup("fp64")
    nc, nf = mesh.num_cells, mesh.num_faces
    dmesh = H.DeviceMesh(mesh)
    ds = cuda.tensor(s0, device="cuda")
    dg = cuda.zeros((U.grad_rows(2), nc), dtype=cuda.float64, device="cuda")
    df = cuda.zeros((4, nf), dtype=cuda.float64, device="cuda")
    scal = cuda.zeros(2, dtype=cuda.float64, device="cuda")
    nb = H.lib().fvh_time_step_workspace_bytes(nc)
    ws = cuda.zeros(nb // 8 + 1, dtype=cuda.float64, device="cuda")
    status = cuda.full((1,), -1, dtype=cuda.int64, device="cuda")
    sv, gv, fv = U.device_state_view(ds, 2), U.device_gradient_view(dg, 2), U.device_flux_view(df, 2)
    cuda.cuda.synchronize()
    stream, graph, L = cuda.cuda.Stream(), cuda.cuda.CUDAGraph(), H.lib()
    sh = H.stream_handle(stream)
    with cuda.cuda.stream(stream):
        graph.capture_begin()
        H.check(L.fvh_evaluate_time_step(C.byref(dmesh.view), C.byref(sv), C.byref(p), scal.data_ptr(),
                                         scal.data_ptr() + 8, ws.data_ptr(), nb, status.data_ptr(), sh))
        for _ in range(2):
            H.check(L.fvh_evaluate_gradients(C.byref(dmesh.view), C.byref(sv), C.byref(gv), C.byref(p), sh))
            H.check(L.fvh_evaluate_fluxes(C.byref(dmesh.view), C.byref(sv), C.byref(gv), C.byref(fv),
                                          C.byref(p), sh))
            H.check(L.fvh_apply_update(C.byref(dmesh.view), C.byref(p), scal.data_ptr() + 8, 0.5,
                                       C.byref(fv), C.byref(sv), scal.data_ptr(), status.data_ptr(), sh))
        graph.capture_end()
    for _ in range(3):
        graph.replay()
    cuda.cuda.synchronize()
    assert int(status.item()) == -1
    state = s0.copy()
    st, t, _ = U.oracle_run(oracle_lib, mesh, state, p, 3)
    assert st == 0 and scal[0].item() == t and np.array_equal(ds.cpu().numpy(), state)
