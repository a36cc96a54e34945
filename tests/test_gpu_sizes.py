"""FP64 runs on both sides of every size at which the kernels change form (few
cells or faces, one variable or two per thread), against the oracle bit for bit:
a run of three steps carries dt from each corrector to the next step."""
import ctypes as C

import numpy as np
import pytest

import flecsale_gb300.hydro as H
from tests import _util as U

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim,n,order", [
    (2, (1, 1), 2), (2, (9, 7), 1), (2, (70, 70), 1),         # 9,940 faces
    (2, (71, 70), 2),                                          # 10,081 faces
    (2, (96, 64), 2), (2, (97, 64), 2),                        # 6,144 and 6,208 cells
    (2, (160, 125), 2), (2, (160, 126), 1),                    # 20,000 and 20,160 cells
    (3, (16, 16, 24), 2), (3, (17, 19, 20), 2),                # 6,144 and 6,460 cells
    (3, (45, 32, 64), 2), (3, (46, 32, 64), 2),                # 92,160 and 94,208 cells
    (2, (512, 512), 2), (2, (513, 512), 2)])                   # 262,144 and 262,656 cells
def test_run_bitwise(cuda, oracle_lib, dim, n, order):
    mesh = H.HostMesh.box(dim, n, [0] * dim, [1] * dim, 0.15, 5)
    p = H.make_params(dim, flux="hllc" if dim == 2 else "rusanov", order=order, cfl=0.3,
                      final_time=1e9)
    x = mesh.arrays()["cell_centroid"]
    w = 0.05 * np.sin(2 * np.pi * (2 * x + np.arange(dim)[:, None]))
    state = H.state_from_dvp(dim, 1 + w.sum(0) + (x[0] < 0.5), w, 1 + 1.4 * w.sum(0) + (x[0] < 0.5))
    one = state.copy()
    st, t, _ = U.oracle_run(oracle_lib, mesh, state, p, 3)
    dmesh, dstate = H.DeviceMesh(mesh), H.DeviceState(dim, mesh.num_cells)
    solver = H.Solver(dmesh, p)
    stream = cuda.cuda.Stream()
    dstate.upload(one, stream)
    solver.reset(0.0, stream)
    if st != 0:  # (one cell has no neighbours: its least-squares system is singular)
        with pytest.raises(H.FvhError) as e:
            solver.run(dstate, 3, stream=stream)
        assert e.value.code == st
        return
    assert solver.run(dstate, 3, stream=stream) == 3
    out = dstate.download(stream)
    stream.synchronize()
    assert solver.soln_time(stream) == t and np.array_equal(out, state)
    # step by step (each step takes dt from the state), then a run again
    dstate.upload(one, stream)
    solver.reset(0.0, stream)
    for _ in range(2):
        solver.step(dstate, stream)
    solver.run(dstate, 1, stream=stream)
    again = dstate.download(stream)
    stream.synchronize()
    assert np.array_equal(again, state)


@pytest.mark.parametrize("steps", [1, 10])
def test_first_order_ignores_what_its_gradients_hold(cuda, oracle_lib, steps):
    """A first-order solver's gradients are zero in every run and step, also after
    the caller has filled them through the solver's own view."""
    mesh = H.HostMesh.box(2, (24, 17), [0, 0], [1, 1], 0.15, 5)
    p = H.make_params(2, flux="hlle", order=1, cfl=0.3, final_time=1e9)
    second = H.make_params(2, flux="hlle", order=2, cfl=0.3, final_time=1e9)
    x = mesh.arrays()["cell_centroid"]
    state = H.state_from_dvp(2, 1 + (x[0] < 0.5), 0.1 * x, 1 + (x[0] < 0.5))
    one = state.copy()
    U.oracle_run(oracle_lib, mesh, state, p, 2 * steps)
    dmesh, dstate = H.DeviceMesh(mesh), H.DeviceState(2, mesh.num_cells)
    solver = H.Solver(dmesh, p)
    stream = cuda.cuda.Stream()
    dstate.upload(one, stream)
    solver.reset(0.0, stream)
    for _ in range(2):
        H.check(H.lib().fvh_evaluate_gradients(C.byref(dmesh.view), C.byref(dstate.view),
                                               C.byref(solver.gradients), C.byref(second),
                                               C.c_void_p(stream.cuda_stream)))
        if steps == 1:
            solver.step(dstate, stream)
        else:
            solver.run(dstate, steps, stream=stream)
    out = dstate.download(stream)
    stream.synchronize()
    assert np.array_equal(out, state)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("legacy", [False, True])
def test_graphed_and_plain_launches_agree(cuda, precision, legacy):
    """Runs on two states in turn (launched as they are, or captured, by the number
    of steps) and twice on one (captured) give the bits of single steps."""
    mesh = H.HostMesh.box(2, (24, 17), [0, 0], [1, 1], 0.15, 5)
    p = H.make_params(2, flux="hllc", cfl=0.3, final_time=1e9, precision=precision)
    x = mesh.arrays()["cell_centroid"]
    one = H.state_from_dvp(2, 1 + (x[0] < 0.5), 0.1 * x, 1 + (x[0] < 0.5))
    dmesh = H.DeviceMesh(mesh)
    solver = H.Solver(dmesh, p)
    stream = None if legacy else cuda.cuda.Stream()
    want = {}
    states = [H.DeviceState(2, mesh.num_cells) for _ in range(2)]
    for n in (1, 9, 127, 128):
        states[0].upload(one, stream)
        solver.reset(0.0, stream)
        for _ in range(n):
            solver.step(states[0], stream)
        want[n] = states[0].download(stream)
        for s in (1, 1, 0, 1):
            states[s].upload(one, stream)
            solver.reset(0.0, stream)
            assert solver.run(states[s], n, stream=stream) == n
            assert np.array_equal(states[s].download(stream), want[n]), (n, s)
