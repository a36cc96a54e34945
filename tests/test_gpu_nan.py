"""States with NaNs: a run's steps, which carry the CFL maximum from one to the
next, give the bits, the time and the status of single steps, which fold the cells
anew.  (A maximum in the reference's order, a < b ? b : a, keeps or drops a NaN by
where it stands.)"""
import numpy as np
import pytest

import flecsale_gb300.hydro as H

pytestmark = pytest.mark.gpu


def _steps(solver, dstate, s0, n, stream):
    dstate.upload(s0, stream)
    solver.reset(0.0, stream)
    for _ in range(n):
        solver.step(dstate, stream)
    return dstate.download(stream), solver.status(stream)


def _run(solver, dstate, s0, n, stream):
    dstate.upload(s0, stream)
    solver.reset(0.0, stream)
    try:
        assert solver.run(dstate, n, stream=stream) == n
        code = 0
    except H.FvhError as e:
        code = e.code
    out, status = dstate.download(stream), solver.status(stream)
    assert code == status[0]
    return out, status


def _same(a, b):
    assert np.array_equal(a[0], b[0], equal_nan=True)
    assert np.array_equal(a[1], b[1], equal_nan=True), (a[1], b[1])


@pytest.mark.parametrize("dim,n", [(2, (24, 17)), (2, (97, 90)), (2, (160, 126)), (2, (513, 512)),
                                   (3, (9, 8, 7)), (3, (27, 26, 25)), (3, (46, 45, 46))])
@pytest.mark.parametrize("order", [1, 2])
@pytest.mark.parametrize("where", ["first", "one", "some", "all"])
def test_run_equals_steps(cuda, dim, n, order, where):
    mesh = H.HostMesh.box(dim, n, [0] * dim, [1] * dim, 0.15, 5)
    nc = mesh.num_cells
    p = H.make_params(dim, flux="hllc", order=order, cfl=0.3, final_time=1e9)
    x = mesh.arrays()["cell_centroid"]
    s0 = H.state_from_dvp(dim, 1 + (x[0] < 0.5), 0.1 * x, 1 + (x[0] < 0.5))
    bad = {"first": [0], "one": [nc // 3], "all": np.arange(nc),
           "some": np.random.default_rng(3).choice(nc, nc // 50, replace=False)}[where]
    for plane in (1 + dim, 2 + dim, 4 + dim):  # e, p, a
        s0[plane][bad] = np.nan
    dmesh, dstate = H.DeviceMesh(mesh), H.DeviceState(dim, nc)
    solver = H.Solver(dmesh, p)
    stream = cuda.cuda.Stream()
    for steps in (2, 3, 12):  # (12: four steps a graph on small meshes)
        want = _steps(solver, dstate, s0, steps, stream)
        _same(_run(solver, dstate, s0, steps, stream), want)
    # finite again: nothing of the NaNs stays behind
    s0 = H.state_from_dvp(dim, 1 + (x[0] < 0.5), 0.1 * x, 1 + (x[0] < 0.5))
    want = _steps(solver, dstate, s0, 3, stream)
    assert want[1][0] == 0 and np.isfinite(want[0]).all()
    _same(_run(solver, dstate, s0, 3, stream), want)


@pytest.mark.parametrize("n", [(1, 1), (1, 2), (2, 1)])
def test_singular_least_squares(cuda, n):
    """Cells in a row: NaN gradients, and a NaN state from the first step on, which
    is reported when its time is no number."""
    mesh = H.HostMesh.box(2, n, [0, 0], [1, 1], 0.15, 5)
    p = H.make_params(2, flux="hllc", cfl=0.3, final_time=1e9)
    x = mesh.arrays()["cell_centroid"]
    s0 = H.state_from_dvp(2, 1 + x[0], 0.1 * x, 1 + x[0])
    dstate = H.DeviceState(2, mesh.num_cells)
    solver = H.Solver(H.DeviceMesh(mesh), p)
    stream = cuda.cuda.Stream()
    for steps in (1, 2, 3):
        want = _steps(solver, dstate, s0, steps, stream)
        _same(_run(solver, dstate, s0, steps, stream), want)
    assert want[1][0] == H.ERR_INFINITE_DT and np.isnan(want[1][1])
