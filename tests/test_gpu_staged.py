"""The staged 2D gradients (neighbour records brought to shared memory by bulk
copies) at the edges of their chunks, and beside other solvers, bit for bit
against the global-memory kernel."""
import numpy as np
import pytest

import flecsale_gb300.hydro as H
from tests import _util as U

pytestmark = pytest.mark.gpu
STAGED = 4


def _solver(n, limiter="barth_jespersen", tri=False):
    mesh = U.tri_mesh(n, 3) if tri else H.HostMesh.box(2, n, [0, 0], [1, 1], 0.2, 4)
    p = H.make_params(2, flux="hllc", cfl=0.4, precision="mixed", boundary="outflow",
                      limiter=limiter, final_time=10.0, swap=False)
    x = mesh.arrays()["cell_centroid"]
    w = 0.05 * np.sin(2 * np.pi * (2 * x + np.arange(2)[:, None]))
    s0 = H.state_from_dvp(2, 1 + w.sum(0) + (x[0] < 0.5), w, 1 + 1.4 * w.sum(0) + (x[0] < 0.5))
    return H.Solver(H.DeviceMesh(mesh), p), H.DeviceState(2, mesh.num_cells), s0


def _run(solver, dstate, s0, schedule):
    solver.set_shape(128, 1, schedule)
    dstate.upload(s0)
    solver.reset(0.0)
    try:  # (cells in a row have a singular least-squares system: no time step)
        solver.run(dstate, 4)
    except H.FvhError as e:
        return np.array([e.code])
    return dstate.download()


# one chunk and its remainders, two chunks and one cell, many chunks a block
@pytest.mark.parametrize("n", [(1, 2), (127, 1), (16, 8), (43, 3), (129, 2), (97, 61), (640, 480)])
@pytest.mark.parametrize("limiter", ["barth_jespersen", "none"])
def test_staged_equals_global(cuda, n, limiter):
    solver, dstate, s0 = _solver(n, limiter)
    want = _run(solver, dstate, s0, 1)
    try:
        got = _run(solver, dstate, s0, 1 | STAGED)
    except H.FvhError as e:  # a mesh whose chunks need more records than a byte numbers
        assert e.code == H.ERR_INVALID_ARGUMENT and n == (129, 2)
        return
    assert np.array_equal(got, want, equal_nan=True)
    assert want.ndim == 2 or min(n) < 3


def test_solvers_of_different_stage_sizes(cuda):
    """A solver created later, with smaller stages, leaves the first as it was."""
    big, dbig, sbig = _solver((97, 61))
    small, dsmall, ssmall = _solver((12, 9))
    want = _run(big, dbig, sbig, 0), _run(small, dsmall, ssmall, 0)
    assert np.array_equal(_run(big, dbig, sbig, STAGED), want[0])
    assert np.array_equal(_run(small, dsmall, ssmall, STAGED), want[1])
    assert np.array_equal(_run(big, dbig, sbig, STAGED), want[0])
