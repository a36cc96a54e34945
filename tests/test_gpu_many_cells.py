"""The FP64 kernels for many cells against the oracle, bit for bit, where they are
hard: the limiter's edge fields, operands beyond the integer pipes' range and every
combination of options, on meshes above the sizes up to which the few-cells kernels
serve (6,144 cells for gradients with tables and 16,384 without, 10,000 faces,
20,000 cells for the update)."""
import ctypes as C

import numpy as np
import pytest

import flecsale_gb300.hydro as H
from tests import _util as U
from tests import test_gpu_limiter as limiter
from tests import test_gpu_parity as parity

pytestmark = pytest.mark.gpu

# one variable a thread with tables, two a thread with tables
MESHES = {
    "131x127": lambda j: H.HostMesh.box(2, (131, 127), [0, 0], [1, 1], 0.2 * j, 3),
    "513x512": lambda j: H.HostMesh.box(2, (513, 512), [0, 0], [1, 1], 0.2 * j, 3),
    "27x26x25": lambda j: H.HostMesh.box(3, (27, 26, 25), [0] * 3, [1] * 3, 0.15 * j, 3),
    "46x45x46": lambda j: H.HostMesh.box(3, (46, 45, 46), [0] * 3, [1] * 3, 0.15 * j, 3),
}


def _step_bitwise(oracle_lib, mesh, dmesh, p, state, nsteps=1):
    """A run on the solver's tables; what it started from is lost."""
    dstate = H.DeviceState(mesh.dim, mesh.num_cells)
    solver = H.Solver(dmesh, p)
    dstate.upload(state)
    solver.reset(0.0)
    try:
        solver.run(dstate, nsteps)
        code = 0
    except H.FvhError as e:
        code = e.code
    out = dstate.download()
    st, t, _ = U.oracle_run(oracle_lib, mesh, state, p, nsteps)
    assert code == st
    if st == 0:  # (the oracle stops half-way where the state goes negative)
        assert solver.soln_time() == t and np.array_equal(out, state, equal_nan=True)
    return st


def _solver_gradients(torch, solver, dim, nc):
    """The solver's own gradient planes, which stand one after another."""
    at = C.cast(solver.gradients.density[0], C.c_void_p).value

    class Planes:
        __cuda_array_interface__ = {"shape": (U.grad_rows(dim), nc), "typestr": "<f8",
                                    "data": (at, False), "version": 2}
    return torch.as_tensor(Planes(), device="cuda").cpu().numpy()


@pytest.mark.parametrize("jitter", [0, 1])
@pytest.mark.parametrize("name", list(MESHES))
@pytest.mark.parametrize("kind", limiter.KINDS)
def test_limiter_bitwise(cuda, oracle_lib, name, jitter, kind):
    mesh = MESHES[name](jitter)
    dim = mesh.dim
    state = limiter._state(kind, mesh, np.random.default_rng(100 + limiter.KINDS.index(kind)))
    # kinetic energies below the internal ones, so that closing the state keeps it positive
    state[1:1 + dim] *= {"huge": 1e-14, "mixed": 2.0 ** -220}.get(kind, 1)
    dmesh = H.DeviceMesh(mesh)
    # the task, without tables
    p = H.make_params(dim, flux="hllc", cfl=0.3, final_time=1e30)
    ds = cuda.tensor(state, device="cuda")
    dg = cuda.zeros((U.grad_rows(dim), mesh.num_cells), dtype=cuda.float64, device="cuda")
    sv, gv = U.device_state_view(ds, dim), U.device_gradient_view(dg, dim)
    cuda.cuda.synchronize()
    H.check(H.lib().fvh_evaluate_gradients(C.byref(dmesh.view), C.byref(sv), C.byref(gv),
                                           C.byref(p), None))
    cuda.cuda.synchronize()
    want = U.oracle_gradients(oracle_lib, mesh, state, p)
    assert np.array_equal(dg.cpu().numpy(), want, equal_nan=True)
    # the solver, with its tables: at the final time dt is 0, each update only closes
    # the state, and the gradients left behind are the corrector's
    p0 = H.make_params(dim, flux="rusanov", cfl=0.3, final_time=0.0)
    after = state.copy()
    finite = True
    for stage in range(2):
        want = U.oracle_gradients(oracle_lib, mesh, after, p0)
        f = U.oracle_fluxes(oracle_lib, mesh, after, want, p0)
        finite = finite and np.isfinite(f).all()  # (p / d of a reconstructed d can overflow)
        assert U.oracle_update(oracle_lib, mesh, after, f, p0, 0.0, 0.5)[0] == 0
    if finite:
        dstate = H.DeviceState(dim, mesh.num_cells)
        solver = H.Solver(dmesh, p0)
        dstate.upload(state)
        solver.reset(0.0)
        solver.step(dstate)
        out = dstate.download()
        assert solver.status()[0] == 0
        assert np.array_equal(_solver_gradients(cuda, solver, dim, mesh.num_cells), want)
        assert np.array_equal(out, after)
    else:
        assert kind == "mixed"
    # a step forward, where the field stays positive in it
    _step_bitwise(oracle_lib, mesh, dmesh, p, state)


# 20,691 cells and 41,674 faces; 21,924 cells
@pytest.mark.parametrize("case", parity.CASES, ids=lambda c: "-".join(str(x) for x in c))
def test_tasks_bitwise(cuda, case):
    n = (171, 121) if case[0] == 2 else (29, 28, 27)
    parity.test_tasks_bitwise(cuda, (case[0], n, *case[2:]))


@pytest.mark.parametrize("mesh", ["triangles", "mixed", "tetrahedra"])
@pytest.mark.parametrize("flux", ["hlle", "hllc", "rusanov"])
def test_unstructured_run_bitwise(cuda, oracle_lib, mesh, flux):
    m = {"triangles": lambda: U.tri_mesh((120, 90)), "mixed": lambda: U.tri_mesh((150, 121), 3),
         "tetrahedra": lambda: U.tet_mesh((16, 15, 15))}[mesh]()
    assert m.num_cells > 20000
    p = H.make_params(m.dim, flux=flux, cfl=0.3, final_time=1e9, swap=False)
    x = m.arrays()["cell_centroid"]
    w = 0.05 * np.sin(2 * np.pi * (2 * x + np.arange(m.dim)[:, None]))
    state = H.state_from_dvp(m.dim, 1 + w.sum(0) + (x[0] < 0.5), w, 1 + 1.4 * w.sum(0) + (x[0] < 0.5))
    assert _step_bitwise(oracle_lib, m, H.DeviceMesh(m), p, state, 3) == 0


@pytest.mark.parametrize("name", ["151x139", "513x512", "46x45x46"])
@pytest.mark.parametrize("flux", ["hlle", "hllc", "rusanov"])
@pytest.mark.parametrize("limited", [True, False])
@pytest.mark.parametrize("boundary,swap", [("wall", True), ("outflow", False)])
def test_options_run_bitwise(cuda, oracle_lib, name, flux, limited, boundary, swap):
    mesh = H.HostMesh.box(2, (151, 139), [0, 0], [1, 1], 0.2, 3) if name == "151x139" \
        else MESHES[name](1)
    p = H.make_params(mesh.dim, flux=flux, limiter="barth_jespersen" if limited else "none",
                      boundary=boundary, swap=swap, cfl=0.3, final_time=1e9)
    x = mesh.arrays()["cell_centroid"]
    w = 0.02 * np.sin(2 * np.pi * (2 * x + np.arange(mesh.dim)[:, None]))
    # velocities on both sides of the sound speed: every side of the Riemann fluxes
    v = np.zeros_like(w)
    v[0] = 2.5 * np.sin(2 * np.pi * x[1])
    state = H.state_from_dvp(mesh.dim, 1.5 + w.sum(0), v + w, 2 + 1.4 * w.sum(0))
    assert _step_bitwise(oracle_lib, mesh, H.DeviceMesh(mesh), p, state, 3) == 0


@pytest.mark.parametrize("dim,flux,scale", [(2, "hllc", 1e-170), (2, "hllc", 2.0 ** -495),
                                            (2, "hlle", 1e170), (3, "rusanov", 1e-170),
                                            (3, "hlle", 2.0 ** -495)])
def test_extreme_magnitudes_take_the_fp64_redo_bitwise(cuda, oracle_lib, dim, flux, scale):
    """Density and pressure scaled so that operands leave the 2^+-500 range of the
    integer-pipe arithmetic: gradients, face fluxes and updates are evaluated again
    with the FP64 instructions (nearly all, or those of a few cells)."""
    mesh = H.HostMesh.box(dim, (171, 121) if dim == 2 else (29, 28, 27), [0] * dim, [1] * dim,
                          0.15, 3)
    p = H.make_params(dim, flux=flux, cfl=0.4, swap=False, boundary="outflow")
    state = H.initial_state("four_quadrant" if dim == 2 else "inner_cube", mesh, p)
    for row in (0, dim + 2):  # density, pressure
        state[row] *= scale
    assert _step_bitwise(oracle_lib, mesh, H.DeviceMesh(mesh), p, state, 3) == 0


@pytest.mark.parametrize("n", [(151, 139), (513, 512)])
def test_offsets_beyond_the_integer_pipe_range(cuda, oracle_lib, n):
    """x_nbr - x_c below 2^-500: such a mesh computes its offsets on the fly."""
    mesh = H.HostMesh.box(2, n, [0, 0], [1e-155, 1e100], 0.0, 3)
    p = H.make_params(2, flux="hllc", cfl=0.3, final_time=1e30)
    state = limiter._state("smooth", mesh, np.random.default_rng(1))
    assert _step_bitwise(oracle_lib, mesh, H.DeviceMesh(mesh), p, state) == 0
