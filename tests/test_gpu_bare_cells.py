"""Cells with empty lists, which a caller's own mesh view may hold: one without
faces, neighbours and vertices (it keeps its state), and one without vertices (no
vertex limits its gradients).  They stand last, so that nothing follows their place
in the lists."""
import ctypes as C

import numpy as np
import pytest

import flecsale_gb300.hydro as H
from tests import _util as U

pytestmark = pytest.mark.gpu


class Mesh:
    """A mesh view on numpy arrays (mesh.view, for the oracle) and on copies of them
    in device memory (mesh.device.view)."""

    def __init__(self, torch, dim, arrays):
        self.dim, self.arrays = dim, {k: np.ascontiguousarray(v) for k, v in arrays.items()}
        self.num_cells = len(arrays["cell_volume"])
        self.num_faces = len(arrays["face_area"])
        self.view = self._view(lambda a: a.ctypes.data)
        self._on_device = {}
        self.device = type("Device", (), {})()
        self.device.view = self._view(lambda a: self._copy(torch, a))

    def _copy(self, torch, a):
        t = torch.from_numpy(a.copy()).cuda()
        self._on_device[len(self._on_device)] = t
        return t.data_ptr()

    def _view(self, at):
        v = H.MeshView()
        v.dim, v.num_cells, v.num_faces = self.dim, self.num_cells, self.num_faces
        v.num_vertices = self.arrays["vertex_coord"].shape[1]
        for k, a in self.arrays.items():
            if k in ("cell_centroid", "face_centroid", "face_normal", "vertex_coord"):
                for d in range(self.dim):
                    getattr(v, k)[d] = C.cast(C.c_void_p(at(a[d])), C.POINTER(C.c_double))
            else:
                ct = C.c_int32 if a.dtype == np.int32 else C.c_double
                setattr(v, k, C.cast(C.c_void_p(at(a)), C.POINTER(ct)))
        return v


def _state(dim, x):
    w = 0.05 * np.sin(2 * np.pi * (2 * x + np.arange(dim)[:, None]))
    return H.state_from_dvp(dim, 1 + w.sum(0) + (x[0] < 0.5), w, 1 + 1.4 * w.sum(0) + (x[0] < 0.5))


def _with_lone_cell(torch, dim, n):
    """A box mesh and the same with one more cell, whose lists are empty."""
    box = H.HostMesh.box(dim, n, [0] * dim, [1] * dim, 0.15, 5)
    a = dict(box.arrays())
    for k in ("cell_face_offsets", "cell_nbr_offsets", "cell_vertex_offsets"):
        a[k] = np.append(a[k], a[k][-1])
    a["cell_volume"] = np.append(a["cell_volume"], a["cell_volume"][-1])
    a["cell_centroid"] = np.concatenate([a["cell_centroid"], np.full((dim, 1), 0.5)], 1)
    return box, Mesh(torch, dim, a)


def _run(mesh, p, state, schedule=None):
    dstate = H.DeviceState(p.dim, state.shape[1])
    solver = H.Solver(mesh, p)
    if schedule is not None:
        solver.set_shape(128, 1, schedule)
    dstate.upload(state)
    solver.reset(0.0)
    assert solver.run(dstate, 3) == 3
    return dstate.download(), solver.soln_time()


@pytest.mark.parametrize("dim,n", [(2, (9, 7)), (2, (160, 126)), (3, (5, 4, 3)), (3, (29, 28, 27))])
@pytest.mark.parametrize("order", [1, 2])
def test_lone_cell_fp64(cuda, oracle_lib, dim, n, order):
    _, mesh = _with_lone_cell(cuda, dim, n)
    p = H.make_params(dim, flux="hllc", order=order, cfl=0.3, final_time=1e9)
    state = _state(dim, mesh.arrays["cell_centroid"])
    out, t = _run(mesh.device, p, state)
    st, want_t, _ = U.oracle_run(oracle_lib, mesh, state, p, 3)
    assert st == 0 and t == want_t and np.array_equal(out, state)


@pytest.mark.parametrize("dim,n", [(2, (9, 7)), (2, (60, 50)), (3, (5, 4, 3)), (3, (12, 11, 10))])
@pytest.mark.parametrize("schedule", [0, 1, 2, 4, 5])  # (4: the staged gradients, 2D)
def test_lone_cell_mixed(cuda, dim, n, schedule):
    if dim == 3 and schedule >= 4:
        return
    box, mesh = _with_lone_cell(cuda, dim, n)
    p = H.make_params(dim, flux="hllc", cfl=0.3, final_time=1e9, precision="mixed")
    state = _state(dim, mesh.arrays["cell_centroid"])
    out, t = _run(mesh.device, p, state, schedule)
    want, want_t = _run(H.DeviceMesh(box), p, state[:, :-1].copy(), schedule)
    assert t == want_t and np.array_equal(out[:, :-1], want)
    # density, velocity and energy stay; the rest is closed from them
    assert np.array_equal(out[:2 + dim, -1], state[:2 + dim, -1])


@pytest.mark.parametrize("dim,n", [(2, (24, 17)), (2, (131, 127)), (2, (513, 512)),
                                   (3, (27, 26, 25)), (3, (46, 45, 46))])
def test_cell_without_vertices(cuda, oracle_lib, dim, n):
    """Beside large values the limiter's FP32 bounds do not decide, so it looks for
    the vertices that do."""
    a = dict(H.HostMesh.box(dim, n, [0] * dim, [1] * dim, 0.15, 5).arrays())
    a["cell_vertex_offsets"] = a["cell_vertex_offsets"].copy()
    a["cell_vertex_offsets"][-1] = a["cell_vertex_offsets"][-2]
    a["cell_vertices"] = a["cell_vertices"][:a["cell_vertex_offsets"][-1]]
    mesh = Mesh(cuda, dim, a)
    nc = mesh.num_cells
    state = _state(dim, mesh.arrays["cell_centroid"])
    state[:, -1] += 1.0  # above all neighbours: no room over it
    state[(0, 1 + dim, 2 + dim, 4 + dim), :] += 1e7
    p = H.make_params(dim, flux="rusanov", cfl=0.3, final_time=1e9)
    ds = cuda.tensor(state, device="cuda")
    dg = cuda.zeros((U.grad_rows(dim), nc), dtype=cuda.float64, device="cuda")
    sv, gv = U.device_state_view(ds, dim), U.device_gradient_view(dg, dim)
    cuda.cuda.synchronize()
    H.check(H.lib().fvh_evaluate_gradients(C.byref(mesh.device.view), C.byref(sv), C.byref(gv),
                                           C.byref(p), None))
    cuda.cuda.synchronize()
    want = U.oracle_gradients(oracle_lib, mesh, state, p)
    assert np.isfinite(want).all() and np.array_equal(dg.cpu().numpy(), want)
    dstate = H.DeviceState(dim, nc)
    solver = H.Solver(mesh.device, p)
    dstate.upload(state)
    solver.reset(0.0)
    solver.step(dstate)
    out = dstate.download()
    assert U.oracle_run(oracle_lib, mesh, state, p, 1)[0] == 0
    assert solver.status()[0] == 0 and np.array_equal(out, state)
