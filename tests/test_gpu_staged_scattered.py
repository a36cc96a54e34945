"""The staged 2D gradients on a mesh numbered at random: a chunk's records are then
nearly all runs of one, and its list is a third of its stage."""
import numpy as np
import pytest

import flecsale_gb300.hydro as H

pytestmark = pytest.mark.gpu
STAGED = 4


def _mesh(n, every, seed):
    """A jittered quad box, its quads joined in pairs on every `every`-th diagonal,
    cells and vertices numbered at random."""
    x = H.HostMesh.box(2, n, [0, 0], [1, 1], 0.2, seed).arrays()["vertex_coord"].T
    nx, ny = n
    w = nx + 1
    cells = []
    for j in range(ny):
        i = 0
        while i < nx:
            wide = 2 if (i - j) % every == 0 and i + 1 < nx else 1
            row = [j * w + i + t for t in range(wide + 1)]
            cells.append(row + [v + w for v in reversed(row)])
            i += wide
    rng = np.random.default_rng(seed)
    to = rng.permutation(len(x))
    coords = np.empty_like(x)
    coords[to] = x
    cells = [to[cells[c]] for c in rng.permutation(len(cells))]
    offsets = np.cumsum([0] + [len(c) for c in cells]).astype(np.int32)
    return H.HostMesh.from_cells(2, coords, offsets, np.concatenate(cells).astype(np.int32))


# 446 to 462 runs a chunk in stages of 17.8 to 18.6 KB
@pytest.mark.parametrize("n,every,seed", [((148, 36), 5, 1), ((160, 36), 5, 3), ((172, 36), 7, 2)])
@pytest.mark.parametrize("limiter", ["barth_jespersen", "none"])
def test_staged_equals_global(cuda, n, every, seed, limiter):
    mesh = _mesh(n, every, seed)
    p = H.make_params(2, flux="hllc", cfl=0.4, precision="mixed", limiter=limiter,
                      final_time=10.0, swap=False)
    x = mesh.arrays()["cell_centroid"]
    w = 0.05 * np.sin(2 * np.pi * (2 * x + np.arange(2)[:, None]))
    s0 = H.state_from_dvp(2, 1 + w.sum(0) + (x[0] < 0.5), w, 1 + 1.4 * w.sum(0) + (x[0] < 0.5))
    solver, dstate = H.Solver(H.DeviceMesh(mesh), p), H.DeviceState(2, mesh.num_cells)
    out = []
    for schedule in (1, 1 | STAGED):
        solver.set_shape(128, 1, schedule)
        dstate.upload(s0)
        solver.reset(0.0)
        assert solver.run(dstate, 4) == 4
        out.append(dstate.download())
    assert np.isfinite(out[0]).all() and np.array_equal(out[0], out[1])
