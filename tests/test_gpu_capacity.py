"""Steps that need more slots than params.capacity allows: the cells' ranges
end with the arrays, so the steps after one that did not fit stay in bounds,
the calls that synchronise report PFEM2GPU_ERR_CAPACITY, every slot holds a
particle of a cell or none, and a new particle set makes the handle whole."""
import numpy as np
import pytest

from pfem2dealii_b200 import _lib
from pfem2dealii_b200.handler import ParticleHandler

from . import cases
from .test_gpu_failures import code_of

pytestmark = pytest.mark.gpu


def _set(case, n_of, seed):
    m = case.mesh
    rng = np.random.default_rng(seed)
    cell = np.repeat(np.arange(m.n_cells), n_of)
    n = len(cell)
    xi = rng.uniform(0.05, 0.95, (n, m.dim)).astype(np.float32).astype(np.float64)
    X = m.vertices[m.cells[cell]]
    x = X[:, 0] + xi * (X[:, -1] - X[:, 0])
    v = rng.normal(size=xi.shape)
    return {"id": np.arange(1, n + 1, dtype=np.uint32), "cell": cell.astype(np.int32), "x": x, "xi": xi, "v": v}, n


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("which,dense", [
    (lambda: cases.channel(16, 4, dt=0.05), ()),
    (lambda: cases.channel(64, 64, q=(2, 2), maxpp=3, dt=0.01), ()),
    # cells beyond a tile, one of them the last to fit and one beyond
    (lambda: cases.channel(16, 4, maxpp=60, dt=0.05), (3, 40, 61, 62, 63)),
    (lambda: cases.duct(24, 6, 6, q=(2, 2, 2), maxpp=60, dt=0.05), (5, 700, 860, 863)),
])
def test_steps_beyond_the_capacity(which, dense, precision):
    import torch

    c = which()
    npart = int(np.prod(c.q))
    n_of = np.full(c.mesh.n_cells, max(1, npart // 2))
    n_of[list(dense)] = 900
    P, n = _set(c, n_of, 1)
    # half the parts are empty: the first step's new particles do not fit
    g = ParticleHandler(c.mesh.dim, cases.params(c, capacity=n + 5), precision)
    g.initialize_maps(c.mesh)
    g.set_particles(P, n)
    dV = torch.from_numpy(np.ascontiguousarray(c.V)).cuda()
    dVold = torch.from_numpy(np.ascontiguousarray(c.Vold)).cuda()
    out = torch.empty_like(dV)
    for _ in range(4):
        g.step_device(dV, dVold, out)
    assert code_of(g.particles) == _lib.ERR_CAPACITY and g.stats()["error_flags"] == 1
    for _ in range(4):
        g.step_device(dV, dVold, out)
    assert code_of(g.particles) == _lib.ERR_CAPACITY and g.stats()["error_flags"] == 1
    # a set that fits: the handle is as a new one
    fit = np.zeros(c.mesh.n_cells, int)
    fit[: c.mesh.n_cells // 4] = max(1, npart // 2)
    Q, k = _set(c, fit, 2)
    h = ParticleHandler(c.mesh.dim, cases.params(c, capacity=n + 5), precision)
    h.initialize_maps(c.mesh)
    runs = []
    for p in (g, h):
        p.set_particles(Q, k)
        V = [p.step(c.V, c.Vold) for _ in range(2)]
        R = p.particles()
        runs.append([R[key] for key in ("id", "cell", "xi", "v")] + V)
        p.close()
    for a, b in zip(*runs):
        assert np.array_equal(a, b, equal_nan=True)
