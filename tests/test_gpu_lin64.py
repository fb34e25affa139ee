"""The FP64 form on hex meshes whose inverse maps are decided from their
affine guess (locate_lin64): sub-steps that end on a face, within 1e-9 of it
on either side (mapped in full by the search kernel) and just beyond that,
chunks of particles over more cells than one stage holds, far moves and
meshes far from the origin, where the rounding bound decides per mesh.  Bit
for bit the oracle's particles and counters."""
import numpy as np
import pytest

from oracle.oracle import forward_map
from pfem2dealii_b200 import mesh as M

from . import cases
from .test_gpu_parity import STAT_KEYS, assert_same_particles, make

pytestmark = pytest.mark.gpu

OFFSETS = [0.0, 1e-16, 1e-15, 1e-13, 1e-12, 1e-11, 1e-10, 9e-10, 1.1e-9, 1e-8, 1e-6, 0.3, 0.6]


@pytest.mark.parametrize("origin,size,rk2,dt", [
    ((0.0, 0.0, 0.0), (8.0, 1.0, 1.0), 0, 0.25),
    ((0.0, 0.0, 0.0), (8.0, 1.0, 1.0), 1, 0.25),
    ((0.3, -7.7, 1e3), (1.7, 0.9, 0.3), 0, 0.01),   # |x| / h beyond the bound: Newton
    ((0.0, 0.0, 0.0), (8.0, 1.0, 1.0), 0, 3.0),     # most particles leave the vertex patch
])
def test_fp64_points_at_faces_bit_exact(origin, size, rk2, dt):
    m = M.hyper_rectangle(origin, tuple(o + s for o, s in zip(origin, size)), (8, 3, 2))
    rng = np.random.default_rng(1)
    V = rng.uniform(-0.4, 0.4, (3, m.n_dofs))
    V[:, : m.n_dofs // 2] = np.round(V[:, : m.n_dofs // 2] * 8) / 8
    c = cases.Case("faces", m, V, 0.5 * V, (2, 2, 2), 2, 2, dt)
    o, g = make(c, oracle_kw={"integrator": rk2}, capacity=20000, integrator=rk2)
    P = {k: [] for k in ("cell", "xi")}
    for cell in range(m.n_cells):
        if cell % 3 == 1:
            continue  # chunks that span many cells, some of them empty
        for off in OFFSETS:
            for s in (-1, 1):
                xi = rng.uniform(0.05, 0.95, 3)
                d = rng.integers(0, 3)
                xi[d] = np.clip((s > 0) - s * off, 0.0, 1.0)  # at a face, the offset inside
                P["cell"].append(cell)
                P["xi"].append(xi)
    n = len(P["cell"])
    xi = np.array(P["xi"])
    cell = np.array(P["cell"], np.int32)
    x = np.array([forward_map(m.vertices[m.cells[k]], z) for k, z in zip(cell, xi)])
    P = {"id": np.arange(1, n + 1, dtype=np.uint32), "cell": cell, "x": x, "xi": xi, "v": rng.normal(size=xi.shape)}
    o.set_particles(P, n)
    g.set_particles(P, n)
    for _ in range(4):
        # a velocity that carries the particles at faces by the offsets' sizes
        V = c.V * 10.0 ** rng.uniform(-13, 0)
        o.step(V, c.Vold)
        g.step(V, c.Vold)
        assert_same_particles(o.particles(), g.particles())
        so, sg = o.stats(), g.stats()
        for k in STAT_KEYS:
            assert so[k] == sg[k], k


def test_fp64_sparse_cells_bit_exact():
    """One particle in every fourth cell: an advect chunk spans more cells
    than its stage holds."""
    c = cases.duct(24, 12, 12, q=(1, 1, 1), S=2, dt=0.2)
    m = c.mesh
    cell = np.arange(0, m.n_cells, 4, dtype=np.int32)
    xi = np.random.default_rng(2).uniform(0, 1, (len(cell), 3))
    x = np.array([forward_map(m.vertices[m.cells[k]], z) for k, z in zip(cell, xi)])
    P = {"id": np.arange(1, len(cell) + 1, dtype=np.uint32), "cell": cell, "x": x, "xi": xi, "v": np.zeros_like(xi)}
    o, g = make(c)
    o.set_particles(P, len(cell))
    g.set_particles(P, len(cell))
    for _ in range(3):
        o.step(c.V, c.Vold)
        g.step(c.V, c.Vold)
        assert_same_particles(o.particles(), g.particles())
        assert o.stats()["searched"] == g.stats()["searched"]
