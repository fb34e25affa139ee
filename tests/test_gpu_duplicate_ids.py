"""Particles that share ids (a caller's set, or 32-bit ids that wrapped):
every particle keeps a place of its own in the write pass, in cells that fit a
tile and in larger ones, and among equal keys the earlier particle goes first,
in the layout and in the count correction."""
import numpy as np
import pytest

from . import cases
from .test_gpu_parity import V_RTOL_FP64, assert_v_close, make
from .test_gpu_write_runs import BIG, COUNTS, _mesh

pytestmark = pytest.mark.gpu


def _case(maxpp, dt):
    m = _mesh((128, 64))
    # zero on the boundary: no particle leaves the mesh
    s = np.sin(np.pi * m.vertices[:, 0] / 2.0) * np.sin(np.pi * m.vertices[:, 1])
    V = np.zeros((2, m.n_dofs))
    V[:, m.cell_dofs.ravel()] = np.stack([s, 0.7 * s])[:, m.cells.ravel()]
    c = cases.Case("ids", m, V, 0.9 * V, (4, 4), maxpp, 2, dt)
    n_of = np.full(m.n_cells, 16)
    for k in range(4):
        b = 69 + 631 * k - BIG
        n_of[b:b + len(COUNTS)] = COUNTS
    rng = np.random.default_rng(4)
    cell = np.repeat(np.arange(m.n_cells), n_of)
    n = len(cell)
    xi = ((rng.integers(0, 4, (n, 2)) + rng.uniform(0.02, 0.98, (n, 2))) / 4).astype(np.float32).astype(np.float64)
    X = m.vertices[m.cells[cell]]
    x = X[:, 0] + xi * (X[:, -1] - X[:, 0])
    v = rng.normal(size=(n, 2)).astype(np.float32).astype(np.float64)
    return c, {"id": rng.integers(1, 6, n).astype(np.uint32), "cell": cell.astype(np.int32), "x": x, "xi": xi, "v": v}


def _rows(P, keys=("x", "xi", "v")):
    r = np.column_stack([P["id"].astype(np.float64), P["cell"].astype(np.float64)] + [P[k] for k in keys])
    return r[np.lexsort(r.T)]


@pytest.mark.parametrize("maxpp,steps", [(10 ** 6, 4), (2, 1)])
def test_fp64_equals_the_oracle(maxpp, steps):
    """Uploaded by cell, so the earlier particle is the same one for the
    oracle's stable order; new particles repeat live ids (next_id 0)."""
    c, P = _case(maxpp, 0.01)
    o, g = make(c, capacity=400000)
    for h in (o, g):
        h.set_particles(P, 0)
    assert np.array_equal(_rows(o.particles()), _rows(g.particles()))
    for _ in range(steps):
        Vo, Vg = o.step(c.V, c.Vold), g.step(c.V, c.Vold)
        assert np.array_equal(_rows(o.particles()), _rows(g.particles()))
        assert_v_close(Vo, Vg, V_RTOL_FP64)
        for k in ("n_particles", "removed", "seeded", "lost", "next_id"):
            assert o.stats()[k] == g.stats()[k], k
    g.close()


def test_fp32_keeps_every_particle():
    c, P = _case(10 ** 6, 0.0)
    o, g = make(c, capacity=400000, precision="fp32")
    for h in (o, g):
        h.set_particles(P, 0)
    for _ in range(2):
        Vo, Vg = o.step(c.V, c.V), g.step(c.V, c.V)
        assert np.array_equal(_rows(o.particles(), ("xi",)), _rows(g.particles(), ("xi",)))
        assert_v_close(Vo, Vg, 2e-6)  # as for the tiles' edges: under 32 roundings of 6e-8
    g.close()


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("seed", [0, 77])
def test_same_run_twice(precision, seed):
    c, P = _case(2, 0.01)
    runs = []
    for _ in range(2):
        _, g = make(c, precision=precision, capacity=400000, removal_seed=seed)
        g.set_particles(P, 0)
        V = [g.step(c.V, c.Vold) for _ in range(4)]
        Q = g.particles()
        runs.append([Q[k] for k in ("id", "cell", "xi", "v")] + V)
        g.close()
    for a, b in zip(*runs):
        assert np.array_equal(a, b, equal_nan=True)
