"""The 2D inverse map where the closed form decides that a point lies outside
its quad (mild_quad64): the rule's claim against the oracle's Newton on the
CPU, and both forms' trajectories over quads on both sides of the rule, with
particles that end at, just beside and up to half a cell beyond a face."""
import numpy as np
import pytest

from oracle.oracle import forward_map, inverse_map
from pfem2dealii_b200 import mesh as M

from . import cases
from .test_gpu_parity import STAT_KEYS, assert_same_particles, make


def _mild(X):
    A = np.stack([(X[1] - X[0] + X[3] - X[2]) / 2, (X[2] - X[0] + X[3] - X[1]) / 2], 1)
    Ai = np.linalg.inv(A)
    g = X[3] - X[1] - X[2] + X[0]
    return (np.abs(Ai @ g).sum() <= 0.1 and np.abs(X).max() * np.abs(Ai).sum(1).max() <= 1600.0
            and np.linalg.det(A) > 0.0)


def test_newton_converges_to_the_nearby_root_in_mild_quads():
    """Points 1e-6 to a quarter cell outside a mild quad: the oracle's map
    succeeds and gives the point they were made from.  The images are exact
    to 4 u xm, so the solution to 4 u xm |A^-1| x 1.2 < 1e-12; Newton's end
    test adds 1e-11."""
    rng = np.random.default_rng(5)
    n = 0
    while n < 20000:
        h = 10.0 ** rng.uniform(-4, 2)
        A = rng.normal(size=(2, 2)) * [1.0, 10.0 ** rng.uniform(-1.5, 1.5)]
        g = A @ rng.dirichlet([1, 1]) * rng.uniform(-0.1, 0.1)
        o = rng.uniform(-1, 1, 2) * 10.0 ** rng.uniform(-2, 3)
        X = np.array([o + h * (A @ [i & 1, i >> 1] + (g if i == 3 else 0.0)) for i in range(4)])
        if np.linalg.det(A) <= 0.0 or not _mild(X):
            continue
        n += 1
        xi = rng.uniform(-0.25, 1.25, 2)
        d = rng.integers(2)
        off = 10.0 ** rng.uniform(-6, np.log10(0.25))
        xi[d] = -off if rng.integers(2) else 1.0 + off
        got = inverse_map(X, forward_map(X, xi))
        assert got is not None
        assert np.abs(got - xi).max() <= 2e-11
        assert not np.all((got >= 0.0) & (got <= 1.0))


OFFSETS = [0.0, 1e-13, 1e-12, 1e-11, 1e-9, 5e-7, 1.5e-6, 1e-4, 0.2, 0.3]


@pytest.mark.gpu
@pytest.mark.parametrize("amplitude,origin,size", [
    (0.02, (0.0, 0.0), (4.0, 1.0)),       # every quad mild
    (0.06, (-3.0, 1.0), (1e-3, 2e-3)),    # |x| / h beyond the bound: none mild
    (0.06, (0.0, 0.0), (2.0, 2.0)),       # two in three mild
    (0.30, (0.0, 0.0), (1.0, 1.0)),       # hardly a mild one
])
def test_fp64_quads_bit_exact(amplitude, origin, size):
    nx, ny = 9, 7
    m = M.hyper_rectangle(origin, tuple(o + s for o, s in zip(origin, size)), (nx, ny))
    rng = np.random.default_rng(3)
    h = np.array(size) / (nx, ny)
    lo, hi = np.array(origin), np.array(origin) + size
    inner = np.all((m.vertices > lo + h / 2) & (m.vertices < hi - h / 2), axis=1)
    m.vertices[inner] += rng.uniform(-amplitude, amplitude, (inner.sum(), 2)) * h
    share = np.mean([_mild(m.vertices[k]) for k in m.cells])
    assert share == 1.0 if amplitude == 0.02 else share < 1.0
    # a uniform velocity of some cell sizes a step: particles leave along every face
    V = np.ones((2, m.n_dofs)) * h[:, None] * [[0.31], [-0.17]]
    c = cases.Case("quads", m, V, 0.5 * V, (2, 2), 3, 2, 1.0)
    o, g = make(c, capacity=40000)
    P = {"cell": [], "xi": []}
    for cell in range(m.n_cells):
        for off in OFFSETS:
            for s in (-1, 1):
                xi = rng.uniform(0.02, 0.98, 2)
                d = rng.integers(0, 2)
                xi[d] = np.clip((s > 0) - s * off, 0.0, 1.0)
                P["cell"].append(cell)
                P["xi"].append(xi)
    n = len(P["cell"])
    cell, xi = np.array(P["cell"], np.int32), np.array(P["xi"])
    x = np.array([forward_map(m.vertices[m.cells[k]], z) for k, z in zip(cell, xi)])
    P = {"id": np.arange(1, n + 1, dtype=np.uint32), "cell": cell, "x": x, "xi": xi, "v": rng.normal(size=xi.shape)}
    o.set_particles(P, n)
    g.set_particles(P, n)
    for scale in (1.0, 1e-5, 1e-10, 1.0, 2.5):
        Vs = V * scale * np.where(rng.integers(2, size=(2, 1)), 1.0, -1.0)
        o.step(Vs, c.Vold)
        g.step(Vs, c.Vold)
        assert_same_particles(o.particles(), g.particles())
        so, sg = o.stats(), g.stats()
        for k in STAT_KEYS:
            assert so[k] == sg[k], k
