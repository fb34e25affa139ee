"""The write pass's tiles of several cells, which need more cells than the
grid has blocks: tiles that overflow and are worked through in runs, a cell
beyond a tile first, inside and last in its tile, and blocks whose tiles are
such cells alone, drawn one after the other.  A uniform velocity moves every
particle by the same part of a cell, and no sub-step ends near a face or a
part boundary, so both forms take the oracle's decisions: ids, cells and
counters are equal in both, the FP64 form's particles bit for bit."""
import numpy as np
import pytest

from pfem2dealii_b200 import mesh as M

from . import cases
from .test_gpu_parity import V_RTOL_FP64, assert_same_particles, assert_v_close, by_id, make

pytestmark = pytest.mark.gpu

# particles of consecutive cells, the 700 beyond any tile in their middle
COUNTS = [0, 1, 31, 33, 479, 481, 0, 250, 250, 250, 700, 5, 511, 513, 0, 64, 97, 640, 641, 32]
BIG = COUNTS.index(700)
SUB = np.array([0.185, 0.115, 0.085])  # cells a sub-step, S = 2
STEPS = 3


def _start(m, shape, q, n_of, rng):
    """n_of[c] particles in cell c: FP32-exact reference coordinates that stay
    2e-3 of a part away from every face and part boundary at all sub-steps."""
    dim = m.dim
    cell = np.repeat(np.arange(m.n_cells), n_of)
    n = len(cell)
    xi = np.empty((n, dim))
    for d in range(dim):
        ok = np.zeros(n, bool)
        while not ok.all():
            t = rng.uniform(0.01, 0.99, n).astype(np.float32).astype(np.float64)
            f = q[d] * (t[:, None] + SUB[d] * np.arange(2 * STEPS + 1))
            good = (np.abs(f - np.round(f)) > 2e-3).all(1) & ~ok
            xi[good, d] = t[good]
            ok |= good
    X = m.vertices[m.cells[cell]]
    x = X[:, 0] + xi * (X[:, -1] - X[:, 0])
    v = rng.normal(size=xi.shape).astype(np.float32).astype(np.float64)
    return {"id": (rng.permutation(n) + 1).astype(np.uint32), "cell": cell.astype(np.int32), "x": x, "xi": xi, "v": v}, n


def _mesh(shape):
    # cells of 1/64: their vertices and every whole displacement are exact
    return M.hyper_rectangle((0.0,) * len(shape), tuple(k / 64.0 for k in shape), shape)


def _run(shape, q, maxpp, n_of, precision):
    m = _mesh(shape)
    rng = np.random.default_rng(11)
    V = np.repeat(2.0 * SUB[:m.dim, None] / 64.0, m.n_dofs, axis=1)
    c = cases.Case("runs", m, V, V, q, maxpp, 2, 1.0)
    P, n = _start(m, shape, q, n_of, rng)
    o, g = make(c, precision=precision, capacity=4 * n + 4 * m.n_cells * int(np.prod(q)))
    o.set_particles(P, n)
    g.set_particles(P, n)
    for _ in range(STEPS):
        Vo, Vg = o.step(V, V), g.step(V, V)
        so, sg = o.stats(), g.stats()
        for k in ("n_particles", "removed", "seeded", "lost", "next_id"):
            assert so[k] == sg[k], k
        if precision == "fp64":
            assert_same_particles(o.particles(), g.particles())
            assert_v_close(Vo, Vg, V_RTOL_FP64)
        else:
            a, b = by_id(o.particles()), by_id(g.particles())
            assert np.array_equal(a["id"], b["id"]) and np.array_equal(a["cell"], b["cell"])
            # a coordinate's step: 2 sub-steps, each a handful of roundings of 6e-8; the sums of up to
            # 1000 terms as in the tile tests, under 32 roundings, over 8 coordinate errors of 1e-6
            assert np.max(np.abs(a["xi"] - b["xi"])) <= 2e-6
            assert_v_close(Vo, Vg, 2e-5)
    g.close()


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("shape,q,maxpp,patterns", [
    ((128, 64), (4, 4), 2, 12),
    ((128, 64), (4, 4), 40, 12),
    ((128, 64), (3, 5), -1, 12),
    ((32, 16, 16), (2, 3, 1), 0, 12),
    ((32, 16, 16), (3, 3, 3), 2, 4),
])
def test_tiles_of_several_cells(shape, q, maxpp, patterns, precision):
    nc = int(np.prod(shape))
    n_of = np.full(nc, int(np.prod(q)))
    for k in range(patterns):
        # 631 = 1 modulo tiles of 10 and of 14 cells: the 700 is first, inside and last in its tile
        b = 69 + 631 * k - BIG
        n_of[b:b + len(COUNTS)] = COUNTS
    # at most 8 blocks on each of 148 SMs, and tiles by load of more cells than one block's share
    assert nc > 4 * 8 * 148 and n_of.sum() < 32 * nc
    _run(shape, q, maxpp, n_of, precision)


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_blocks_of_cells_beyond_a_tile(precision):
    """Every tile is one cell beyond it, more tiles than blocks in one form
    and fewer in the other: nothing but the tickets orders a block's warps."""
    shape = (40, 20)
    _run(shape, (4, 4), 80, np.full(int(np.prod(shape)), 700), precision)
