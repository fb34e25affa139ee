"""The write pass's tiles at the sizes where they can go wrong: cells of 0, 1
and one particle either side of a warp round, several cells that together
overflow a tile, single cells beyond one (the general path), arrival lists
beyond their slots, and the largest part grid.  FP64 form against the oracle
bit for bit with motion; FP32 form without motion against the oracle's ids,
cells and counts, and its projection."""
import numpy as np
import pytest

from oracle.oracle import forward_map
from pfem2dealii_b200 import mesh as M

from . import cases
from .test_gpu_parity import V_RTOL_FP64, assert_same_particles, assert_v_close, by_id, make

pytestmark = pytest.mark.gpu

# particles of consecutive cells; the rest of the mesh holds one per part
COUNTS = [0, 1, 31, 32, 33, 63, 64, 65, 96, 97, 479, 481, 0, 0, 511, 513, 700, 5, 250, 250, 250]
CONFIGS = [
    ("channel", (4, 4), 2),
    ("channel", (15, 15), 2),  # 256 extended parts
    ("duct", (3, 3, 3), 2),
    ("cube", (4, 4, 4), 5),
    ("duct", (2, 3, 1), 0),
    ("channel", (3, 5), -1),
]


def _setup(which, q, maxpp, dt):
    m = {"channel": lambda: M.hyper_rectangle((0.0, 0.0), (4.0, 1.0), (11, 5)),
         "duct": lambda: M.hyper_rectangle((0.0, 0.0, 0.0), (3.0, 1.0, 1.0), (5, 3, 3)),
         "cube": lambda: M.perturbed_cube(4)}[which]()
    fn = {"channel": M.channel_profile(), "duct": M.duct_profile(), "cube": M.taylor_green_3d()}[which]
    V = M.field_at_dofs(m, fn)
    c = cases.Case(which, m, V, 0.9 * V, q, maxpp, 2, dt)
    rng = np.random.default_rng(3)
    npart = int(np.prod(q))
    n_of = np.full(m.n_cells, npart)
    n_of[2:2 + len(COUNTS)] = COUNTS
    cell = np.repeat(np.arange(m.n_cells), n_of)
    n = len(cell)
    # off the part boundaries, representable in FP32
    part = np.stack([rng.integers(0, k, n) for k in q], 1)
    xi = ((part + rng.uniform(0.02, 0.98, part.shape)) / np.array(q)).astype(np.float32).astype(np.float64)
    x = np.array([forward_map(m.vertices[m.cells[k]], z) for k, z in zip(cell, xi)])
    v = rng.normal(size=xi.shape).astype(np.float32).astype(np.float64)
    ids = (rng.permutation(n) + 1).astype(np.uint32)
    return c, {"id": ids, "cell": cell.astype(np.int32), "x": x, "xi": xi, "v": v}, n


@pytest.mark.parametrize("which,q,maxpp", CONFIGS)
def test_fp64_tile_edges_bit_exact(which, q, maxpp):
    c, P, n = _setup(which, q, maxpp, 0.05)
    o, g = make(c, capacity=40000)
    o.set_particles(P, n)
    g.set_particles(P, n)
    assert_same_particles(o.particles(), g.particles())
    assert_v_close(o.project(), g.project_particle_fields(), V_RTOL_FP64)
    for _ in range(3):
        Vo, Vg = o.step(c.V, c.Vold), g.step(c.V, c.Vold)
        assert_same_particles(o.particles(), g.particles())
        assert_v_close(Vo, Vg, V_RTOL_FP64)
        for k in ("n_particles", "removed", "seeded", "lost", "next_id"):
            assert o.stats()[k] == g.stats()[k], k


@pytest.mark.parametrize("which,q,maxpp", CONFIGS)
def test_fp32_tile_edges_without_motion(which, q, maxpp):
    c, P, n = _setup(which, q, maxpp, 0.0)
    o, g = make(c, capacity=40000, precision="fp32")
    o.set_particles(P, n)
    g.set_particles(P, n)
    for _ in range(2):
        Vo, Vg = o.step(c.V, c.V), g.step(c.V, c.V)
        a, b = by_id(o.particles()), by_id(g.particles())
        assert np.array_equal(a["id"], b["id"]) and np.array_equal(a["cell"], b["cell"])
        # sums of up to 700 terms: 5 tree levels, the compensated add, products of 4 factors and
        # inputs, each 2^-24, over numerator and denominator: under 32 roundings of 6e-8
        assert_v_close(Vo, Vg, 2e-6)
