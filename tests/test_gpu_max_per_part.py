"""The largest max_particles_per_cell_part: no particle is removed, as in the
oracle (the kernels compare counts with max + 1)."""
import pytest

from . import cases
from .test_gpu_parity import STAT_KEYS, assert_same_particles, make

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("maxpp", [2 ** 31 - 2, 2 ** 31 - 1])
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_largest_max_removes_nothing(maxpp, precision):
    c = cases.channel(32, 8, maxpp=maxpp, dt=0.02)
    o, g = make(c, precision=precision)
    o.seed(c.V)
    g.seed_particles(c.V)
    for _ in range(4):
        o.step(c.V, c.Vold)
        g.step(c.V, c.Vold)
    assert g.stats()["removed"] == o.stats()["removed"] == 0
    if precision == "fp64":
        assert_same_particles(o.particles(), g.particles())
        for k in STAT_KEYS:
            assert o.stats()[k] == g.stats()[k], k
    g.close()
