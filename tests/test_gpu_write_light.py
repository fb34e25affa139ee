"""The FP32 write pass's two instances (few particles per part, or more) give
the same particles and projections bit for bit: a run that crosses the line
between them, with the host reading the density after every step, only now and
then, and never."""
import numpy as np
import pytest

from . import cases
from .test_gpu_parity import make

pytestmark = pytest.mark.gpu

STEPS = 120


@pytest.mark.parametrize("which,most", [
    (lambda: cases.channel(48, 12, dt=0.03), 16 + 2),
    (lambda: cases.channel(48, 12, q=(3, 2), maxpp=1, dt=0.03), 6 + 1),
    (lambda: cases.duct(24, 6, 6, q=(2, 2, 2), maxpp=1, dt=0.05), 8 + 1),
])
def test_instances_agree_across_the_line(which, most):
    import torch

    c = which()
    runs = []
    for sync in (1, 7, 0):
        _, g = make(c, precision="fp32", capacity=60000)
        g.seed_particles(c.V)
        dV = torch.from_numpy(np.ascontiguousarray(c.V)).cuda()
        out = torch.empty_like(dV)
        g.project_particle_fields_device(out)
        first = g.stats()["n_particles"]
        for s in range(STEPS):
            g.step_device(dV, None, out)
            if sync and s % sync == 0:
                g.stats()
        P = g.particles()
        last = g.stats()["n_particles"]
        assert first < most * c.mesh.n_cells <= last, (first, last)  # the run crosses the line
        runs.append([P[k] for k in ("id", "cell", "xi", "v")] + [out.cpu().numpy(), g.project_particle_fields()])
        g.close()
    for r in runs[1:]:
        for a, b in zip(runs[0], r):
            assert np.array_equal(a, b, equal_nan=True)
