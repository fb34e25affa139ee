"""The window's reverse sweep where its instances differ by dimension, form
and mesh: the FP32 form on twisted hexes, segments of a single sub-step
(shorter than the states read ahead), and windows without a correction, whose
flush adds one set of gradients."""
import dataclasses

import numpy as np
import pytest

from . import cases
from .test_gpu_adjoint import CASES, G_RTOL_FP64, objective, rel, setup

pytestmark = pytest.mark.gpu


def test_fp32_twisted_hexes_against_fp64():
    c = CASES["cube"]()
    o, _ = setup(c, "fp64")
    _, g32 = setup(c, "fp32")
    K, C = 6, 3
    U0 = o.window_forward(K, c.V, c.Vold)
    gU = objective(U0)[1](U0)
    _, gv0_o, gV_o, gVo_o = o.window_adjoint(K, c.V, gU, Vold=c.Vold)
    _, gv0, gV, gVo = g32.adjoint(K, C, c.V, gU, Vold=c.Vold)
    po, p32 = o.particles(), g32.particles()
    common, ia, ib = np.intersect1d(po["id"], p32["id"], return_indices=True)
    assert len(common) >= 0.99 * len(po["id"])
    # as for the FP32 form on the duct and the cylinder
    assert rel(gv0[ib], gv0_o[ia]) <= 1e-4
    assert rel(gV, gV_o) <= 1e-4
    assert rel(gVo, gVo_o) <= 1e-4


@pytest.mark.parametrize("which", ["channel", "duct", "cube"])
@pytest.mark.parametrize("substeps,K,C", [(1, 3, 1), (2, 3, 1), (3, 4, 4)])
@pytest.mark.parametrize("correct", [False, True])
def test_fp64_short_segments(which, substeps, K, C, correct):
    c = dataclasses.replace(CASES[which](), substeps=substeps)
    o, g = setup(c)
    Vold = c.Vold if correct else None
    U0 = o.window_forward(K, c.V, Vold)
    gU = objective(U0)[1](U0)
    _, gv0_o, gV_o, gVo_o = o.window_adjoint(K, c.V, gU, Vold=Vold)
    _, gv0, gV, gVo = g.adjoint(K, C, c.V, gU, Vold=Vold)
    po, pg = o.particles(), g.particles()
    oo, og = np.argsort(po["id"]), np.argsort(pg["id"])
    assert rel(gv0[og], gv0_o[oo]) <= G_RTOL_FP64
    assert rel(gV, gV_o) <= G_RTOL_FP64
    if correct:
        assert rel(gVo, gVo_o) <= G_RTOL_FP64


@pytest.mark.parametrize("n", [12, 13, 15, 17])
def test_fp32_twisted_hexes_sizes(n):
    """27 n^3 particles: one round of the reverse sweep's blocks (3 an SM on 148 SMs), a little more, two, and more."""
    c = cases.cube(n, q=(3, 3, 3), dt=0.3 / n)
    o, _ = setup(c, "fp64", pre_steps=0)
    _, g32 = setup(c, "fp32", pre_steps=0)
    K, C = 3, 2
    U0 = o.window_forward(K, c.V, c.Vold)
    gU = objective(U0)[1](U0)
    _, gv0_o, gV_o, gVo_o = o.window_adjoint(K, c.V, gU, Vold=c.Vold)
    _, gv0, gV, gVo = g32.adjoint(K, C, c.V, gU, Vold=c.Vold)
    po, p32 = o.particles(), g32.particles()
    assert len(p32["id"]) == 27 * n**3
    oo, og = np.argsort(po["id"]), np.argsort(p32["id"])
    assert rel(gv0[og], gv0_o[oo]) <= 1e-4
    assert rel(gV, gV_o) <= 1e-4
    assert rel(gVo, gVo_o) <= 1e-4
