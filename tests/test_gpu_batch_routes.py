"""Batched 2D solves take the routes that test_batch_routes.py names on this device
too (nothing declined for want of residency), and many alike, side by side on lanes
or in clusters, end bit for bit as alone.

The tests that compare those kernels with line passes (test_gpu_cluster.py,
test_gpu_batch_grid.py) rely on it: 512^2 complex64, and 384^2 with the gauge, run on
the grid stepper, 320^2 complex64 and 160^2 complex128 as line passes.
"""
import numpy as np
import pytest

import gpue_b200 as G
from test_batch_routes import LENGTHS, routes
from test_gpu_cluster import batch

pytestmark = pytest.mark.gpu

STEPS = 40


@pytest.mark.parametrize("prec", ["FP64", "FP32"])
@pytest.mark.parametrize("gstate,omega", [(0, 0.0), (1, 0.4)])
def test_resident_routes_are_taken(prec, gstate, omega):
    p = getattr(G, "PREC_" + prec)
    for n in LENGTHS:
        _, stats = batch([(n, p, omega, 0)], gstate, STEPS)
        if n in set.union(*routes(prec, omega)):
            assert stats["kernel_launches"] == 1, n  # every step in one launch
    _, stats = batch([(640, p, omega, 0)], gstate, STEPS)  # line passes: several a step
    assert stats["kernel_launches"] > 2 * STEPS


@pytest.mark.parametrize("prec,n,count", [(G.PREC_FP32, 384, 9), (G.PREC_FP32, 512, 5),
                                          (G.PREC_FP32, 256, 8), (G.PREC_FP64, 256, 8)])
@pytest.mark.parametrize("gstate,omega", [(0, 0.0), (1, 0.4)])
def test_many_alike_end_as_alone(prec, n, count, gstate, omega):
    many, _ = batch([(n, prec, omega, k) for k in range(count)], gstate, 30, every=10)
    for k in (0, 1, count - 1):
        one, _ = batch([(n, prec, omega, k)], gstate, 30, every=10)
        assert np.array_equal(one[0][0], many[k][0]), k
        assert one[0][1] == many[k][1], k


@pytest.mark.parametrize("gstate", [0, 1])
def test_all_routes_at_once(gstate):
    """Grids on several lanes beside clusters and line passes: no wait runs out, and
    every solve ends as alone."""
    specs = ([(384, G.PREC_FP32, 0.3, k) for k in range(5)] +
             [(512, G.PREC_FP32, 0.0, k) for k in range(3)] +
             [(768, G.PREC_FP32, 0.0, 0), (768, G.PREC_FP64, 0.0, 0), (1024, G.PREC_FP32, 0.0, 0),
              (640, G.PREC_FP32, 0.0, 0), (256, G.PREC_FP32, 0.0, 0), (128, G.PREC_FP64, 0.3, 0)])
    got, _ = batch(specs, gstate, 30, every=10)
    for q, (psi, r) in zip(specs, got):
        (alone, ra), = batch([q], gstate, 30, every=10)[0]
        assert np.array_equal(alone, psi), q
        assert ra == r, q
