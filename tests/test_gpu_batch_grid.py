"""Batched 2D solves on the grid-wide stepper (grid_eligible in batch.cu), at both
sides of its lines: 384^2 with the gauge and 512^2 complex64, 768^2 and 1024^2, and
640^2 and complex128 512^2, which stay on line passes.

Each solve against the same one stepped alone by line passes, and alone in a
batch against the mix, bit for bit.  The bounds are those of two orders of the
same sums: 40 steps of at most 8 transforms of 10 levels, at 2^-53 (1e-14 a
step) and 2^-24 (5e-6 a step, adding as a random walk).
"""
import numpy as np
import pytest

import gpue_b200 as G
from test_gpu_cluster import TOL, batch, solver

pytestmark = pytest.mark.gpu

LENGTHS = {G.PREC_FP32: (384, 512, 640, 768, 1024), G.PREC_FP64: (512, 640, 768, 1024)}


@pytest.mark.parametrize("prec", [G.PREC_FP64, G.PREC_FP32])
@pytest.mark.parametrize("gstate,omega", [(0, 0.0), (0, 0.5), (1, 0.0), (1, 0.5)])
def test_matches_lone_solves_and_any_company(prec, gstate, omega):
    specs = [(n, prec, omega, k) for k, n in enumerate(LENGTHS[prec])]
    got, _ = batch(specs, gstate, 41, every=20)
    for q, (psi, r) in zip(specs, got):
        with solver(*q, line=True) as s:
            ref = s.evolve(41, gstate, energy_every=20,
                           norm_guard=1 if gstate and prec == G.PREC_FP32 else 0,
                           norm_guard_period=1)
            psi_ref = s.get_wfc()
        err = np.linalg.norm(psi - psi_ref) / np.linalg.norm(psi_ref)
        assert err < TOL[prec], (q, err)
        assert r["steps_done"] == 41
        assert abs(r["energy"] - ref["energy"]) < TOL[prec] * abs(ref["energy"]), q
        (alone, _), = batch([q], gstate, 41, every=20)[0]
        assert np.array_equal(alone, psi), q
