"""The cluster-resident 2D stepper (cluster_step.cuh) that batched and served
solves of up to 512^2 complex64 and 256^2 complex128 run on.

Each length against the solve stepped alone (the grid-wide stepper, or line
passes), in both time kinds, with and without the rotation gauge; and the same
solve in batches that give it different cluster sizes, bit for bit.  The bounds
are those of two orders of the same sums: 40 steps of at most 8 transforms of
10 levels, at 2^-53 (1e-14 a step) and 2^-24 (5e-6 a step, adding as a random
walk).
"""
import numpy as np
import pytest

import gpue_b200 as G

pytestmark = pytest.mark.gpu

LENGTHS = {G.PREC_FP32: (16, 32, 64, 96, 128, 160, 192, 256, 320, 384, 512),
           G.PREC_FP64: (16, 32, 64, 96, 128, 160, 192, 256)}
TOL = {G.PREC_FP64: 1e-12, G.PREC_FP32: 4e-5}


def start(n, seed):
    x = -8.0 + 8.0 / (n >> 1) * np.arange(n)
    rng = np.random.Generator(np.random.PCG64(seed))
    psi = np.exp(-(x[None, :] ** 2 + x[:, None] ** 2) / 9) * (
        1 + 0.02 * rng.standard_normal((n, n))) * np.exp(0.3j * x[None, :])
    return psi / np.sqrt(np.sum(np.abs(psi) ** 2) * (8.0 / (n >> 1)) ** 2)


def solver(n, prec, omega, k, line=False):
    p = G.make_params(2, n, 8.0, g=100.0 + 10 * k, wy=1.0 + 0.02 * k, omega=omega,
                      gauge=omega != 0.0, gdt=1e-4, dt=1e-4, precision=prec)
    s = G.Solver(p)
    if line:
        q = s.plan(0)
        s.set_plan(0, q["ra"], q["rb"], q["rc"], q["threads_per_line"])
    s.set_wfc(start(n, k))
    return s


def batch(specs, gstate, steps, every=0):
    ss = [solver(*q) for q in specs]
    with G.Batch(ss) as b:
        res, stats = b.evolve(gstate, steps, energy_every=every)
    out = [(s.get_wfc(), r) for s, r in zip(ss, res)]
    for s in ss:
        s.close()
    return out, stats


@pytest.mark.parametrize("prec", [G.PREC_FP64, G.PREC_FP32])
@pytest.mark.parametrize("gstate,omega", [(0, 0.0), (0, 0.5), (1, 0.0), (1, 0.5)])
def test_matches_lone_solves(prec, gstate, omega):
    specs = [(n, prec, omega, k) for k, n in enumerate(LENGTHS[prec])]
    got, _ = batch(specs, gstate, 41, every=20)
    for (n, _, _, k), (psi, r) in zip(specs, got):
        with solver(n, prec, omega, k, line=True) as s:
            ref = s.evolve(41, gstate, energy_every=20,
                           norm_guard=1 if gstate and prec == G.PREC_FP32 else 0,
                           norm_guard_period=1)
            psi_ref = s.get_wfc()
        err = np.linalg.norm(psi - psi_ref) / np.linalg.norm(psi_ref)
        assert err < TOL[prec], (n, err)
        assert r["steps_done"] == 41
        assert abs(r["energy"] - ref["energy"]) < TOL[prec] * abs(ref["energy"]), n


@pytest.mark.parametrize("prec,n", [(G.PREC_FP32, 96), (G.PREC_FP32, 128), (G.PREC_FP32, 256),
                                    (G.PREC_FP64, 128)])
@pytest.mark.parametrize("gstate,omega", [(0, 0.0), (1, 0.4)])
def test_result_is_the_same_for_any_cluster_size(prec, n, gstate, omega):
    """Alone a solve gets the largest cluster, among 100 the smallest."""
    one, _ = batch([(n, prec, omega, 0)], gstate, 30)
    many, _ = batch([(n, prec, omega, k) for k in range(100)], gstate, 30)
    few, _ = batch([(n, prec, omega, k) for k in range(12)], gstate, 30)
    assert np.array_equal(one[0][0], many[0][0])
    assert np.array_equal(one[0][0], few[0][0])
    assert np.array_equal(many[11][0], few[11][0])

