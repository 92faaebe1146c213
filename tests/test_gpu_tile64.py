"""The tile-stream passes (tstream.cuh) in complex128, and in both precisions
with the rotation gauge, against the line passes (GPUE_XY, GPUE_PLANE and
GPUE_ZTMA off).

Both sides run the same transforms and factors from the same state, so they
differ by rounding: 6 to 10 transforms of 8 levels a step, at most 1e-14 in
complex128 and 5e-6 in complex64 (unbiased over the steps).
"""
import os

import numpy as np
import pytest

import gpue_b200 as G

pytestmark = pytest.mark.gpu

OFF = {"GPUE_XY": "0", "GPUE_PLANE": "0", "GPUE_ZTMA": "0"}
TOL = {G.PREC_FP64: 1e-12, G.PREC_FP32: 2e-5}


def start(n, seed=3):
    rng = np.random.Generator(np.random.PCG64(seed))
    x = -6.0 + 6.0 / (n >> 1) * np.arange(n)
    r2 = x[None, None, :] ** 2 + x[None, :, None] ** 2 + 2 * x[:, None, None] ** 2
    psi = np.exp(-r2 / 6) * (1 + 0.02 * rng.standard_normal((n, n, n))) * np.exp(
        0.4j * x[None, None, :] - 0.2j * x[None, :, None])
    return psi / np.sqrt(np.sum(np.abs(psi) ** 2) * (6.0 / (n >> 1)) ** 3)


def run(n, prec, gstate, omega, steps, lines, psi0, polish=0, yscale=1.0, **kw):
    old = {k: os.environ.get(k) for k in OFF}
    if lines:
        os.environ.update(OFF)
    try:
        p = G.make_params(3, n, 6.0, wz=2.0, g=300.0, omega=omega, gauge=omega != 0.0,
                          gdt=1e-4, dt=1e-4, precision=prec)
        p.yMax *= yscale
        with G.Solver(p) as s:
            s.set_wfc(psi0)
            r = s.evolve(steps, gstate, polish_steps=polish, **kw)
            return s.get_wfc(), s.energy(), r
    finally:
        for k, v in old.items():
            if v is None:
                os.environ.pop(k, None)
            else:
                os.environ[k] = v


def close(a, b, prec):
    assert np.linalg.norm(a[0] - b[0]) / np.linalg.norm(b[0]) < TOL[prec]
    assert abs(a[1] - b[1]) < TOL[prec] * abs(b[1])
    assert abs(a[2]["norm"] - b[2]["norm"]) < TOL[prec] * b[2]["norm"]


@pytest.mark.parametrize("n", [128, 160, 192, 256])
@pytest.mark.parametrize("gstate,omega", [(0, 0.0), (1, 0.0), (0, 0.5), (1, 0.5)])
def test_complex128_matches_line_passes(n, gstate, omega):
    psi0 = start(n)
    steps = 5 if n < 256 else 3
    a = run(n, G.PREC_FP64, gstate, omega, steps, False, psi0)
    b = run(n, G.PREC_FP64, gstate, omega, steps, True, psi0)
    assert a[2]["kernel_launches"] < b[2]["kernel_launches"]
    close(a, b, G.PREC_FP64)


@pytest.mark.parametrize("gstate", [0, 1])
def test_complex64_gauge_matches_line_passes(gstate):
    psi0 = start(192)
    a = run(192, G.PREC_FP32, gstate, 0.6, 5, False, psi0)
    b = run(192, G.PREC_FP32, gstate, 0.6, 5, True, psi0)
    assert a[2]["kernel_launches"] < b[2]["kernel_launches"]
    close(a, b, G.PREC_FP32)


def test_box_lengths_that_differ():
    """The gauge factor of each axis takes that axis' momentum spacing."""
    psi0 = start(128)
    for gstate in (0, 1):
        a = run(128, G.PREC_FP64, gstate, 0.5, 4, False, psi0, yscale=1.3)
        b = run(128, G.PREC_FP64, gstate, 0.5, 4, True, psi0, yscale=1.3)
        close(a, b, G.PREC_FP64)


def test_runs_repeat_bit_for_bit():
    """The norm does not depend on which CTA took which tile."""
    psi0 = start(128)
    runs = [run(128, G.PREC_FP64, 0, 0.0, 12, False, psi0) for _ in range(3)]
    assert all(np.array_equal(runs[0][0], r[0]) for r in runs[1:])
    sliced = run(128, G.PREC_FP64, 0, 0.0, 12, False, psi0, graph_chunk=5)
    assert np.array_equal(runs[0][0], sliced[0])


def test_polish_steps():
    psi0 = start(128)
    a = run(128, G.PREC_FP32, 0, 0.0, 3, False, psi0, polish=4)
    b = run(128, G.PREC_FP32, 0, 0.0, 3, True, psi0, polish=4)
    close(a, b, G.PREC_FP32)


@pytest.mark.parametrize("gstate,omega", [(0, 0.0), (1, 0.5)])
def test_batched_solves_match_lone_ones(gstate, omega):
    psi = [start(128, k) for k in range(2)]
    ss = []
    for k in range(2):
        s = G.Solver(G.make_params(3, 128, 6.0, wz=2.0, g=300.0, omega=omega, gauge=omega != 0.0,
                                   gdt=1e-4, dt=1e-4, precision=G.PREC_FP64))
        s.set_wfc(psi[k])
        ss.append(s)
    with G.Batch(ss) as b:
        b.evolve(gstate, 6)
    for k, s in enumerate(ss):
        ref = run(128, G.PREC_FP64, gstate, omega, 6, False, psi[k])[0]
        assert np.linalg.norm(s.get_wfc() - ref) / np.linalg.norm(ref) < TOL[G.PREC_FP64]
        s.close()
