"""The resident 2D stepper (stepper.cuh): many steps in one cooperative launch.

Every length against the line passes (a context whose plan was set by hand
steps through them), in both precisions and time kinds, with and without the
rotation gauge, and with full-field tables.  Both sides run the same steps
from the same state, so they differ by rounding alone: a complex128 step adds
at most about 8 transforms of 10 levels at 2^-53 (1e-14), a complex64 one the
same at 2^-24 (5e-6 at worst, unbiased over the steps); the bounds hold 30 and
10 such steps.
"""
import numpy as np
import pytest

import gpue_b200 as G

pytestmark = pytest.mark.gpu

LENGTHS = (16, 32, 64, 96, 128, 160, 192, 256, 320, 384, 512, 640, 768, 1024)
TOL = {G.PREC_FP64: 1e-12, G.PREC_FP32: 2e-5}


def start(n, box, seed=5):
    x = -box + box / (n >> 1) * np.arange(n)
    rng = np.random.Generator(np.random.PCG64(seed))
    psi = np.exp(-(x[None, :] ** 2 + x[:, None] ** 2) / (0.12 * box * box))
    psi = psi * (1 + 0.02 * rng.standard_normal((n, n))) * np.exp(
        1j * (0.3 * x[None, :] - 0.2 * x[:, None] * x[None, :] / box))
    return psi / np.sqrt(np.sum(np.abs(psi) ** 2) * (box / (n >> 1)) ** 2)


def run(n, prec, gstate, omega, steps, lines=False, setup=None, calls=None, dt=1e-4, g=150.0,
        **kw):
    p = G.make_params(2, n, 8.0, g=g, omega=omega, gauge=omega != 0.0, gdt=dt, dt=dt,
                      precision=prec)
    with G.Solver(p) as s:
        if setup:
            setup(s)
        if lines:
            for axis in (0, 1):
                q = s.plan(axis)
                s.set_plan(axis, q["ra"], q["rb"], q["rc"], q["threads_per_line"])
        s.set_wfc(start(n, 8.0))
        off = 0
        for k in calls or [steps]:
            r = s.evolve(k, gstate, step_offset=off, **kw)
            off += k
        return s.get_wfc(), r


def rel(a, b):
    return float(np.linalg.norm(a - b) / np.linalg.norm(b))


@pytest.mark.parametrize("prec", [G.PREC_FP64, G.PREC_FP32])
@pytest.mark.parametrize("n", LENGTHS)
def test_matches_line_passes(n, prec):
    steps = 30 if prec == G.PREC_FP64 else 10
    for gstate, omega in ((0, 0.0), (0, 0.6), (1, 0.0), (1, 0.6)):
        a, ra = run(n, prec, gstate, omega, steps)
        b, rb = run(n, prec, gstate, omega, steps, lines=True)
        assert ra["kernel_launches"] < rb["kernel_launches"]
        assert rel(a, b) < TOL[prec], (gstate, omega)
        assert abs(ra["norm"] - rb["norm"]) < TOL[prec] * max(1.0, rb["norm"])


@pytest.mark.parametrize("prec", [G.PREC_FP64, G.PREC_FP32])
@pytest.mark.parametrize("gstate", [0, 1])
def test_large_angles(prec, gstate):
    """Nonlinear and gauge angles past the small-angle series' range."""
    kw = dict(dt=4e-3, g=2000.0)
    a, _ = run(64, prec, gstate, 0.8, 10, **kw)
    b, _ = run(64, prec, gstate, 0.8, 10, lines=True, **kw)
    assert rel(a, b) < TOL[prec]


@pytest.mark.parametrize("prec", [G.PREC_FP64, G.PREC_FP32])
@pytest.mark.parametrize("gstate,omega", [(0, 0.0), (0, 0.5), (1, 0.5)])
def test_slices_and_checks(prec, gstate, omega):
    """A walk of any length repeats the same steps: slices of every residue,
    long walks (their middle is a repeated pattern) and runs cut by energy
    checks end bit for bit where one call does (without the norm guard, which
    every call starts afresh)."""
    one, _ = run(96, prec, gstate, omega, 61, norm_guard=0)
    for calls in ([1] * 5 + [56], [23, 38], [24, 25, 12]):
        got, _ = run(96, prec, gstate, omega, 61, calls=calls, norm_guard=0)
        if gstate == 0:  # every call returns the renormalised state
            assert rel(got, one) < TOL[prec]
        else:
            assert np.array_equal(got, one)
    got, _ = run(96, prec, gstate, omega, 61, graph_chunk=7, norm_guard=0)
    assert np.array_equal(got, one)
    got, r = run(96, prec, gstate, omega, 61, energy_every=10, norm_guard=0)
    assert r["n_energies"] == 7 and np.array_equal(got, one)


@pytest.mark.parametrize("period", [1, 2, 4])
def test_norm_guard(period):
    a, ra = run(128, G.PREC_FP32, 1, 0.5, 37, norm_guard=1, norm_guard_period=period)
    b, rb = run(128, G.PREC_FP32, 1, 0.5, 37, lines=True, norm_guard=1,
                norm_guard_period=period)
    # 37 steps of at most 5e-6 that add as a random walk
    assert rel(a, b) < 4e-5 and abs(ra["norm"] - rb["norm"]) < 1e-6


@pytest.mark.parametrize("prec", [G.PREC_FP64, G.PREC_FP32])
@pytest.mark.parametrize("n", [16, 160, 320, 1024])
def test_field_tables(n, prec):
    x = -8.0 + 8.0 / (n >> 1) * np.arange(n)
    V = 0.5 * (x[None, :] ** 2 + 1.2 * x[:, None] ** 2) + 3 * np.cos(2 * x)[None, :] ** 2
    ax = np.broadcast_to(-0.4 * x[:, None], (n, n)).copy()
    ay = np.broadcast_to(0.4 * x[None, :] + 0.01 * np.sin(x)[None, :], (n, n)).copy()
    steps = 20 if prec == G.PREC_FP64 else 10

    def potential(s):
        s.set_potential_table(V)

    def gauge(s):
        s.set_gauge_tables(ax, ay)

    for setup, omega in ((potential, 0.0), (potential, 0.5), (gauge, 0.5)):
        for gstate in (0, 1):
            a, _ = run(n, prec, gstate, omega, steps, setup=setup)
            b, _ = run(n, prec, gstate, omega, steps, setup=setup, lines=True)
            assert rel(a, b) < TOL[prec], (setup.__name__, gstate)


def test_two_solvers_step_side_by_side():
    """Resident launches of different contexts from two threads: each ends as
    it does alone."""
    import threading
    ref = [run(n, G.PREC_FP64, 0, 0.0, 120)[0] for n in (256, 384)]
    got = [None, None]

    def work(i, n):
        for _ in range(5):
            got[i] = run(n, G.PREC_FP64, 0, 0.0, 120)[0]

    ts = [threading.Thread(target=work, args=a) for a in enumerate((256, 384))]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    for a, b in zip(got, ref):
        assert np.array_equal(a, b)
