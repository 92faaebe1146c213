"""The 2D grid stepper's bounded waits that run out, without a fault.

GPUE_TEST_STEP_WAIT (a test hook, read at each launch) makes every barrier wait
for CTAs that never come ("barrier"), or every norm for a pass number that no
CTA writes ("norm"), for 0.1 s each.  The CTAs leave the walk and the call
reports GPUE_ERR_TIMEOUT.  What they leave behind is clean: the same context,
given its state again, steps bit for bit like one that never saw the hook.
"""
import time

import numpy as np
import pytest

import cases
import gpue_b200 as G
from helpers import product_params

pytestmark = pytest.mark.gpu


def case(n, **kw):
    return dict(cases.DEFAULTS, dim=2, n=n, box=8.0, g=100.0, gdt=1e-4, dt=1e-4, init="gauss",
                seed=821, **kw)


@pytest.mark.parametrize("hook,gstate", [("barrier", 0), ("norm", 0), ("barrier", 1), ("norm", 1)])
@pytest.mark.parametrize("n,prec", [(128, G.PREC_FP64), (256, G.PREC_FP32), (1024, G.PREC_FP32)])
def test_evolve_reports_it_and_recovers(monkeypatch, hook, gstate, n, prec):
    c = case(n)
    psi0 = cases.initial_psi(c)
    opts = dict(norm_guard=1, norm_guard_period=1) if gstate else {}
    with G.Solver(product_params(c, prec)) as s:
        s.set_wfc(psi0)
        s.evolve(6, gstate, **opts)
        want = s.get_wfc()
        s.set_wfc(psi0)
        monkeypatch.setenv("GPUE_TEST_STEP_WAIT", hook)
        t0 = time.time()
        with pytest.raises(G.GpueError) as e:
            s.evolve(6, gstate, **opts)
        assert e.value.status == 7  # GPUE_ERR_TIMEOUT
        assert time.time() - t0 < 30
        monkeypatch.delenv("GPUE_TEST_STEP_WAIT")
        for _ in range(2):
            s.set_wfc(psi0)
            s.evolve(6, gstate, **opts)
            assert np.array_equal(s.get_wfc(), want)


def test_batch_names_the_solve(monkeypatch):
    """In a batch the waits are the solve's own: its neighbour on a cluster ends as alone."""
    big, small = case(768), case(128)
    with G.Solver(product_params(big, G.PREC_FP32)) as a, \
            G.Solver(product_params(small, G.PREC_FP32)) as b:
        b.set_wfc(cases.initial_psi(small))
        with G.Batch([b]) as one:
            one.evolve(0, 4)
        want = b.get_wfc()
        a.set_wfc(cases.initial_psi(big))
        b.set_wfc(cases.initial_psi(small))
        monkeypatch.setenv("GPUE_TEST_STEP_WAIT", "barrier")
        with G.Batch([a, b]) as two:
            with pytest.raises(G.GpueError) as e:
                two.evolve(0, 4)
        assert e.value.status == 7 and "solve 0 " in str(e.value)
        assert np.array_equal(b.get_wfc(), want)
