"""A bounded device wait that runs out in a batch or a served tick is reported
for the solve it spoils, and for no other.

GPUE_TEST_PLANE_WAIT=1 (read when a context plans its passes) makes the y-tiles
of a 3D tile pass wait, a second at most, for one x-tile more than a plane has:
no fault, no hang, the kernels record it and return.  A solve beside it that
was made without the hook ends as it does without such company.
"""
import numpy as np
import pytest

import cases
import gpue_b200 as G
from helpers import dV, product_params

pytestmark = pytest.mark.gpu

C3 = dict(cases.DEFAULTS, dim=3, n=64, box=8.0, wz=2.0, g=100.0, gdt=1e-4, init="gauss",
          seed=811)
C2 = dict(cases.DEFAULTS, dim=2, n=128, box=8.0, g=100.0, gdt=1e-4, init="gauss", seed=812)


def solver(c, monkeypatch=None):
    if monkeypatch:
        monkeypatch.setenv("GPUE_TEST_PLANE_WAIT", "1")
    s = G.Solver(product_params(c, G.PREC_FP32))
    if monkeypatch:
        monkeypatch.delenv("GPUE_TEST_PLANE_WAIT")
    s.set_wfc(cases.initial_psi(c))
    return s


def test_batch(monkeypatch):
    monkeypatch.setenv("GPUE_BATCH_TILE_MIN", "1")  # 64^3 takes the tile passes
    with solver(C2) as ref:
        with G.Batch([ref]) as b:
            b.evolve(0, 2)
        want = ref.get_wfc()
    with solver(C3, monkeypatch) as bad, solver(C2) as good:
        with G.Batch([good, bad]) as b:
            with pytest.raises(G.GpueError) as e:
                b.evolve(0, 2)
        assert e.value.status == 7  # GPUE_ERR_TIMEOUT
        assert "solve 1 " in str(e.value)
        assert np.array_equal(good.get_wfc(), want)
        # the report is not left over for the next call on either context
        good.evolve(1, 0)
        bad.get_wfc()
        assert abs(good.norm() - 1.0) < 1e-5


def test_server(monkeypatch):
    monkeypatch.setenv("GPUE_BATCH_TILE_MIN", "1")
    monkeypatch.setenv("GPUE_TEST_PLANE_WAIT", "1")  # 2D solves have no plane waits
    with G.Server(precision=G.PREC_FP32, check_steps=2) as S:
        for tag, c in ((0, C3), (1, C2)):
            S.submit(product_params(c, G.PREC_FP32), 0, 2, cases.initial_psi(c), tag)
        got = {}
        for _ in range(60):
            for r in S.poll(timeout=2.0):
                got[r["tag"]] = r
            if len(got) == 2:
                break
        st = S.stats()
    assert got[0]["status"] == 7 and np.isnan(got[0]["energy"])
    assert got[1]["status"] == 0
    assert st["timed_out"] == 1 and st["failed"] == 1 and st["completed"] == 1
    psi = got[1]["psi"]
    assert abs(np.sum(np.abs(psi) ** 2) * dV(C2) - 1.0) < 1e-5
