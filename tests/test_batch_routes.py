"""How clusters are shared out among batched 2D solves.  CPU test over the fake CUDA runtime (fake_cudart.cpp), which
records every launch."""
import pytest

from fake_device import fake  # noqa: F401

BATCH = """
def batch(specs, gstate=0, steps=3):
    ss = [G.Solver(G.make_params(2, n, 8.0, g=100.0, omega=om, gauge=om != 0.0, precision=prec))
          for n, prec, om in specs]
    for s in ss:
        s.set_wfc(psi(s.params.xDim))
    with G.Batch(ss) as b:
        b.evolve(gstate, steps)
    for s in ss:
        s.close()
"""


@pytest.mark.parametrize("count", [1, 7, 8, 9, 12, 16, 17, 40, 100])
def test_equal_solves_get_equal_clusters(fake, count):  # noqa: F811
    """One launch, one cluster size, and all of them resident at once while they can be
    (the fake device: 8 GPCs of 18 SMs)."""
    _, launches = fake(BATCH + "batch([(96, G.PREC_FP32, 0.0)] * %d)" % count)
    many = [q for q in launches if "k_cluster_many" in q["kernel"]]
    assert len(many) == 1
    size = many[0]["cluster"]
    assert many[0]["grid"] == count * size
    fits = [s for s in (16, 8, 4, 2, 1) if count <= 8 * (18 // s)]
    assert size == fits[0]

