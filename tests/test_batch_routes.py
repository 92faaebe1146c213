"""Which kernels batched 2D solves run on, by length, precision and gauge, and how
clusters are shared out.  CPU test over the fake CUDA runtime (fake_cudart.cpp), which
records every launch; the same routes on a real device are in test_gpu_batch_routes.py."""
import pytest

from fake_device import fake  # noqa: F401

LENGTHS = (16, 32, 64, 96, 128, 160, 192, 256, 320, 384, 512, 640, 768, 1024)
# the routes' lines (batch.cu, kernels_cluster_*.cu)
CLUSTER = {"FP32": {16, 32, 64, 96, 128, 160, 192, 256}, "FP64": {16, 32, 64, 96, 128, 192, 256}}
GRID = {"FP32": {512, 768, 1024}, "FP64": {768, 1024}}


def routes(prec, omega):
    """The lengths on clusters and on the grid; complex64 384^2 goes by the gauge."""
    c, g = set(CLUSTER[prec]), set(GRID[prec])
    if prec == "FP32":
        (g if omega else c).add(384)
    return c, g


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


def kinds(launches):
    out = set()
    for q in launches:
        for name in ("k_cluster_many", "k_step2d", "k_pass_batch", "k_batch_mega"):
            if name in q["kernel"]:
                out.add(name)
    return out


@pytest.mark.parametrize("prec", ["FP32", "FP64"])
@pytest.mark.parametrize("gstate,omega", [(0, 0.0), (0, 0.5), (1, 0.0), (1, 0.5)])
def test_route_of_each_length(fake, prec, gstate, omega):  # noqa: F811
    on_cluster, on_grid = routes(prec, omega)
    for n in LENGTHS:
        _, launches = fake(BATCH + "batch([(%d, G.PREC_%s, %g)], %d)" % (n, prec, omega, gstate))
        if n in on_cluster:
            assert kinds(launches) == {"k_cluster_many"}, n
        elif n in on_grid:
            assert kinds(launches) == {"k_step2d"}, n
        else:
            assert kinds(launches) <= {"k_pass_batch", "k_batch_mega"}, n


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


@pytest.mark.parametrize("n,omega", [(384, 0.3), (512, 0.0)])
def test_grids_share_lanes(fake, n, omega):  # noqa: F811
    """One cooperative launch per solve, whatever lane it is on."""
    _, launches = fake(BATCH + "batch([(%d, G.PREC_FP32, %g)] * 9)" % (n, omega))
    grids = [q for q in launches if "k_step2d" in q["kernel"]]
    assert len(grids) == 9 and all(q["coop"] for q in grids)
