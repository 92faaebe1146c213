"""Contexts on two devices of one process: every launch on the second one finds
the shared memory and cluster sizes it needs allowed there, whatever ran on the
first.  CPU test: the library runs over a fake CUDA runtime of two devices
(fake_cudart.cpp) that checks each launch against the attributes of its device."""
from fake_device import fake  # noqa: F401


def check(launches, kernel):
    assert not [q for q in launches if q["status"]]
    for d in (0, 1):
        assert [q for q in launches if q["device"] == d and kernel in q["kernel"]], (d, kernel)


def test_lone_solves_on_clusters(fake):  # noqa: F811
    _, launches = fake("""
for dev in (0, 1):
    for prec in (G.PREC_FP64, G.PREC_FP32):
        for n in (16, 32, 64):
            for gstate in (0, 1):
                with G.Solver(G.make_params(2, n, 8.0, precision=prec, device=dev)) as s:
                    s.set_wfc(psi(n))
                    s.evolve(3, gstate)
""")
    check(launches, "k_cluster_one")


def test_lone_solves_on_grids_and_tiles(fake):  # noqa: F811
    _, launches = fake("""
for dev in (0, 1):
    for prec in (G.PREC_FP64, G.PREC_FP32):
        for dim, n in ((2, 128), (2, 640), (2, 1024), (3, 64), (3, 128)):
            with G.Solver(G.make_params(dim, n, 8.0, precision=prec, device=dev)) as s:
                s.set_wfc(psi(n, dim))
                s.evolve(3, 0)
""")
    check(launches, "k_step2d")
    check(launches, "k_tstream")


def test_batches_on_clusters(fake):  # noqa: F811
    _, launches = fake("""
for dev in (0, 1):
    for prec, lengths in ((G.PREC_FP64, (64, 128, 256)), (G.PREC_FP32, (64, 192, 320, 384))):
        for count in (1, 9):
            ss = [G.Solver(G.make_params(2, n, 8.0, precision=prec, device=dev))
                  for n in lengths for _ in range(count)]
            for s in ss:
                s.set_wfc(psi(s.params.xDim))
            with G.Batch(ss) as b:
                b.evolve(0, 3)
            for s in ss:
                s.close()
""")
    check(launches, "k_cluster_many")
