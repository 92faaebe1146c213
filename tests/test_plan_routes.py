"""A 2D context that was given a line plan (gpue_set_plan) steps as line passes until
gpue_autotune chooses for it again, and then on the resident steppers as one that never
was.  CPU test over the fake CUDA runtime (fake_cudart.cpp), by the kernels launched."""
import pytest

from fake_device import fake  # noqa: F401


@pytest.mark.parametrize("prec", ["FP32", "FP64"])
@pytest.mark.parametrize("n,kernel", [(64, "k_cluster_one"), (256, "k_step2d")])
def test_autotune_ends_a_plan_set_by_hand(fake, prec, n, kernel):  # noqa: F811
    def kinds(calls):
        _, launches = fake("""
with G.Solver(G.make_params(2, %d, 8.0, precision=G.PREC_%s)) as s:
    s.set_wfc(psi(%d))
    q = s.plan(0)
    %s
    s.evolve(3, 1)
""" % (n, prec, n, calls))
        last = [q["kernel"] for q in launches if "k_norm" not in q["kernel"] and
                "k_convert" not in q["kernel"] and "k_scale" not in q["kernel"]]
        return kernel in last[-1]

    plan = 's.set_plan(0, q["ra"], q["rb"], q["rc"], q["threads_per_line"])'
    assert kinds("pass")
    assert not kinds(plan)
    assert kinds(plan + "; s.autotune()")
    assert not kinds("s.autotune(); " + plan)
