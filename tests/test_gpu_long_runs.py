"""What a call of many iterations keeps to, whichever plans it runs on (engine.cpp, iterations)."""
import pytest

from simulador_quantico_b200 import workloads as wl

pytestmark = pytest.mark.gpu


def one_iteration(n, seed):
    g = wl.grover_search(n, seed, 1)
    return wl.CircuitSpec("one", n, 0, g.gates, [g.calls[1]])


@pytest.mark.parametrize("renorm_every,norm", [(50, 1.0), (1000, 4.0)])
def test_renormalisation_counts_through_the_call(sq, renorm_every, norm):
    """15 iterations take at least 66 passes, eight of them planned as one 33: the 50th falls after those."""
    n = 24
    plan = sq.Plan(one_iteration(n, 777).build(sq.Circuit()), n, "f32", renorm_every=renorm_every).upload()
    assert plan.stats()["passes"] == 5
    st = sq.State(n, "f32").set_basis(3)
    st.scale(2.0)
    for _ in range(2):  # the call that builds the longer plan, and one that has it
        l0 = sq.kernel_launches()
        st.execute(plan, 15)
        assert 66 <= sq.kernel_launches() - l0 <= 75
    # 150 passes of FP32 rounding
    assert abs(st.norm() - norm) < 1e-4 * norm
    st.free()
