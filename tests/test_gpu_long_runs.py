"""What a call of many iterations keeps to, whichever plans it runs on (engine.cpp, iterations)."""
import threading

import pytest

from simulador_quantico_b200 import workloads as wl
from tests import native

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


def test_longer_plan_is_built_beside_another_threads_capture(sq):
    """A thread captures in the global mode, which refuses other threads' allocations: the call's result is that of
    single runs and the capture stays whole."""
    torch = pytest.importorskip("torch")
    n = 22
    plan = sq.Plan(one_iteration(n, 4242).build(sq.Circuit()), n, "f64").upload()
    a, b = sq.State(n, "f64").set_basis(1), sq.State(n, "f64").set_basis(1)
    x = torch.zeros(1024, device="cuda")
    for _ in range(24):
        b.execute(plan)
    sq.synchronize()
    failed = []

    def call():
        try:
            a.execute(plan, 24)
        except Exception as e:
            failed.append(e)

    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=torch.cuda.Stream(), capture_error_mode="global"):
        x.add_(1.0)
        t = threading.Thread(target=call)
        t.start()
        t.join()
        x.add_(1.0)
    g.replay()
    torch.cuda.synchronize()
    assert not failed and float(x.sum()) == 2048.0
    # 24 iterations of 2 n gates rounded in another order
    assert a.max_abs_diff(b) < 1e-14
    l0 = sq.kernel_launches()
    a.execute(plan, 24)
    assert sq.kernel_launches() - l0 == 3 * 33  # built in that first call


RETRY = r"""
struct Failing : DevAllocator {
    int fail_at, calls = 0;
    cudaError_t alloc(void **p, size_t bytes) override {
        return ++calls == fail_at ? cudaErrorMemoryAllocation : cudaMalloc(p, bytes);
    }
    void free(void *p, size_t) override { cudaFree(p); }
};
int main() {
    const int n = 22;
    hgm_circuit *c = hgm_circuit_new();
    const double s = std::sqrt(0.5), h[8] = {s, 0, s, 0, s, 0, -s, 0}, z[8] = {1, 0, 0, 0, 0, 0, -1, 0};
    for (int side = 0; side < 2; side++) {
        hgm_circuit_append_op(c, 0, ((int64_t(1) << n) - 1) ^ 1, side ? 6 : 0, z);
        for (int t = 0; t < n; t++) hgm_circuit_append_op(c, t, 0, 0, h);
    }
    hgm_plan *p;
    hgm_plan_opts o;
    hgm_plan_default_opts(&o, HGM_F64);
    if (hgm_plan_create(c, n, &o, &p)) return 2;
    Failing a;
    a.fail_at = 2;  // the plan's own stream is the first, the longer plan's the second
    reinterpret_cast<Plan *>(p)->allocator = &a;
    hgm_state *x;
    if (hgm_state_create(n, HGM_F64, &x) || hgm_state_set_basis(x, 0)) return 3;
    for (int k = 0; k < 3; k++) {
        const int64_t l0 = hgm_kernel_launches();
        if (hgm_execute(x, p, 64, nullptr)) return 4;
        printf("%d ", (int)(hgm_kernel_launches() - l0));
    }
    double norm = 0;
    if (hgm_norm(x, &norm)) return 5;
    printf("%d\n", std::abs(norm - 1.0) < 1e-12);
    hgm_plan_free(p);
}
"""


def test_no_memory_for_the_longer_plan_is_not_for_good(tmp_path):
    first, second, third, ok = native.run(tmp_path, RETRY).split()
    assert int(third) <= int(second) < int(first) and ok == "1"


def test_first_long_call_queues_its_own_iterations_first(sq):
    """The longer plan is planned while the GPU runs the call's first iterations; it serves the rest."""
    n, iterations = 22, 24
    plan = sq.Plan(one_iteration(n, 5).build(sq.Circuit()), n, "f64").upload()
    assert plan.stats()["passes"] == 5
    st = sq.State(n, "f64").set_basis(0)
    l0 = sq.kernel_launches()
    st.execute(plan, iterations)
    first = sq.kernel_launches() - l0
    assert first in [5 * a + 33 * ((24 - a) // 8) + 5 * ((24 - a) % 8) for a in range(1, 17)]
    st.execute(plan, iterations)
    assert sq.kernel_launches() - l0 - first == 3 * 33


def test_long_first_call_runs_on_the_longer_plan_at_once(sq):
    """Planning is a hundredth of the call's 26 ms: no iteration is run ahead of it."""
    n = 25
    plan = sq.Plan(one_iteration(n, 5).build(sq.Circuit()), n, "f64").upload()
    st = sq.State(n, "f64").set_basis(0)
    for _ in range(2):
        l0 = sq.kernel_launches()
        st.execute(plan, 32)
        assert sq.kernel_launches() - l0 == 4 * 33
    st.free()


def one_by_one(sq, circuit, n, prec, iterations):
    """Launches of `iterations` runs, twice; checks them against single runs."""
    plan = sq.Plan(circuit, n, prec).upload()
    a, b = sq.State(n, prec).set_basis(3), sq.State(n, prec).set_basis(3)
    launches = []
    for _ in range(2):
        l0 = sq.kernel_launches()
        a.execute(plan, iterations)
        launches.append(sq.kernel_launches() - l0)
        for _ in range(iterations):
            b.execute(plan)
    # unitary gates on a unit state, rounded in another order: growth with the
    # square root of the gates in a row at most, 2 x 24 x 300 of them
    assert a.max_abs_diff(b) < (1e-13 if prec == "f64" else 2e-5)
    a.free()
    b.free()
    return launches, plan.stats()["passes_run"] * iterations


@pytest.mark.parametrize("n,prec", [(22, "f64"), (23, "f32")])
def test_runs_that_end_in_swaps_stay_single(sq, n, prec):
    """Only the last of eight QFTs could end in a permutation pass."""
    launches, single = one_by_one(sq, wl.qft(n, 0).build(sq.Circuit()), n, prec, 24)
    assert launches == [single, single]


@pytest.mark.parametrize("layers,longer", [(2, True), (20, False)])
def test_plans_are_compared_by_their_time(sq, layers, longer):
    """Two layers merge over runs; twenty are as many gates in as many passes, and more planning than the runs cover."""
    launches, single = one_by_one(sq, wl.random_layered(23, layers, 3).build(sq.Circuit()), 23, "f32", 24)
    assert (launches[1] < single) == longer and launches[0] <= single
