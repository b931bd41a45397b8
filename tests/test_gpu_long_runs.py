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
