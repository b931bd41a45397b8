"""An upload that runs out of device memory leaves nothing behind and can be tried again."""
import pytest

from tests import native

# An allocator whose k-th call fails once; host memory stands for the device's
# where there is no GPU.
PROGRAM = r"""
struct Failing : DevAllocator {
    int fail_at, calls = 0, live = 0;
    bool device;
    Failing(int k, bool d) : fail_at(k), device(d) {}
    cudaError_t alloc(void **p, size_t bytes) override {
        if (++calls == fail_at) return cudaErrorMemoryAllocation;
        live++;
        if (device) return cudaMalloc(p, bytes);
        *p = malloc(bytes);
        return cudaSuccess;
    }
    void free(void *p, size_t) override {
        live--;
        if (device) cudaFree(p);
        else ::free(p);
    }
};
static void plan_of(Plan &p, int n) {
    std::vector<Op> ops;
    const double h = std::sqrt(0.5);
    for (int r = 0; r < 3; r++)
        for (int t = 0; t < n; t++) {
            Op o;
            o.target = t;
            o.cmask = o.cval = r == 1 ? uint64_t(1) << ((t + 1) % n) : 0;
            o.m[0] = o.m[1] = o.m[2] = h;
            o.m[3] = -h;
            ops.push_back(o);
        }
    hgm_plan_opts opts;
    hgm_plan_default_opts(&opts, HGM_F32);
    opts.renorm_every = 2;
    if (build_plan(ops, n, opts, &p)) exit(2);
}
int main(int argc, char **argv) {
    const int n = 18, k = atoi(argv[1]);
    const bool device = atoi(argv[2]);
    Failing a(k, device);
    {
        Plan p;
        plan_of(p, n);
        const void *stream = p.tiles[1].stream;
        p.allocator = &a;
        const int first = upload_plan(&p);
        printf("%d %d %d %d %d %d\n", first, a.live, p.d_ops != nullptr, p.d_chain != nullptr, (int)chain_eligible(&p, 1),
               p.tiles[1].stream == stream);
        State s;
        s.qubits = n;
        s.precision = HGM_F32;
        printf("%d\n", launch_plan(&s, &p, 1, nullptr));  // refused, before it looks at the state
        if (device) {
            Plan q;
            plan_of(q, n);
            hgm_state *x, *y;
            double d = -1;
            if (upload_plan(&p) || upload_plan(&q) || hgm_state_create(n, HGM_F32, &x) || hgm_state_create(n, HGM_F32, &y)) return 3;
            hgm_state_set_basis(x, 5);
            hgm_state_set_basis(y, 5);
            if (launch_plan_chain((State *)x, &p, 1, nullptr) || launch_plan((State *)y, &q, 1, nullptr) ||
                hgm_max_abs_diff(x, y, &d))
                return 4;
            printf("%g %d\n", d, a.live);
        }
    }
    printf("%d\n", a.live);
}
"""
NOMEM, INVALID = 3, 1


@pytest.mark.parametrize("k", [1, 2, 3, 4])
def test_failed_allocation(tmp_path, k):
    out = native.run(tmp_path, PROGRAM, k, 0).split("\n")
    assert out[0] == f"{NOMEM} 0 0 0 0 1"
    assert out[1] == str(INVALID)
    assert out[2] == "0"


@pytest.mark.gpu
@pytest.mark.parametrize("k", [1, 2, 3, 4])
def test_second_upload_runs(tmp_path, k):
    """The same plan, chained, against another run pass by pass: the same gates, so FP32 rounding of the norms apart."""
    out = native.run(tmp_path, PROGRAM, k, 1).split("\n")
    assert out[:2] == [f"{NOMEM} 0 0 0 0 1", str(INVALID)]
    d, live = out[2].split()
    # amplitudes below 1; the two orders of a norm's sum differ by less than a few units of 2^-24
    assert float(d) < 1e-6 and live == "4" and out[3] == "0"
