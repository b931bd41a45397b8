// C-ABI of the engine: runtime, plans, device states, execution and
// device-resident measurement (include/hgm_b200.h).
#include <cuda_runtime.h>

#include <cstdlib>

#include <cmath>
#include <cstring>
#include <memory>
#include <mutex>

#include "hgm_dropin_layout.h"
#include "hgm_internal.h"

using namespace hgm;

namespace {

int cuda_fail(cudaError_t e, const char *what) {
    return fail(e == cudaErrorMemoryAllocation ? HGM_ERR_NOMEM : HGM_ERR_CUDA, "%s: %s", what, cudaGetErrorString(e));
}

template <typename Real>
void ops_from_ref_pts(void *const *pts, std::vector<Op> &out) {
    for (long i = 0; pts[i] != nullptr; i++) {
        const RefPTLayout *pt = reinterpret_cast<const RefPTLayout *>(pts[i]);
        const Real *m = reinterpret_cast<const Real *>(pt->matrix);
        Op op;
        op.target = pt->target_bit;
        op.cmask = (uint64_t)pt->control_mask;
        op.cval = (uint64_t)pt->control_value;
        for (int k = 0; k < 4; k++) op.m[k] = cplx((double)m[2 * k], (double)m[2 * k + 1]);
        out.push_back(op);
    }
}

}  // namespace

namespace {
std::mutex g_lease_mu;

void free_plan_now(Plan *pl) {
    // launches are asynchronous: the plan's device records may still be in use
    if (pl->uploaded) cudaDeviceSynchronize();
    delete pl;
}
}  // namespace

namespace hgm {
namespace {

// ---- iterations --------------------------------------------------------------
// A plan run many times cannot merge the last pass of one run with the first
// of the next.  Planned UNROLL times over, it can: a Grover iteration of 18 to
// 26 qubits takes 4.1 passes instead of 5.  Only for states whose passes are
// launches of their own (a chained run's pass costs a few microseconds).
//
// The longer plan is built by the first call of at least UNROLL iterations
// whose own iterations keep the GPU busy meanwhile: as many as cover the
// planning (plan_us; measured 0.35 us an op on the B200's host) at the least
// time their passes can take are queued first, and what is left then runs on
// it.  Where the planning is less than a fiftieth of that time for the whole
// call, it comes first: the iterations queued ahead, and the remainder they
// leave, would lose more merged passes than that (26-qubit FP64 search, first
// call of 32 iterations: 53.5 ms behind queued ones, 51.9 planned first, 57.1 as
// single runs).  A call that cannot cover it, and the calls of fewer
// iterations, run the plan itself.
//
// Of the plan's runs and the longer plan the cheaper serves, by passes,
// transposes and stream units (plan_cost).  Both timed on one B200, eight runs
// against one longer plan: searches of 22 to 27 qubits 0.88-0.92, 26 qubits
// FP32 one layer 0.62, two 0.86, ten 0.97, FP64 three layers 0.80, QFTs without
// their swaps 0.61, random gates 0.35 to 1.04.  Of 49 circuits the rule takes
// the 28 at 0.35 to 0.996 and leaves 21 at 0.92 to 1.04.  A plan that ends in a
// permutation pass (a QFT) stays as it is: within the longer plan its swaps are
// CNOTs again (27 qubits FP32: 101 ms for 32 runs, 208 ms as four longer plans).
constexpr int UNROLL = 8;
constexpr size_t UNROLL_MAX_OPS = 1024;  // beyond, a pass saved is less than 3% of a run
constexpr double PASS_BYTES_PER_US = 6.6e6;

int64_t state_bytes(const Plan *p) { return (int64_t(1) << p->qubits) * (p->precision == HGM_F64 ? 16 : 8); }

// Planning and upload of the longer plan, in us.
double plan_us(const Plan *p) { return 150.0 + 0.5 * UNROLL * (double)p->ops.size(); }

// The least time of one run of the plan, in us.
double run_us(const Plan *p) { return 2.0 * (double)state_bytes(p) / PASS_BYTES_PER_US * (double)p->tiles.size(); }
// Iterations that keep the GPU busy for the planning.
int64_t iterations_ahead(const Plan *p) { return (int64_t)std::ceil(plan_us(p) / run_us(p)); }

// A plan's time in passes over memory: what a pass saved gives back, a
// transpose, and the ops' 16-byte units.
double plan_cost(const Plan *p) {
    return 0.5 * (double)p->tiles.size() + 0.2 * (double)p->n_transposes + 0.03 * (double)(p->stream.size() / 4);
}
bool worth_unrolling(const Plan *p, const Plan *u) {
    return (u->lean || !p->lean) && plan_cost(u) < 0.97 * UNROLL * plan_cost(p);
}

bool can_unroll(const Plan *p, int iterations) {
    return !p->small && !p->ops.empty() && !p->tiles.empty() && iterations >= UNROLL && !(p->tiles.back().flags & PASS_PERMUTE);
}

// The longer plan, if it is ready.
Plan *unrolled_plan(Plan *p, int iterations) {
    if (!can_unroll(p, iterations)) return nullptr;
    std::unique_lock<std::mutex> lk(p->unroll_mu, std::try_to_lock);
    return lk.owns_lock() && p->unrolled && p->unrolled->uploaded ? p->unrolled.get() : nullptr;
}

// Whether this call is to build it: not while another thread does, nor inside
// a capture, which forbids the allocation.
bool may_build(Plan *p, int iterations, cudaStream_t st) {
    if (!can_unroll(p, iterations) || iterations < iterations_ahead(p)) return false;
    std::unique_lock<std::mutex> lk(p->unroll_mu, std::try_to_lock);
    if (!lk.owns_lock() || p->no_unroll || (p->unrolled && p->unrolled->uploaded)) return false;
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(st, &cap) == cudaSuccess && cap == cudaStreamCaptureStatusNone) return true;
    cudaGetLastError();
    return false;
}

// Builds the longer plan.  Without memory for it, it stays planned and a later
// call tries the upload again.
void build_unrolled(Plan *p) {
    std::unique_lock<std::mutex> lk(p->unroll_mu, std::try_to_lock);
    if (!lk.owns_lock() || p->no_unroll) return;
    if (!p->unrolled) {
        std::vector<Op> ops;
        ops.reserve(p->ops.size() * UNROLL);
        for (int k = 0; k < UNROLL; k++) ops.insert(ops.end(), p->ops.begin(), p->ops.end());
        std::unique_ptr<Plan> u(new Plan());
        u->allocator = p->allocator;
        if (build_plan(ops, p->qubits, p->opts, u.get()) || !worth_unrolling(p, u.get())) {
            p->no_unroll = true;
            return;
        }
        p->unrolled = std::move(u);
    }
    OutsideCapture elsewhere;
    upload_plan(p->unrolled.get());
}

}  // namespace

void plan_lease(const Plan *plan) {
    std::lock_guard<std::mutex> lk(g_lease_mu);
    const_cast<Plan *>(plan)->leases++;
}
void plan_unlease(const Plan *plan) {
    Plan *pl = const_cast<Plan *>(plan);
    bool now = false;
    {
        std::lock_guard<std::mutex> lk(g_lease_mu);
        now = --pl->leases == 0 && pl->free_pending;
    }
    if (now) free_plan_now(pl);
}
}  // namespace hgm

extern "C" {

int hgm_init(int device) {
    // The server runs up to 16 streams; with the driver's default of 8
    // hardware queues, two streams share a queue and a long pass on one holds
    // back the other's kernels (served throughput swung between 183 and 264
    // circuits/s with 8, held at 266-268 with 32).  Takes effect only if no
    // CUDA context exists yet in this process; a value the user set stays.
    setenv("CUDA_DEVICE_MAX_CONNECTIONS", "32", 0);
    cudaError_t e = cudaSetDevice(device);
    if (e != cudaSuccess) return cuda_fail(e, "cudaSetDevice");
    e = cudaFree(0);
    if (e != cudaSuccess) return cuda_fail(e, "context init");
    return default_stream() ? HGM_OK : HGM_ERR_CUDA;
}

int hgm_synchronize(void) {
    cudaError_t e = cudaDeviceSynchronize();
    return e == cudaSuccess ? HGM_OK : cuda_fail(e, "cudaDeviceSynchronize");
}

int hgm_pinned_alloc(int64_t bytes, void **out) {
    if (!out || bytes <= 0) return fail(HGM_ERR_INVALID, "bad pinned allocation request");
    cudaError_t e = cudaMallocHost(out, (size_t)bytes);
    return e == cudaSuccess ? HGM_OK : cuda_fail(e, "cudaMallocHost");
}

void hgm_pinned_free(void *p) {
    if (p) cudaFreeHost(p);
}

int hgm_mem_info(int64_t *free_bytes, int64_t *total_bytes) {
    size_t f = 0, t = 0;
    cudaError_t e = cudaMemGetInfo(&f, &t);
    if (e != cudaSuccess) return cuda_fail(e, "cudaMemGetInfo");
    if (free_bytes) *free_bytes = (int64_t)f;
    if (total_bytes) *total_bytes = (int64_t)t;
    return HGM_OK;
}

void hgm_plan_default_opts(hgm_plan_opts *o, int precision) {
    o->precision = precision;
    o->warp_bits = -1;
    o->low_bits = -1;
    o->fuse = 1;
    o->window = 0;
    o->renorm_every = precision == HGM_F32 ? 64 : 0;
    o->chained = 1;
    // both precisions (FP64 saves 2 of 8 instructions per amplitude: 26- to
    // 30-qubit FP64 layered circuits 3-4% faster)
    o->split_layers = 1;
    o->reg_bits = -1;
}

static int finish_plan(const std::vector<Op> &ops, int qubits, const hgm_plan_opts *opts, hgm_plan **out) {
    if (!out) return fail(HGM_ERR_INVALID, "null output");
    hgm_plan_opts o;
    if (opts) o = *opts;
    else hgm_plan_default_opts(&o, HGM_F64);
    if (o.precision != HGM_F64 && o.precision != HGM_F32) return fail(HGM_ERR_INVALID, "bad precision");
    std::unique_ptr<Plan> p(new Plan());
    int rc = build_plan(ops, qubits, o, p.get());
    if (rc) return rc;
    if (p->qubits < 64 && state_bytes(p.get()) > CHAIN_MAX_BYTES && ops.size() <= UNROLL_MAX_OPS) {
        p->ops = ops;
        p->opts = o;
    }
    *out = reinterpret_cast<hgm_plan *>(p.release());
    return HGM_OK;
}

int hgm_plan_create(const hgm_circuit *c, int qubits, const hgm_plan_opts *opts, hgm_plan **out) {
    if (!c) return fail(HGM_ERR_INVALID, "null circuit");
    return finish_plan(reinterpret_cast<const Circuit *>(c)->ops, qubits, opts, out);
}

int hgm_plan_create_from_ref_pts(void *const *pts, int pt_precision, int qubits, const hgm_plan_opts *opts,
                                 hgm_plan **out) {
    if (!pts) return fail(HGM_ERR_INVALID, "null PT list");
    std::vector<Op> ops;
    if (pt_precision == HGM_F64) ops_from_ref_pts<double>(pts, ops);
    else ops_from_ref_pts<float>(pts, ops);
    return finish_plan(ops, qubits, opts, out);
}


void hgm_plan_free(hgm_plan *p) {
    Plan *pl = reinterpret_cast<Plan *>(p);
    if (!pl) return;
    {
        // a plan that queued server requests still use is freed by the last of them
        std::lock_guard<std::mutex> lk(g_lease_mu);
        if (pl->leases > 0) {
            pl->free_pending = true;
            return;
        }
    }
    free_plan_now(pl);
}

int hgm_plan_upload(hgm_plan *p) {
    if (!p) return fail(HGM_ERR_INVALID, "null plan");
    return upload_plan(reinterpret_cast<Plan *>(p));
}

int hgm_plan_stats(const hgm_plan *p, int64_t *n_ops, int64_t *n_passes, int64_t *n_phases, int64_t *n_transposes) {
    if (!p) return fail(HGM_ERR_INVALID, "null plan");
    const Plan *pl = reinterpret_cast<const Plan *>(p);
    if (n_ops) *n_ops = pl->n_ops;
    if (n_passes) *n_passes = pl->small ? (pl->n_small_ops ? 1 : 0) : (int64_t)pl->passes.size();
    if (n_phases) *n_phases = (int64_t)pl->phases.size();
    if (n_transposes) *n_transposes = pl->n_transposes;
    return HGM_OK;
}

int hgm_plan_layouts(const hgm_plan *p, const int8_t **pos, int64_t *n_layouts) {
    const Plan *pl = reinterpret_cast<const Plan *>(p);
    if (!pl) return fail(HGM_ERR_INVALID, "null plan");
    if (pos) *pos = pl->layouts.empty() ? nullptr : pl->layouts[0].pos;
    if (n_layouts) *n_layouts = (int64_t)pl->layouts.size();
    return HGM_OK;
}

int hgm_plan_export(const hgm_plan *p, const void **passes, int64_t *n_passes, const void **phases,
                    int64_t *n_phases, const void **ops, int64_t *ops_bytes, int *warp_bits, int *small) {
    if (!p) return fail(HGM_ERR_INVALID, "null plan");
    const Plan *pl = reinterpret_cast<const Plan *>(p);
    if (passes) *passes = pl->passes.data();
    if (n_passes) *n_passes = (int64_t)pl->passes.size();
    if (phases) *phases = pl->phases.data();
    if (n_phases) *n_phases = (int64_t)pl->phases.size();
    if (ops) *ops = pl->ops_bytes.data();
    if (ops_bytes) *ops_bytes = (int64_t)pl->ops_bytes.size();
    if (warp_bits) *warp_bits = pl->warp_bits;
    if (small) *small = pl->small ? 1 : 0;
    return HGM_OK;
}

int hgm_plan_stream(const hgm_plan *p, const void **units, int64_t *bytes, const void **tiles, int64_t *n_tiles) {
    if (!p) return fail(HGM_ERR_INVALID, "null plan");
    const Plan *pl = reinterpret_cast<const Plan *>(p);
    const bool small = pl->small;
    if (units) *units = small ? (const void *)pl->ops_bytes.data() : (const void *)pl->stream.data();
    if (bytes) *bytes = small ? (int64_t)pl->ops_bytes.size() : (int64_t)(pl->stream.size() * sizeof(uint32_t));
    if (tiles) *tiles = pl->tiles.data();
    if (n_tiles) *n_tiles = (int64_t)pl->tiles.size();
    return HGM_OK;
}

int hgm_state_create(int qubits, int precision, hgm_state **out) {
    if (!out) return fail(HGM_ERR_INVALID, "null output");
    if (qubits < 1 || qubits > 34) return fail(HGM_ERR_UNSUPPORTED, "qubits=%d outside 1..34", qubits);
    if (precision != HGM_F64 && precision != HGM_F32) return fail(HGM_ERR_INVALID, "bad precision");
    if (!default_stream()) return HGM_ERR_CUDA;
    std::unique_ptr<State> s(new State());
    s->qubits = qubits;
    s->precision = precision;
    cudaError_t e = cudaMalloc(&s->d, (size_t)s->bytes());
    if (e != cudaSuccess) {
        cudaGetLastError();
        return cuda_fail(e, "state allocation");
    }
    *out = reinterpret_cast<hgm_state *>(s.release());
    return HGM_OK;
}

void hgm_state_free(hgm_state *s) {
    State *st = reinterpret_cast<State *>(s);
    if (!st || !st->owned) return;  // views are released by their owner
    if (st->d) {
        cudaDeviceSynchronize();  // work queued on the state may still be running
        cudaFree(st->d);
    }
    delete st;
}

int hgm_state_qubits(const hgm_state *s) { return s ? reinterpret_cast<const State *>(s)->qubits : 0; }
int hgm_state_precision(const hgm_state *s) { return s ? reinterpret_cast<const State *>(s)->precision : -1; }
void *hgm_state_device_ptr(hgm_state *s) { return s ? reinterpret_cast<State *>(s)->d : nullptr; }

int hgm_state_set_basis(hgm_state *s, int64_t index) {
    if (!s) return fail(HGM_ERR_INVALID, "null state");
    return launch_set_basis(reinterpret_cast<State *>(s), index, nullptr);
}

int hgm_state_upload(hgm_state *s, const void *host, int64_t bytes) {
    State *st = reinterpret_cast<State *>(s);
    if (!st || !host) return fail(HGM_ERR_INVALID, "null argument");
    if (bytes != st->bytes()) return fail(HGM_ERR_INVALID, "upload of %lld bytes into a %lld-byte state",
                                          (long long)bytes, (long long)st->bytes());
    return copy_state(st->d, host, (size_t)bytes, true, default_stream());
}

int hgm_state_download(const hgm_state *s, void *host, int64_t bytes) {
    const State *st = reinterpret_cast<const State *>(s);
    if (!st || !host) return fail(HGM_ERR_INVALID, "null argument");
    if (bytes != st->bytes()) return fail(HGM_ERR_INVALID, "download of %lld bytes from a %lld-byte state",
                                          (long long)bytes, (long long)st->bytes());
    return copy_state(host, st->d, (size_t)bytes, false, default_stream());
}

int hgm_execute(hgm_state *s, const hgm_plan *p, int iterations, void *stream) {
    if (!s || !p) return fail(HGM_ERR_INVALID, "null argument");
    if (iterations < 0) return fail(HGM_ERR_INVALID, "negative iterations");
    Plan *pl = const_cast<Plan *>(reinterpret_cast<const Plan *>(p));
    int rc = upload_plan(pl);
    if (rc) return rc;
    if (iterations == 0) return HGM_OK;
    // a state that fits in L2 runs every pass in one chained launch
    if (plan_launches(pl, iterations) > 1 && chain_eligible(pl, iterations))
        return launch_plan_chain(reinterpret_cast<State *>(s), pl, iterations, stream);
    // the plan, the longer plan and the plan again, as one sequence of passes
    State *st = reinterpret_cast<State *>(s);
    PlanCursor c;
    c.norms = (double *)pl->d_norm;
    auto run = [&](const Plan *q, int times, int then) {
        iterations = then;
        c.more = then > 0;
        const int err = launch_plan_steps(st, q, times, &c, plan_launches(q, times), stream);
        c.then_plan();
        return err;
    };
    Plan *u = unrolled_plan(pl, iterations);
    if (!u && may_build(pl, iterations, (cudaStream_t)(stream ? stream : default_stream()))) {
        const int ahead = 50.0 * plan_us(pl) <= iterations * run_us(pl) ? 0 : (int)iterations_ahead(pl);
        if (ahead && (rc = run(pl, ahead, iterations - ahead))) return rc;
        build_unrolled(pl);
        u = unrolled_plan(pl, iterations);
    }
    if (u && (rc = run(u, iterations / UNROLL, iterations % UNROLL))) return rc;
    return iterations ? run(pl, iterations, 0) : HGM_OK;
}

int hgm_plan_status(const hgm_plan *p) {
    if (!p) return fail(HGM_ERR_INVALID, "null plan");
    const Plan *pl = reinterpret_cast<const Plan *>(p);
    const void *w = chain_error_word(pl);
    if (!w) return HGM_OK;
    uint64_t err = 0;
    cudaError_t e = cudaDeviceSynchronize();
    if (e == cudaSuccess) e = cudaMemcpy(&err, w, sizeof err, cudaMemcpyDeviceToHost);
    if (e != cudaSuccess) return cuda_fail(e, "plan status");
    return err ? fail(HGM_ERR_TIMEOUT, "a chained pass gave up waiting for the passes before it") : HGM_OK;
}

int hgm_norm(hgm_state *s, double *out) {
    if (!s) return fail(HGM_ERR_INVALID, "null state");
    return reduce_norm(reinterpret_cast<State *>(s), out, nullptr);
}

int hgm_prob_one(hgm_state *s, int bit, double *out) {
    if (!s) return fail(HGM_ERR_INVALID, "null state");
    return reduce_prob_one(reinterpret_cast<State *>(s), bit, out, nullptr);
}

int hgm_measure_qubit(hgm_state *s, int qubit, double sample, int *outcome, double *prob) {
    State *st = reinterpret_cast<State *>(s);
    if (!st) return fail(HGM_ERR_INVALID, "null state");
    if (qubit < 0 || qubit >= st->qubits) return fail(HGM_ERR_INVALID, "qubit %d outside state", qubit);
    const int bit = st->qubits - 1 - qubit;
    double total = 0, one = 0;
    int rc = reduce_split(st, bit, &total, &one, nullptr);
    if (rc) return rc;
    const double zero = total - one;
    // DGM::measure: outcome 0 iff P(0) > sample (dgm_core.cpp:97-113)
    const int value = (zero > sample) ? 0 : 1;
    const double p = value ? one : zero;
    if (!(p > 0)) return fail(HGM_ERR_INVALID, "measured outcome has zero probability");
    // the measured branch, rescaled, moves to the qubit's |0> half
    // (dgm_core.cpp:117-122)
    rc = measure_update(st, bit, value, 1.0 / std::sqrt(p), nullptr);
    if (rc) return rc;
    if (outcome) *outcome = value;
    if (prob) *prob = p;
    return HGM_OK;
}

int hgm_collapse_qubit(hgm_state *s, int qubit, int value, double *prob) {
    State *st = reinterpret_cast<State *>(s);
    if (!st) return fail(HGM_ERR_INVALID, "null state");
    if (qubit < 0 || qubit >= st->qubits) return fail(HGM_ERR_INVALID, "qubit %d outside state", qubit);
    if (value != 0 && value != 1) return fail(HGM_ERR_INVALID, "value %d is not 0 or 1", value);
    const int bit = st->qubits - 1 - qubit;
    double total = 0, one = 0;
    int rc = reduce_split(st, bit, &total, &one, nullptr);
    if (rc) return rc;
    const double p = value ? one : total - one;
    if (!(p > 0)) return fail(HGM_ERR_INVALID, "collapse onto a value of zero probability");
    // DGM::colapse (dgm_core.cpp:129-146): keep the amplitudes whose qubit has
    // `value`, divide them by sqrt of their probability, clear the rest
    rc = collapse(st, bit, value, 1.0 / std::sqrt(p), nullptr);
    if (rc) return rc;
    if (prob) *prob = p;
    return HGM_OK;
}

int hgm_marginal_probs(hgm_state *s, uint64_t mask, double *out, int64_t count) {
    State *st = reinterpret_cast<State *>(s);
    if (!st || !out) return fail(HGM_ERR_INVALID, "null argument");
    const int m = __builtin_popcountll(mask);
    if (m > 62 || count != (int64_t(1) << m))
        return fail(HGM_ERR_INVALID, "output holds %lld values, the mask needs 2^%d", (long long)count, m);
    return marginal_probs(st, mask, out, nullptr);
}

int hgm_marginal_argmax(hgm_state *s, uint64_t mask, int64_t *arg, double *prob) {
    if (!s) return fail(HGM_ERR_INVALID, "null state");
    return marginal_argmax(reinterpret_cast<State *>(s), mask, arg, prob, nullptr);
}

int hgm_inner(hgm_state *a, hgm_state *b, double *re, double *im) {
    if (!a || !b) return fail(HGM_ERR_INVALID, "null state");
    return inner(reinterpret_cast<State *>(a), reinterpret_cast<State *>(b), re, im, nullptr);
}

int hgm_max_abs_diff(hgm_state *a, hgm_state *b, double *out) {
    if (!a || !b) return fail(HGM_ERR_INVALID, "null state");
    return max_abs_diff(reinterpret_cast<State *>(a), reinterpret_cast<State *>(b), out, nullptr);
}

int hgm_scale(hgm_state *s, double f) {
    if (!s) return fail(HGM_ERR_INVALID, "null state");
    return scale_state(reinterpret_cast<State *>(s), f, nullptr);
}

}  // extern "C"
