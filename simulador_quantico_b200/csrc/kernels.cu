// Kernels and launchers of the state-vector engine (sm_100a).
//
//   pass_kernel<Real, W>   one state pass of a plan (kernels.cuh: run_tile)
//   permute_kernel<Real>   a plan's final swaps as one pass
//   chain_kernel<Real, W>  every pass of a small state in one launch
//   small_kernel<Real>     states of < 10 qubits: whole state in one CTA's
//                          shared memory, gates applied one by one
//   reduce_*               FP64 reductions (norm, bit probability, inner
//                          product, max |difference|) with a fixed grid and a
//                          fixed combine order, so a result does not depend
//                          on what else runs on the device
//   collapse / scale / set_basis / marginal argmax
#include <cuda_runtime.h>

#include <atomic>
#include <cstdio>
#include <mutex>
#include <type_traits>

#include "kernels.cuh"

namespace hgm {

// ---------------------------------------------------------------------------
// context: one library stream, a small scratch area for reductions
// ---------------------------------------------------------------------------

namespace {
constexpr int RED_BLOCKS = REDUCE_SCRATCH_BLOCKS;   // 8 x 148 SMs
constexpr int RED_THREADS = 256;
constexpr size_t MARGINAL_SCRATCH = (MARG_SUMS + (size_t(1) << 16)) * sizeof(double);

struct Ctx {
    int device = -1;
    cudaStream_t stream = nullptr;
    cudaStream_t upload = nullptr; // plan uploads
    double *partials = nullptr;    // RED_BLOCKS * 2 doubles
    long long *partial_idx = nullptr;
    double *host_result = nullptr; // 4 doubles (pinned; kernels write it)
    double *marginal = nullptr;    // MARGINAL_SCRATCH bytes
    cudaEvent_t t0 = nullptr, t1 = nullptr;
};
Ctx g_ctx;
std::mutex g_ctx_mu;
// held by a synchronous reduction while it uses the context's scratch
std::mutex g_reduce_mu;
std::atomic<long long> g_launches{0};
}  // namespace

void count_launch(int n) { g_launches += n; }

static int ensure_ctx() {
    if (g_ctx.stream) return HGM_OK;
    std::lock_guard<std::mutex> lk(g_ctx_mu);
    if (g_ctx.stream) return HGM_OK;
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return fail(HGM_ERR_CUDA, "cudaGetDevice: %s", cudaGetErrorString(e));
    g_ctx.device = dev;
    cudaStream_t s;
    if ((e = cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking)) != cudaSuccess)
        return fail(HGM_ERR_CUDA, "cudaStreamCreate: %s", cudaGetErrorString(e));
    if ((e = cudaStreamCreateWithFlags(&g_ctx.upload, cudaStreamNonBlocking)) != cudaSuccess ||
        (e = cudaMalloc(&g_ctx.partials, RED_BLOCKS * 2 * sizeof(double))) != cudaSuccess ||
        (e = cudaMalloc(&g_ctx.partial_idx, RED_BLOCKS * sizeof(long long))) != cudaSuccess ||
        (e = cudaMalloc(&g_ctx.marginal, MARGINAL_SCRATCH)) != cudaSuccess ||
        (e = cudaMallocHost(&g_ctx.host_result, 4 * sizeof(double))) != cudaSuccess ||
        (e = cudaEventCreate(&g_ctx.t0)) != cudaSuccess || (e = cudaEventCreate(&g_ctx.t1)) != cudaSuccess)
        return fail(HGM_ERR_CUDA, "context setup: %s", cudaGetErrorString(e));
    g_ctx.stream = s;
    return HGM_OK;
}

void *default_stream() {
    if (ensure_ctx() != HGM_OK) return nullptr;
    return g_ctx.stream;
}

static inline cudaStream_t pick(void *stream) {
    return stream ? (cudaStream_t)stream : (cudaStream_t)default_stream();
}

static inline int check(const char *what) {
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return fail(HGM_ERR_CUDA, "%s: %s", what, cudaGetErrorString(e));
    return HGM_OK;
}

// Launches a kernel that calls wait_for_kernel_before: it may start while the
// kernel before it on the stream still runs.  set_basis and a one-tile pass: 8.2
// -> 6.7 us; 23-qubit FP32 layered passes (55 us each) 3%, QFT 4% faster.
template <typename... Params, typename... Args>
static cudaError_t launch_behind(void (*kernel)(Params...), unsigned grid, unsigned block, size_t smem, cudaStream_t st,
                                 Args &&...args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, static_cast<Params>(args)...);
}

// ---------------------------------------------------------------------------
// pass kernels
// ---------------------------------------------------------------------------

template <typename Real, int R, int W, bool LEAN>
__global__ void __launch_bounds__(32 << W) __maxnreg__((pass_max_regs<Real, R>()))
    pass_kernel(typename V2<Real>::T *__restrict__ state, const __grid_constant__ TileArgs ta) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    fetch_stream<W>(smem_raw + tile_smem_bytes<Real, R, W>(), ta);
    wait_for_kernel_before();
    let_next_kernel_start();
    run_tile<Real, R, W, LEAN, false>(state, ta, blockIdx.x, smem_raw, ta.ctl);
}

// A permutation pass over a large state, one sub-tile a block.
constexpr int PERM_THREADS = 128;
template <typename Real>
__global__ void __launch_bounds__(PERM_THREADS) permute_kernel(typename V2<Real>::T *__restrict__ state,
                                                               const __grid_constant__ TileArgs ta) {
    __shared__ typename V2<Real>::T sm[2 * PERM_SLOTS];
    wait_for_kernel_before();
    let_next_kernel_start();
    permute_subtile<Real, PERM_THREADS>(state, ta, blockIdx.x, sm, ta.ctl);
}

template <typename Real>
__global__ void __launch_bounds__(256) small_kernel(typename V2<Real>::T *__restrict__ state, int n,
                                                    const SmallOp<Real> *__restrict__ ops, long long n_ops,
                                                    int iterations) {
    using A2 = typename V2<Real>::T;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    A2 *sm = reinterpret_cast<A2 *>(smem_raw);
    const int N = 1 << n, half = N >> 1;
    wait_for_kernel_before();
    let_next_kernel_start();
    for (int i = threadIdx.x; i < N; i += blockDim.x) sm[i] = state[i];
    __syncthreads();
    for (int it = 0; it < iterations; it++) {
        for (long long k = 0; k < n_ops; k++) {
            const SmallOp<Real> &o = ops[k];
            const int t = o.target;
            const uint32_t cm = o.cmask, cv = o.cval;
            const Real m0r = o.m[0], m0i = o.m[1], m1r = o.m[2], m1i = o.m[3];
            const Real m2r = o.m[4], m2i = o.m[5], m3r = o.m[6], m3i = o.m[7];
            for (int p = threadIdx.x; p < half; p += blockDim.x) {
                const int i0 = ((p >> t) << (t + 1)) | (p & ((1 << t) - 1));
                const int i1 = i0 | (1 << t);
                if (((uint32_t)i0 & cm) != cv) continue;
                const A2 x = sm[i0], y = sm[i1];
                A2 o0, o1;
                o0.x = m0r * x.x - m0i * x.y + m1r * y.x - m1i * y.y;
                o0.y = m0r * x.y + m0i * x.x + m1r * y.y + m1i * y.x;
                o1.x = m2r * x.x - m2i * x.y + m3r * y.x - m3i * y.y;
                o1.y = m2r * x.y + m2i * x.x + m3r * y.y + m3i * y.x;
                sm[i0] = o0;
                sm[i1] = o1;
            }
            __syncthreads();
        }
    }
    for (int i = threadIdx.x; i < N; i += blockDim.x) state[i] = sm[i];
}

template <typename Real, int R, int W, bool LEAN>
static int setup_pass_kernel() {
    static bool done = false;
    if (done) return HGM_OK;
    const int smem = cta_smem_bytes<Real, R, W>();
    cudaError_t e =
        cudaFuncSetAttribute(pass_kernel<Real, R, W, LEAN>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e == cudaSuccess && HGM_SMEM_CARVEOUT >= 0)
        e = cudaFuncSetAttribute(pass_kernel<Real, R, W, LEAN>, cudaFuncAttributePreferredSharedMemoryCarveout,
                                 HGM_SMEM_CARVEOUT);
    if (e != cudaSuccess) return fail(HGM_ERR_CUDA, "cudaFuncSetAttribute: %s", cudaGetErrorString(e));
    done = true;
    return HGM_OK;
}

template <typename Real, int R, int W, bool LEAN>
static int launch_pass(void *state, const TileArgs &pa, cudaStream_t st) {
    using A2 = typename V2<Real>::T;
    int rc = setup_pass_kernel<Real, R, W, LEAN>();
    if (rc) return rc;
    const uint64_t tiles = 1ull << (pa.n - pa.k);
    const int smem = cta_smem_bytes<Real, R, W>() - 2 * (STREAM_WINDOW_BYTES - window_bytes<W>(pa));
    const cudaError_t e = launch_behind(pass_kernel<Real, R, W, LEAN>, (unsigned)tiles, 32 << W, smem, st,
                                        reinterpret_cast<A2 *>(state), pa);
    if (e != cudaSuccess) return fail(HGM_ERR_CUDA, "pass_kernel launch: %s", cudaGetErrorString(e));
    count_launch();
    return HGM_OK;
}

// FP64 tiles hold 16 amplitudes a thread (R = 4), FP32 tiles 32 (R = 5) or,
// on request, 16 (plan_reg_bits).
template <typename Real, int R, bool LEAN>
static int launch_pass_w(int W, void *state, const TileArgs &pa, cudaStream_t st) {
    switch (W) {
        case 0: return launch_pass<Real, R, 0, LEAN>(state, pa, st);
        case 1: return launch_pass<Real, R, 1, LEAN>(state, pa, st);
        case 2: return launch_pass<Real, R, 2, LEAN>(state, pa, st);
        default: return launch_pass<Real, R, 3, LEAN>(state, pa, st);
    }
}
template <typename Real, int R>
static int launch_pass_lw(bool lean, int W, void *state, const TileArgs &pa, cudaStream_t st) {
    return lean ? launch_pass_w<Real, R, true>(W, state, pa, st) : launch_pass_w<Real, R, false>(W, state, pa, st);
}

template <typename Real>
static int launch_small(State *s, const Plan *p, int iterations, cudaStream_t st) {
    const int smem = (1 << s->qubits) * (int)sizeof(typename V2<Real>::T);
    const cudaError_t e = launch_behind(small_kernel<Real>, 1, 256, smem, st, reinterpret_cast<typename V2<Real>::T *>(s->d),
                                        s->qubits, reinterpret_cast<const SmallOp<Real> *>(p->d_ops), p->n_small_ops,
                                        iterations);
    count_launch();
    return e == cudaSuccess ? HGM_OK : fail(HGM_ERR_CUDA, "small_kernel launch: %s", cudaGetErrorString(e));
}

int launch_plan_steps(State *s, const Plan *p, int iterations, PlanCursor *c, int64_t max_launches, void *stream) {
    if (s->qubits != p->qubits) return fail(HGM_ERR_INVALID, "plan is for %d qubits, state has %d", p->qubits, s->qubits);
    if (s->precision != p->precision) return fail(HGM_ERR_INVALID, "plan and state precision differ");
    // every device pointer a launch passes must exist: an op list that was
    // never uploaded is refused here, not read through a null pointer
    if (!p->uploaded) return fail(HGM_ERR_INVALID, "plan used before upload_plan");
    cudaStream_t st = pick(stream);
    if (!st) return HGM_ERR_CUDA;
    if (p->small) {
        if (c->next > 0 || max_launches < 1) return HGM_OK;
        c->next = 1;
        return p->n_small_ops ? (p->precision == HGM_F64 ? launch_small<double>(s, p, iterations, st)
                                                         : launch_small<float>(s, p, iterations, st))
                              : HGM_OK;
    }
    const int64_t np = (int64_t)p->tiles.size();
    const int R = p->renorm_every;
    const int64_t total = np * iterations;
    for (int64_t k = 0; k < max_launches && c->next < total; k++, c->next++) {
        const int64_t g = c->next;
        TileArgs pa = p->tiles[g % np];
        if (c->scale_in) {
            pa.ctl.flags |= PASS_SCALE;
            pa.ctl.scale_in = c->scale_in;
            c->scale_in = nullptr;
        }
        if (R > 0 && (c->before + g + 1) % R == 0 && (c->more || g + 1 < total)) {
            if (!c->norms) c->norms = (double *)p->d_norm;
            pa.ctl.flags |= PASS_NORM;
            pa.ctl.norm_out = c->norms + c->slot;
            cudaMemsetAsync(pa.ctl.norm_out, 0, sizeof(double), st);
            c->scale_in = pa.ctl.norm_out;
            c->slot = (c->slot + 1) % 64;
        }
        if (pa.flags & PASS_PERMUTE) {
            const unsigned grid = 1u << (pa.n - PERM_BITS);
            const cudaError_t e = p->precision == HGM_F64
                                      ? launch_behind(permute_kernel<double>, grid, PERM_THREADS, 0, st, (double2 *)s->d, pa)
                                      : launch_behind(permute_kernel<float>, grid, PERM_THREADS, 0, st, (float2 *)s->d, pa);
            if (e != cudaSuccess) return fail(HGM_ERR_CUDA, "permute_kernel launch: %s", cudaGetErrorString(e));
            count_launch();
            continue;
        }
        int rc = p->precision == HGM_F64
                     ? launch_pass_lw<double, HGM_F64_REG_BITS>(p->lean, p->warp_bits, s->d, pa, st)
                 : p->reg_bits == 4 ? launch_pass_lw<float, 4>(p->lean, p->warp_bits, s->d, pa, st)
                                    : launch_pass_lw<float, HGM_F32_REG_BITS>(p->lean, p->warp_bits, s->d, pa, st);
        if (rc) return rc;
    }
    return check("pass_kernel launch");
}

int64_t plan_launches(const Plan *p, int iterations) {
    return p->small ? 1 : (int64_t)p->tiles.size() * iterations;
}

// ---------------------------------------------------------------------------
// chained passes: every pass of a small state in one persistent launch
// ---------------------------------------------------------------------------
// A state that fits in L2 moves through a pass in a few microseconds, so
// launching one kernel per pass leaves it bound by launch latency and the
// tail of each launch.  The chained kernel runs the whole pass sequence in
// one launch.  Its CTAs claim work items (pass g, tile t) in sequence order
// from a counter, and the CTA that claimed an item of pass g waits until
// every item of passes 0..g-1 is done (a second counter) before it loads.
//
// Between two passes a CTA only waits for what the next pass needs: one thread
// claims the next item while another publishes this one, and the arguments and
// the stream of the pass the CTA will probably run next (it takes every
// stride-th item when no other kernel is in the way) are fetched before its
// item is known.  (Claiming an item ahead does the same, but holds it back
// from idle CTAs: the serving mix, whose launches share the SMs, lost 5%.)
// An item only waits for items claimed before it, and a claimed item is held
// by a running CTA, so the sequence always progresses whether or not all of
// the grid is resident.  The wait is bounded (2 s of %globaltimer); a CTA that
// gives up sets the error word and skips its tile.
//
// Scratch (Plan::d_chain): claim counter, done counter, error word, exit
// counter, then CHAIN_NORM_SLOTS FP64 norm slots used in turn, so that a
// sequence of any length (many iterations of a short FP32 plan) runs chained.
// The last CTA to leave zeroes all but the error word for the next launch (no
// memset in front of it: 2 us a call); the holder of item 0 clears the error
// word, which nothing can set before a wait of 2 s has run out.
// Renormalisation k accumulates into slot k % CHAIN_NORM_SLOTS during pass
// (k + 1) * renorm - 1 and is read during the next pass; tile 0 of the pass
// before an accumulating pass zeroes its slot before counting itself done, so
// the zero is seen by every tile of that pass (they wait for the count) and
// comes after the slot's previous reads (three slots: CHAIN_NORM_SLOTS *
// renorm > 2 passes apart).
constexpr unsigned long long CHAIN_WAIT_LIMIT_NS = 2000000000ull;
constexpr int CHAIN_NORM_SLOTS = 3;

__device__ __forceinline__ unsigned long long chain_now_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

__device__ __forceinline__ unsigned long long ld_acquire_u64(const unsigned long long *p) {
    unsigned long long v;
    asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}

template <typename Real, int R, int W, bool LEAN>
__global__ void __launch_bounds__(32 << W) __maxnreg__((pass_max_regs<Real, R>()))
    chain_kernel(typename V2<Real>::T *__restrict__ state, const TileArgs *__restrict__ passes, int npasses,
                 int tile_bits, long long total, int renorm, unsigned long long *ctr, double *norms) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    unsigned char *win = smem_raw + tile_smem_bytes<Real, R, W>();
    // The sequence's state is kept in shared memory by thread 0: in registers
    // it would be live through every tile.  g modulo the plan's passes and the
    // renormalisation period are stepped along with g (64-bit divisions for
    // each item took a microsecond).
    struct Place {
        long long g;
        int pass, phase, slot;
    };
    __shared__ Place s_at, s_guess;
    __shared__ long long s_it, s_next;
    __shared__ PassCtl s_ctl;
    __shared__ int s_skip, s_fetched, s_refetch, s_cur;
    // the arguments of this item's pass and of the guessed next one: the tile
    // code reads them many times (the tile-bit map byte by byte)
    __shared__ __align__(16) TileArgs s_ta[2];
    const long long seq = total >> tile_bits;  // passes in the sequence
    auto fetch_args = [&](TileArgs *dst, int pass) {
        fetch_units(reinterpret_cast<unsigned char *>(dst), reinterpret_cast<const uint4 *>(passes + pass),
                    (int)(sizeof(TileArgs) / 16));
    };
    auto step_to = [&](Place p, long long g) {
        for (; p.g < g; p.g++) {
            if (++p.pass == npasses) p.pass = 0;
            if (renorm > 0 && ++p.phase == renorm) {
                p.phase = 0;
                if (++p.slot == CHAIN_NORM_SLOTS) p.slot = 0;
            }
        }
        return p;
    };
    // most CTAs' first item belongs to the first pass
    fetch_args(&s_ta[0], 0);
    fetch_wait();
    __syncthreads();
    fetch_stream<W>(win, s_ta[0]);
    if (threadIdx.x == 0) {
        s_next = (long long)atomicAdd(&ctr[0], 1ull);
        s_at.g = s_next >> tile_bits;
        s_at.pass = (int)(s_at.g % npasses);
        s_at.phase = renorm > 0 ? (int)(s_at.g % renorm) : 0;
        s_at.slot = renorm > 0 ? (int)(s_at.g / renorm % CHAIN_NORM_SLOTS) : 0;
        s_guess = s_at;
        s_guess.pass = 0;  // what is fetched
        s_fetched = 1;
        s_cur = 1;
    }
    for (;;) {
        // thread 0: the item claimed below (thread 0 itself before the first turn)
        __syncthreads();
        if (threadIdx.x == 0) {
            const long long it = s_next;
            const int here = s_fetched ? s_guess.pass : s_at.pass;  // the pass that is fetched
            const Place at = step_to(s_at, it >> tile_bits);
            const long long g = at.g;
            s_it = it;
            s_at = at;
            s_cur ^= s_fetched;
            s_refetch = at.pass != here;
            if (it < total) {
                // the pass of the item this CTA will probably claim next
                const Place guess = step_to(at, (it + gridDim.x) >> tile_bits);
                s_guess = guess;
                s_fetched = guess.g < seq && guess.pass != at.pass;
                // the plain launcher's schedule: a norm on every renorm-th
                // pass but the last, a rescale on the pass after it
                int32_t flags = 0;
                if (renorm > 0) {
                    if (at.phase + 1 == renorm && g + 1 < seq) flags |= PASS_NORM;
                    if (at.phase == 0 && g > 0) flags |= PASS_SCALE;
                    s_ctl.norm_out = norms + at.slot;
                    s_ctl.scale_in = norms + (at.slot ? at.slot - 1 : CHAIN_NORM_SLOTS - 1);
                }
                s_ctl.flags = flags;
                int skip = 0;
                const unsigned long long need = (unsigned long long)(g << tile_bits);
                if (it == 0) ctr[2] = 0ull;
                if (ld_acquire_u64(&ctr[1]) < need) {
                    const unsigned long long t0 = chain_now_ns();
                    while (ld_acquire_u64(&ctr[1]) < need) {
                        if (chain_now_ns() - t0 > CHAIN_WAIT_LIMIT_NS) {
                            atomicExch(&ctr[2], 1ull);
                            skip = 1;
                            break;
                        }
                        __nanosleep(32);
                    }
                }
                s_skip = skip;
            }
        }
        __syncthreads();
        if (s_it >= total) break;
        if (s_refetch) {  // guessed wrong
            fetch_wait();
            __syncthreads();
            fetch_args(&s_ta[s_cur], s_at.pass);
            fetch_wait();
            __syncthreads();
            fetch_stream<W>(win, s_ta[s_cur]);
        }
        if (s_fetched) fetch_args(&s_ta[s_cur ^ 1], s_guess.pass);
        if (!s_skip)
            run_tile<Real, R, W, LEAN, true>(state, s_ta[s_cur], (uint64_t)(s_it & ((1ll << tile_bits) - 1)), smem_raw,
                                             s_ctl);
        fetch_wait();  // the guessed pass's arguments
        __syncthreads();
        if (threadIdx.x == blockDim.x - 1) s_next = (long long)atomicAdd(&ctr[0], 1ull);
        fetch_stream<W>(win, s_ta[s_cur ^ s_fetched]);
        if (threadIdx.x == 0) {
            // the next pass accumulates a norm: zero its slot first
            if (renorm > 0 && (s_it & ((1ll << tile_bits) - 1)) == 0 && s_at.g + 2 < seq) {
                const int slot = s_at.slot;
                const bool wrap = s_at.phase + 2 > renorm;  // the next pass is in the next period
                if (wrap ? renorm == 1 : s_at.phase + 2 == renorm)
                    norms[wrap ? (slot + 1 == CHAIN_NORM_SLOTS ? 0 : slot + 1) : slot] = 0.0;
            }
            __threadfence();
            atomicAdd(&ctr[1], 1ull);
        }
    }
    fetch_wait();
    if (threadIdx.x == 0) {
        __threadfence();
        if (atomicAdd(&ctr[3], 1ull) + 1 == gridDim.x) {
            ctr[0] = 0ull;
            ctr[1] = 0ull;
            ctr[3] = 0ull;
            if (renorm > 0)
                for (int k = 0; k < CHAIN_NORM_SLOTS; k++) norms[k] = 0.0;
        }
    }
}

template <typename Real, int R, int W, bool LEAN>
static int launch_chain_rw(State *s, const Plan *p, int iterations, cudaStream_t st) {
    using A2 = typename V2<Real>::T;
    static int grid_cap = 0;
    const int smem = cta_smem_bytes<Real, R, W>();
    if (!grid_cap) {
        cudaError_t e = cudaFuncSetAttribute(chain_kernel<Real, R, W, LEAN>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        int per_sm = 0, dev = 0, sms = 0;
        if (e == cudaSuccess) e = cudaGetDevice(&dev);
        if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, chain_kernel<Real, R, W, LEAN>, 32 << W, smem);
        if (e != cudaSuccess || per_sm < 1) return fail(HGM_ERR_CUDA, "chain kernel setup: %s", cudaGetErrorString(e));
        grid_cap = sms * per_sm;
    }
    const int tile_bits = p->qubits - p->tiles[0].k;
    const long long total = ((long long)p->tiles.size() * iterations) << tile_bits;
    const long long ntiles = 1ll << tile_bits;
    const unsigned grid = (unsigned)(ntiles < grid_cap ? ntiles : grid_cap);
    unsigned long long *ctr = reinterpret_cast<unsigned long long *>(p->d_chain);
    double *norms = reinterpret_cast<double *>(ctr + 4);
    // not launch_behind: CTAs that start while the kernel before still holds
    // some SMs crowd onto the others and stay there for every pass (20-qubit
    // layered: 148 -> 224 us)
    chain_kernel<Real, R, W, LEAN><<<grid, 32 << W, smem, st>>>(reinterpret_cast<A2 *>(s->d),
                                                          reinterpret_cast<const TileArgs *>(p->d_chain_passes),
                                                          (int)p->tiles.size(), tile_bits, total, p->renorm_every,
                                                          ctr, norms);
    count_launch();
    return check("chain_kernel launch");
}

template <typename Real, int R, bool LEAN>
static int launch_chain_lw(State *s, const Plan *p, int iterations, cudaStream_t st) {
    switch (p->warp_bits) {
        case 0: return launch_chain_rw<Real, R, 0, LEAN>(s, p, iterations, st);
        case 1: return launch_chain_rw<Real, R, 1, LEAN>(s, p, iterations, st);
        case 2: return launch_chain_rw<Real, R, 2, LEAN>(s, p, iterations, st);
        default: return launch_chain_rw<Real, R, 3, LEAN>(s, p, iterations, st);
    }
}
template <typename Real, int R>
static int launch_chain_w(State *s, const Plan *p, int iterations, cudaStream_t st) {
    return p->lean ? launch_chain_lw<Real, R, true>(s, p, iterations, st)
                   : launch_chain_lw<Real, R, false>(s, p, iterations, st);
}

bool chain_eligible(const Plan *p, int iterations) {
    return p->uploaded && !p->small && p->d_chain && p->tiles.size() >= 2 && iterations >= 1;
}

int launch_plan_chain(State *s, const Plan *p, int iterations, void *stream) {
    if (s->qubits != p->qubits || s->precision != p->precision)
        return fail(HGM_ERR_INVALID, "plan and state differ in size or precision");
    if (!chain_eligible(p, iterations)) return fail(HGM_ERR_INVALID, "plan not set up for chained passes");
    cudaStream_t st = pick(stream);
    if (!st) return HGM_ERR_CUDA;
    if (p->precision == HGM_F64) return launch_chain_w<double, HGM_F64_REG_BITS>(s, p, iterations, st);
    return p->reg_bits == 4 ? launch_chain_w<float, 4>(s, p, iterations, st)
                            : launch_chain_w<float, HGM_F32_REG_BITS>(s, p, iterations, st);
}

// Error word of the last chained run of `p` (device address, for an
// asynchronous copy after the run).
const void *chain_error_word(const Plan *p) {
    return p->d_chain ? reinterpret_cast<const unsigned long long *>(p->d_chain) + 2 : nullptr;
}

int launch_plan(State *s, const Plan *p, int iterations, void *stream) {
    PlanCursor c;
    return launch_plan_steps(s, p, iterations, &c, plan_launches(p, iterations), stream);
}

// ---------------------------------------------------------------------------
// plan upload
// ---------------------------------------------------------------------------

static void *&plan_block(Plan *p, int k) {
    if (k == 0) return p->d_ops;
    if (k == 1) return p->d_norm;
    return k == 2 ? p->d_chain : p->d_chain_passes;
}

static void release_blocks(Plan *p) {
    for (int k = 0; k < 4; k++) {
        void *&d = plan_block(p, k);
        if (!d) continue;
        if (p->allocator) p->allocator->free(d, p->d_bytes[k]);
        else cudaFree(d);
        d = nullptr;
    }
}

Plan::~Plan() { release_blocks(this); }

// Allocates the plan's device memory and copies it there.  On failure the
// caller releases what was allocated.
static int upload_blocks(Plan *p) {
    const int64_t state_bytes = (int64_t(1) << p->qubits) * (p->precision == HGM_F64 ? 16 : 8);
    const bool chain = p->chained && !p->small && p->tiles.size() >= 2 && state_bytes <= CHAIN_MAX_BYTES;
    p->chain_slots = chain && p->renorm_every > 0 ? CHAIN_NORM_SLOTS : 0;
    const size_t bytes[4] = {
        p->small ? p->ops_bytes.size() : p->stream.size() * sizeof(uint32_t),
        p->renorm_every > 0 ? 64 * sizeof(double) : 0,
        chain ? (4 + (size_t)p->chain_slots) * sizeof(double) : 0,
        chain ? p->tiles.size() * sizeof(TileArgs) : 0,
    };
    if (!bytes[0] && !bytes[1]) return HGM_OK;  // a plan without gates
    static const char *const what[4] = {"plan ops", "plan norm slots", "plan chain scratch", "plan chain passes"};
    cudaError_t e;
    for (int k = 0; k < 4; k++) {
        if (!bytes[k]) continue;
        p->d_bytes[k] = bytes[k];
        void *&d = plan_block(p, k);
        if ((e = p->allocator ? p->allocator->alloc(&d, bytes[k]) : cudaMalloc(&d, bytes[k])) != cudaSuccess) {
            d = nullptr;
            return fail(HGM_ERR_NOMEM, "%s: %s", what[k], cudaGetErrorString(e));
        }
    }
    if (ensure_ctx()) return HGM_ERR_CUDA;
    // the passes with their streams' device addresses; the plan keeps the
    // offsets until the upload is complete, so that it can be tried again
    std::vector<TileArgs> tiles = p->tiles;
    for (TileArgs &t : tiles)
        if (!(t.flags & PASS_PERMUTE)) t.stream = (const unsigned char *)p->d_ops + reinterpret_cast<size_t>(t.stream);
    const void *const src[4] = {p->small ? (const void *)p->ops_bytes.data() : (const void *)p->stream.data(), nullptr,
                                nullptr, tiles.data()};
    for (int k = 0; k < 4; k++)
        if (bytes[k] && src[k] &&
            (e = cudaMemcpyAsync(plan_block(p, k), src[k], bytes[k], cudaMemcpyHostToDevice, g_ctx.upload)) != cudaSuccess)
            return fail(HGM_ERR_CUDA, "%s copy: %s", what[k], cudaGetErrorString(e));
    // zero for the first launch; every launch leaves it so
    if (chain && (e = cudaMemsetAsync(p->d_chain, 0, bytes[2], g_ctx.upload)) != cudaSuccess)
        return fail(HGM_ERR_CUDA, "plan chain scratch: %s", cudaGetErrorString(e));
    // the plan's launches go to other streams, which do not wait for the copies.
    // (Not the legacy stream: it takes no work while a blocking stream captures.)
    if ((e = cudaStreamSynchronize(g_ctx.upload)) != cudaSuccess)
        return fail(HGM_ERR_CUDA, "plan upload: %s", cudaGetErrorString(e));
    p->tiles.swap(tiles);
    return HGM_OK;
}

int upload_plan(Plan *p) {
    if (p->uploaded) return HGM_OK;
    const int rc = upload_blocks(p);
    if (rc) {  // nothing half done: a later call starts over, and no launch finds some of the memory
        if (g_ctx.upload) cudaStreamSynchronize(g_ctx.upload);  // copies into it may be under way
        release_blocks(p);
        cudaGetLastError();
        return rc;
    }
    p->uploaded = true;
    return HGM_OK;
}

// ---------------------------------------------------------------------------
// elementwise kernels
// ---------------------------------------------------------------------------

// Zeroes the state, four 16-byte stores a thread in a block's run of 16 KiB,
// the one amplitude among them.
// Bound by writing the state: 4 GiB 617 us, 6.96 TB/s, where one amplitude a
// thread and turn took 720 us; 1 GiB FP32 153 against 180 us.
constexpr int BASIS_VECS = 4;
template <typename Real>
__global__ void __launch_bounds__(256) set_basis_kernel(typename V2<Real>::T *s, long long N, long long index) {
    let_next_kernel_start();
    constexpr long long PER = 16 / (long long)sizeof(typename V2<Real>::T);  // amplitudes a store
    const long long vecs = N / PER;
    auto *v = reinterpret_cast<std::conditional_t<PER == 1, double2, float4> *>(s);
    for (long long b = blockIdx.x * 256ll * BASIS_VECS; b < vecs; b += (long long)gridDim.x * 256 * BASIS_VECS) {
#pragma unroll
        for (int k = 0; k < BASIS_VECS; k++) {
            const long long i = b + k * 256 + threadIdx.x;
            if (i >= vecs) break;
            if constexpr (PER == 1) v[i] = make_double2(i == index ? 1.0 : 0.0, 0.0);
            else v[i] = make_float4(2 * i == index ? 1.0f : 0.0f, 0.0f, 2 * i + 1 == index ? 1.0f : 0.0f, 0.0f);
        }
    }
}

template <typename Real>
__global__ void collapse_kernel(typename V2<Real>::T *s, long long N, int bit, int value, double inv_norm) {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < N; i += (long long)gridDim.x * blockDim.x) {
        typename V2<Real>::T v = s[i];
        if ((int)((i >> bit) & 1) == value) {
            v.x = (Real)(v.x * inv_norm);
            v.y = (Real)(v.y * inv_norm);
        } else {
            v.x = 0;
            v.y = 0;
        }
        s[i] = v;
    }
}

// DGM::measure(int)'s state update (src/core/dgm_core.cpp:117-122): for every
// pair of indices differing only in `bit`, the amplitude of the measured
// branch, rescaled, goes to the bit-0 index and the bit-1 index is cleared,
// so the measured qubit is left in |0> whichever value was read.  One thread
// per pair: the pair's two amplitudes are read before either is written.
template <typename Real>
__global__ void measure_update_kernel(typename V2<Real>::T *s, long long half, int bit, int value, double inv_norm) {
    const long long low = (1ll << bit) - 1;
    for (long long p = blockIdx.x * (long long)blockDim.x + threadIdx.x; p < half; p += (long long)gridDim.x * blockDim.x) {
        const long long i0 = ((p & ~low) << 1) | (p & low), i1 = i0 | (1ll << bit);
        typename V2<Real>::T v = s[value ? i1 : i0], z;
        v.x = (Real)(v.x * inv_norm);
        v.y = (Real)(v.y * inv_norm);
        z.x = 0;
        z.y = 0;
        s[i0] = v;
        s[i1] = z;
    }
}

template <typename Real>
__global__ void scale_kernel(typename V2<Real>::T *s, long long N, double f) {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < N; i += (long long)gridDim.x * blockDim.x) {
        typename V2<Real>::T v = s[i];
        v.x = (Real)(v.x * f);
        v.y = (Real)(v.y * f);
        s[i] = v;
    }
}

static unsigned grid_for(long long N) {
    long long g = (N + 255) / 256;
    return (unsigned)(g < RED_BLOCKS ? (g < 1 ? 1 : g) : RED_BLOCKS);
}

int launch_set_basis(State *s, int64_t index, void *stream) {
    cudaStream_t st = pick(stream);
    if (!st) return HGM_ERR_CUDA;
    long long N = 1ll << s->qubits;
    if (index < 0 || index >= N) return fail(HGM_ERR_INVALID, "basis index %lld outside state", (long long)index);
    const long long blocks = (s->bytes() / 16 + 256 * BASIS_VECS - 1) / (256 * BASIS_VECS);
    const unsigned g = (unsigned)(blocks < 8 * RED_BLOCKS ? blocks : 8 * RED_BLOCKS);
    if (s->precision == HGM_F64) set_basis_kernel<double><<<g, 256, 0, st>>>((double2 *)s->d, N, index);
    else set_basis_kernel<float><<<g, 256, 0, st>>>((float2 *)s->d, N, index);
    count_launch();
    return check("set_basis");
}

int collapse(State *s, int bit, int value, double inv_norm, void *stream) {
    cudaStream_t st = pick(stream);
    long long N = 1ll << s->qubits;
    if (s->precision == HGM_F64) collapse_kernel<double><<<grid_for(N), 256, 0, st>>>((double2 *)s->d, N, bit, value, inv_norm);
    else collapse_kernel<float><<<grid_for(N), 256, 0, st>>>((float2 *)s->d, N, bit, value, inv_norm);
    count_launch();
    return check("collapse");
}

int measure_update(State *s, int bit, int value, double inv_norm, void *stream) {
    cudaStream_t st = pick(stream);
    const long long half = 1ll << (s->qubits - 1);
    if (s->precision == HGM_F64)
        measure_update_kernel<double><<<grid_for(half), 256, 0, st>>>((double2 *)s->d, half, bit, value, inv_norm);
    else
        measure_update_kernel<float><<<grid_for(half), 256, 0, st>>>((float2 *)s->d, half, bit, value, inv_norm);
    count_launch();
    return check("measure update");
}

int scale_state(State *s, double f, void *stream) {
    cudaStream_t st = pick(stream);
    long long N = 1ll << s->qubits;
    if (s->precision == HGM_F64) scale_kernel<double><<<grid_for(N), 256, 0, st>>>((double2 *)s->d, N, f);
    else scale_kernel<float><<<grid_for(N), 256, 0, st>>>((float2 *)s->d, N, f);
    count_launch();
    return check("scale");
}

// ---------------------------------------------------------------------------
// FP64 reductions (fixed grid, fixed combine order)
// ---------------------------------------------------------------------------

// RED_SPLIT: the norm and, of it, the share where `bit` is 1, in one read
enum RedMode { RED_NORM = 0, RED_PROB1 = 1, RED_INNER = 2, RED_MAXDIFF = 3, RED_SPLIT = 4 };

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
    for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
__device__ __forceinline__ double warp_max(double v) {
#pragma unroll
    for (int o = 16; o; o >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}

template <typename RA, typename RB, int MODE>
__global__ void __launch_bounds__(RED_THREADS) reduce_kernel(const typename V2<RA>::T *__restrict__ a,
                                                              const typename V2<RB>::T *__restrict__ b, long long N,
                                                              int bit, double *partials) {
    double s0 = 0.0, s1 = 0.0;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < N; i += (long long)gridDim.x * blockDim.x) {
        const typename V2<RA>::T x = a[i];
        if (MODE == RED_NORM) {
            s0 += (double)x.x * x.x + (double)x.y * x.y;
        } else if (MODE == RED_PROB1) {
            if ((i >> bit) & 1) s0 += (double)x.x * x.x + (double)x.y * x.y;
        } else if (MODE == RED_SPLIT) {
            const double q = (double)x.x * x.x + (double)x.y * x.y;
            s0 += q;
            if ((i >> bit) & 1) s1 += q;
        } else if (MODE == RED_INNER) {
            const typename V2<RB>::T y = b[i];
            // conj(x) * y
            s0 += (double)x.x * y.x + (double)x.y * y.y;
            s1 += (double)x.x * y.y - (double)x.y * y.x;
        } else {
            const typename V2<RB>::T y = b[i];
            const double dr = (double)x.x - (double)y.x, di = (double)x.y - (double)y.y;
            s0 = fmax(s0, sqrt(dr * dr + di * di));
        }
    }
    __shared__ double sh[2][RED_THREADS / 32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    if (MODE == RED_MAXDIFF) s0 = warp_max(s0);
    else {
        s0 = warp_sum(s0);
        s1 = warp_sum(s1);
    }
    if (lane == 0) {
        sh[0][w] = s0;
        sh[1][w] = s1;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        double t0 = 0.0, t1 = 0.0;
        for (int k = 0; k < RED_THREADS / 32; k++) {
            if (MODE == RED_MAXDIFF) t0 = fmax(t0, sh[0][k]);
            else t0 += sh[0][k];
            t1 += sh[1][k];
        }
        partials[2 * blockIdx.x] = t0;
        partials[2 * blockIdx.x + 1] = t1;
    }
}

// Combines the block partials: one block, each thread its strided share, then
// the warps' sums, in a fixed order.  (One thread walking the 1184 partials
// alone took 82 us, twice the 41 us that reading a 256 MiB state takes; this
// takes 5 us.)
template <int MODE>
__global__ void __launch_bounds__(RED_THREADS) reduce_final(const double *partials, int nblocks, double *out,
                                                            int n_out) {
    double t0 = 0.0, t1 = 0.0;
    for (int k = threadIdx.x; k < nblocks; k += RED_THREADS) {
        if (MODE == RED_MAXDIFF) t0 = fmax(t0, partials[2 * k]);
        else t0 += partials[2 * k];
        t1 += partials[2 * k + 1];
    }
    if (MODE == RED_MAXDIFF) t0 = warp_max(t0);
    else t0 = warp_sum(t0);
    t1 = warp_sum(t1);
    __shared__ double sh[2][RED_THREADS / 32];
    if ((threadIdx.x & 31) == 0) {
        sh[0][threadIdx.x >> 5] = t0;
        sh[1][threadIdx.x >> 5] = t1;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        t0 = t1 = 0.0;
        for (int k = 0; k < RED_THREADS / 32; k++) {
            if (MODE == RED_MAXDIFF) t0 = fmax(t0, sh[0][k]);
            else t0 += sh[0][k];
            t1 += sh[1][k];
        }
        out[0] = t0;
        if (n_out > 1) out[1] = t1;
    }
}

// Synchronous reductions share the context's scratch and its page-locked
// result words, which the last kernel writes itself (no copy behind it).
template <typename RA, typename RB, int MODE>
static int run_reduce(const void *a, const void *b, int qubits, int bit, double *o0, double *o1, cudaStream_t st) {
    const long long N = 1ll << qubits;
    const unsigned g = grid_for(N);
    std::lock_guard<std::mutex> lk(g_reduce_mu);
    reduce_kernel<RA, RB, MODE><<<g, RED_THREADS, 0, st>>>((const typename V2<RA>::T *)a,
                                                           (const typename V2<RB>::T *)b, N, bit, g_ctx.partials);
    reduce_final<MODE><<<1, RED_THREADS, 0, st>>>(g_ctx.partials, (int)g, g_ctx.host_result, 2);
    count_launch(2);
    int rc = check("reduction launch");
    cudaError_t e = cudaStreamSynchronize(st);
    if (rc) return rc;
    if (e != cudaSuccess) return fail(HGM_ERR_CUDA, "reduction: %s", cudaGetErrorString(e));
    if (o0) *o0 = g_ctx.host_result[0];
    if (o1) *o1 = g_ctx.host_result[1];
    return HGM_OK;
}

int launch_norm_async(State *s, double *partials, double *out, void *stream) {
    cudaStream_t st = (cudaStream_t)stream;
    const long long N = 1ll << s->qubits;
    const unsigned g = grid_for(N);
    if (s->precision == HGM_F64)
        reduce_kernel<double, double, RED_NORM><<<g, RED_THREADS, 0, st>>>((const double2 *)s->d, nullptr, N, 0, partials);
    else
        reduce_kernel<float, float, RED_NORM><<<g, RED_THREADS, 0, st>>>((const float2 *)s->d, nullptr, N, 0, partials);
    reduce_final<RED_NORM><<<1, RED_THREADS, 0, st>>>(partials, (int)g, out, 2);
    count_launch(2);
    return check("norm reduction launch");
}

int reduce_norm(State *s, double *out, void *stream) {
    cudaStream_t st = pick(stream);
    if (!st) return HGM_ERR_CUDA;
    return s->precision == HGM_F64 ? run_reduce<double, double, RED_NORM>(s->d, nullptr, s->qubits, 0, out, nullptr, st)
                                   : run_reduce<float, float, RED_NORM>(s->d, nullptr, s->qubits, 0, out, nullptr, st);
}

int reduce_prob_one(State *s, int bit, double *out, void *stream) {
    cudaStream_t st = pick(stream);
    if (!st) return HGM_ERR_CUDA;
    if (bit < 0 || bit >= s->qubits) return fail(HGM_ERR_INVALID, "bit %d outside state", bit);
    return s->precision == HGM_F64 ? run_reduce<double, double, RED_PROB1>(s->d, nullptr, s->qubits, bit, out, nullptr, st)
                                   : run_reduce<float, float, RED_PROB1>(s->d, nullptr, s->qubits, bit, out, nullptr, st);
}

int reduce_split(State *s, int bit, double *total, double *one, void *stream) {
    cudaStream_t st = pick(stream);
    if (!st) return HGM_ERR_CUDA;
    if (bit < 0 || bit >= s->qubits) return fail(HGM_ERR_INVALID, "bit %d outside state", bit);
    return s->precision == HGM_F64 ? run_reduce<double, double, RED_SPLIT>(s->d, nullptr, s->qubits, bit, total, one, st)
                                   : run_reduce<float, float, RED_SPLIT>(s->d, nullptr, s->qubits, bit, total, one, st);
}

template <int MODE>
static int two_state(State *a, State *b, double *o0, double *o1, cudaStream_t st) {
    if (a->qubits != b->qubits) return fail(HGM_ERR_INVALID, "states differ in size");
    if (a->precision == HGM_F64 && b->precision == HGM_F64)
        return run_reduce<double, double, MODE>(a->d, b->d, a->qubits, 0, o0, o1, st);
    if (a->precision == HGM_F64) return run_reduce<double, float, MODE>(a->d, b->d, a->qubits, 0, o0, o1, st);
    if (b->precision == HGM_F64) return run_reduce<float, double, MODE>(a->d, b->d, a->qubits, 0, o0, o1, st);
    return run_reduce<float, float, MODE>(a->d, b->d, a->qubits, 0, o0, o1, st);
}

int inner(State *a, State *b, double *re, double *im, void *stream) {
    cudaStream_t st = pick(stream);
    if (!st) return HGM_ERR_CUDA;
    return two_state<RED_INNER>(a, b, re, im, st);
}

int max_abs_diff(State *a, State *b, double *out, void *stream) {
    cudaStream_t st = pick(stream);
    if (!st) return HGM_ERR_CUDA;
    return two_state<RED_MAXDIFF>(a, b, out, nullptr, st);
}

// ---- marginals ---------------------------------------------------------------
// For every value x of the bits in `mask` (bit j of x is the j-th lowest mask
// bit), p(x) = sum over the other bits of |a|^2; either all of them
// (DGM::measure(vector), src/core/dgm_core.cpp:150-162) or the x with the
// largest p (lowest on ties).
//
// A block reads whole runs of the lowest 11 index bits (16 KiB FP32, 32 KiB
// FP64): lanes and warps are bits 0..7, each thread's eight accumulators bits
// 8..10, so loads are contiguous whatever the mask is and eight are in flight
// a thread.  A unit is one value of the mask bits above those and one of `nch`
// equal chunks of the other high bits; the block walks the chunk by adding to
// a masked index, ((c | ~mask) + 1) & mask, which steps through the deposited
// values without depositing bits one by one.  At the unit's end the sums are
// folded over the accumulators, lanes and warps whose bit is outside the
// mask, always in the same order.
// Bound by reading the state once.  25 qubits FP32, 11 bits: 52 us, 5.2 TB/s (one
// thread per value before, 8 blocks, a bit deposit per element: 17.9 ms; a
// block's warps on scattered 256-byte runs: 113 us, waiting on DRAM).  The
// argmax over all 25 bits: 1064 us before, now 42-45 us (6 TB/s).  The plain
// sums of an FP32 state keep to 32 registers (eight blocks an SM): with 40 the
// reading of 28 qubits takes 368 us instead of 347.
constexpr int MARG_WARPS = RED_THREADS / 32;
constexpr int MARG_LOW = 11, MARG_ACC = 8;

__device__ __forceinline__ unsigned long long deposit_bits(unsigned long long v, unsigned long long mask) {
    unsigned long long out = 0;
    while (mask) {
        const unsigned long long low = mask & (0ull - mask);
        if (v & 1ull) out |= low;
        v >>= 1;
        mask ^= low;
    }
    return out;
}

// The better of two (probability, value) candidates: the larger probability,
// then the lower value; a NaN never wins.
__device__ __forceinline__ void keep_best(double &p, long long &i, double q, long long j) {
    if (q > p || (q == p && j < i)) {
        p = q;
        i = j;
    }
}

// Block-wide best; the result is valid in thread 0.
__device__ __forceinline__ void block_best(double &p, long long &i) {
#pragma unroll
    for (int o = 16; o; o >>= 1) {
        const double q = __shfl_xor_sync(0xffffffffu, p, o);
        const long long j = __shfl_xor_sync(0xffffffffu, i, o);
        keep_best(p, i, q, j);
    }
    __shared__ double sp[MARG_WARPS];
    __shared__ long long si[MARG_WARPS];
    if ((threadIdx.x & 31) == 0) {
        sp[threadIdx.x >> 5] = p;
        si[threadIdx.x >> 5] = i;
    }
    __syncthreads();
    if (threadIdx.x == 0)
        for (int k = 1; k < MARG_WARPS; k++) keep_best(p, i, sp[k], si[k]);
}

// ARGMAX: block b's best to pbest[b], ibest[b] (nch must be 1); otherwise value
// x's sum over chunk c to out[c * M + x], M values in all.
template <typename Real, bool ARGMAX>
__global__ void __launch_bounds__(RED_THREADS) marginal_kernel(const typename V2<Real>::T *__restrict__ s, int n,
                                                                unsigned long long mask, int nch, long long M, double *out,
                                                                double *pbest, long long *ibest) {
    const int tid = threadIdx.x;
    const int lb = n < MARG_LOW ? n : MARG_LOW, nh = n - lb;
    const uint32_t mlo = (uint32_t)mask & ((1u << lb) - 1u);
    const unsigned long long mhi = mask >> lb, chi = ~mhi & ((1ull << nh) - 1ull);
    const int m_lo = __popc(mlo);
    const long long units = (1ll << __popcll(mhi)) * nch, count = (1ll << __popcll(chi)) / nch;
    const int accs = lb > 8 ? 1 << (lb - 8) : 1;  // accumulators in use
    const bool live = tid < (1 << lb);
    __shared__ double sh[MARG_ACC][RED_THREADS];
    double best = -1.0;
    long long besti = 0;
    for (long long u = blockIdx.x; u < units; u += gridDim.x) {
        const long long xh = u / nch, chunk = u % nch;
        const unsigned long long hi = deposit_bits((unsigned long long)xh, mhi);
        unsigned long long c = deposit_bits((unsigned long long)(chunk * count), chi);
        double p[MARG_ACC];
#pragma unroll
        for (int k = 0; k < MARG_ACC; k++) p[k] = 0.0;
        if (accs == MARG_ACC) {
#pragma unroll 2
            for (long long j = 0; j < count; j++) {
                const typename V2<Real>::T *__restrict__ src = s + ((hi | c) << MARG_LOW) + tid;
#pragma unroll
                for (int k = 0; k < MARG_ACC; k++) {
                    const typename V2<Real>::T v = __ldcs(src + k * RED_THREADS);
                    p[k] += (double)v.x * v.x + (double)v.y * v.y;
                }
                c = ((c | ~chi) + 1ull) & chi;
            }
        } else if (live) {  // a state of fewer than 11 qubits: one run
            for (int k = 0; k < accs; k++) {
                const typename V2<Real>::T v = s[tid + k * RED_THREADS];
                const double q = (double)v.x * v.x + (double)v.y * v.y;
#pragma unroll
                for (int r = 0; r < MARG_ACC; r++)
                    if (r == k) p[r] = q;
            }
        }
        // fold over the accumulators, lanes and warps outside the mask; an
        // unused accumulator, lane or warp holds zero
#pragma unroll
        for (int b = 0; b < 3; b++)
            if (!((mlo >> (8 + b)) & 1u)) {
#pragma unroll
                for (int k = 0; k < MARG_ACC; k++)
                    if (!(k & (1 << b))) p[k] += p[k | (1 << b)];
            }
        for (int b = 0; b < 5; b++)
            if (!((mlo >> b) & 1u)) {
#pragma unroll
                for (int k = 0; k < MARG_ACC; k++) p[k] += __shfl_xor_sync(0xffffffffu, p[k], 1 << b);
            }
#pragma unroll
        for (int k = 0; k < MARG_ACC; k++) sh[k][tid] = p[k];
        __syncthreads();
        const uint32_t over = ~mlo & 0xe0u;  // warp bits outside the mask
        if (live && !((uint32_t)tid & ~mlo)) {
            for (int k = 0; k < accs; k++) {
                if (((uint32_t)k << 8) & ~mlo) continue;
                double t = 0.0;
                uint32_t w = 0;
                do {
                    t += sh[k][(uint32_t)tid | w];
                    w = ((w | ~over) + 1u) & over;
                } while (w);
                uint32_t xl = 0;  // this run position's mask bits, packed
                const uint32_t pos = (uint32_t)tid | ((uint32_t)k << 8);
                for (uint32_t m = mlo, j = 0; m; m &= m - 1, j++) xl |= ((pos >> (__ffs((int)m) - 1)) & 1u) << j;
                const long long x = (xh << m_lo) | xl;
                if (ARGMAX) keep_best(best, besti, t, x);
                else out[chunk * M + x] = t;
            }
        }
        __syncthreads();
    }
    if (ARGMAX) {
        block_best(best, besti);
        if (threadIdx.x == 0) {
            pbest[blockIdx.x] = best;
            ibest[blockIdx.x] = besti;
        }
    }
}

// Argmax over every index bit (a search without ancilla): no sums, one
// streaming read.
template <typename Real>
__global__ void __launch_bounds__(RED_THREADS) argmax_all_kernel(const typename V2<Real>::T *__restrict__ s,
                                                                  long long N, double *pbest, long long *ibest) {
    double best = -1.0;
    long long besti = 0;
#pragma unroll 4
    for (long long i = blockIdx.x * (long long)RED_THREADS + threadIdx.x; i < N; i += (long long)gridDim.x * RED_THREADS) {
        const typename V2<Real>::T v = __ldcs(s + i);
        const double p = (double)v.x * v.x + (double)v.y * v.y;
        if (p > best) {
            best = p;
            besti = i;
        }
    }
    block_best(best, besti);
    if (threadIdx.x == 0) {
        pbest[blockIdx.x] = best;
        ibest[blockIdx.x] = besti;
    }
}

__global__ void __launch_bounds__(RED_THREADS) marginal_final(const double *pbest, const long long *ibest, int nb,
                                                               double *out) {
    double b = -1.0;
    long long bi = 0;
    for (int k = threadIdx.x; k < nb; k += RED_THREADS) keep_best(b, bi, pbest[k], ibest[k]);
    block_best(b, bi);
    if (threadIdx.x == 0) {
        out[0] = b;
        out[1] = (double)bi;
    }
}

// The chunks' sums of every value: `g` values a block's turn, each summed by as
// many threads as the block has for it, then in a tree over those.  g: four
// doubles fill a sector, and few values over many chunks want many blocks (32
// values of 2048 chunks by one block: 20 us more); many values want few turns (2^19
// values of 2 chunks by fours: 160 us more).  ARGMAX: the block's best, in `out` if it is the only block.
static int chunk_group(long long M) { return M < 4 ? (int)M : M <= 4096 ? 4 : 32; }
template <bool ARGMAX>
__global__ void __launch_bounds__(RED_THREADS) marginal_chunks_kernel(const double *__restrict__ partial, long long M,
                                                                       int nch, int g, double *out, double *pbest,
                                                                       long long *ibest) {
    __shared__ double sh[RED_THREADS];
    const int tid = threadIdx.x, rows = RED_THREADS / g;
    double best = -1.0;
    long long besti = 0;
    for (long long x0 = (long long)blockIdx.x * g; x0 < M; x0 += (long long)gridDim.x * g) {
        double p = 0.0;
#pragma unroll 8
        for (int c = tid / g; c < nch; c += rows) p += partial[c * M + x0 + (tid & (g - 1))];
        sh[tid] = p;
        __syncthreads();
        for (int h = RED_THREADS / 2; h >= g; h >>= 1) {
            if (tid < h) sh[tid] += sh[tid + h];
            __syncthreads();
        }
        if (tid < g) {
            if (ARGMAX) keep_best(best, besti, sh[tid], x0 + tid);
            else out[x0 + tid] = sh[tid];
        }
        __syncthreads();
    }
    if (ARGMAX) {
        block_best(best, besti);
        if (tid == 0 && gridDim.x == 1) {
            out[0] = best;
            out[1] = (double)besti;
        } else if (tid == 0) {
            pbest[blockIdx.x] = best;
            ibest[blockIdx.x] = besti;
        }
    }
}
static unsigned chunks_grid(long long M) {
    const long long blocks = M / chunk_group(M);
    return (unsigned)(blocks < RED_BLOCKS ? blocks : RED_BLOCKS);
}

// Chunks a unit is split into: until there are RED_BLOCKS blocks while the
// partial sums (M * nch) are few, then until there are MARG_BLOCKS (MARG_SUMS
// sums at most, a unit's being 2^11 at most) while the sums are a sixteenth of
// the amplitudes or there are fewer than 256 blocks; always as long as a chunk keeps
// four runs and the sums fit `cap`.  FP32, the lowest 8 to 10 bits with 512 and
// 1024 of MARG_BLOCKS: 25 qubits 86 and 72 us, 28 qubits 484 and 341 us (6.3
// TB/s); 13.4 and 106 ms where the sums had to fit 2368.
int marginal_chunks(int n, uint64_t mask, long long cap, long long *units) {
    constexpr long long FEW = 1 << 16;
    const int lb = n < MARG_LOW ? n : MARG_LOW;
    const long long M = 1ll << __builtin_popcountll(mask), U = 1ll << __builtin_popcountll(mask >> lb);
    const long long C = (1ll << (n - lb)) / U;
    int nch = 1;
    while (U * nch < RED_BLOCKS && C / nch >= 8 && 2 * M * nch <= cap &&
           (2 * M * nch <= FEW || (U * nch < MARG_BLOCKS && (U * nch < 256 || 2 * M * nch <= (1ll << n) / 16))))
        nch *= 2;
    *units = U * nch;
    return nch;
}

int64_t marginal_sums(int n, uint64_t mask) {
    long long units = 0;
    const int nch = marginal_chunks(n, mask, MARG_SUMS, &units);
    return nch > 1 ? (int64_t(1) << __builtin_popcountll(mask)) * nch : 0;
}

// Queues the marginal argmax of `mask` over state s: its probability and
// value land in out[0], out[1].  Scratch: pbest and ibest of RED_BLOCKS
// entries, sums of n_sums.
static int queue_marginal(State *s, uint64_t mask, double *pbest, long long *ibest, double *sums, int64_t n_sums,
                          double *out, cudaStream_t st) {
    const int n = s->qubits;
    if (n < 64 && (mask >> n)) return fail(HGM_ERR_INVALID, "mask beyond state bits");
    const long long N = 1ll << n, M = 1ll << __builtin_popcountll(mask);
    unsigned last = 0;  // blocks whose bests are still to be compared
    if (M == N) {
        last = grid_for(N);
        if (s->precision == HGM_F64)
            argmax_all_kernel<double><<<last, RED_THREADS, 0, st>>>((const double2 *)s->d, N, pbest, ibest);
        else
            argmax_all_kernel<float><<<last, RED_THREADS, 0, st>>>((const float2 *)s->d, N, pbest, ibest);
    } else {
        long long units = 0;
        const int nch = marginal_chunks(n, mask, n_sums, &units);
        if (nch > 1) {
            const unsigned g = (unsigned)units;
            if (s->precision == HGM_F64)
                marginal_kernel<double, false><<<g, RED_THREADS, 0, st>>>((const double2 *)s->d, n, mask, nch, M, sums, nullptr, nullptr);
            else
                marginal_kernel<float, false><<<g, RED_THREADS, 0, st>>>((const float2 *)s->d, n, mask, nch, M, sums, nullptr, nullptr);
            const unsigned blocks = chunks_grid(M);
            marginal_chunks_kernel<true><<<blocks, RED_THREADS, 0, st>>>(sums, M, nch, chunk_group(M), out, pbest, ibest);
            count_launch();
            last = blocks > 1 ? blocks : 0;
        } else {
            last = (unsigned)(units < RED_BLOCKS ? units : RED_BLOCKS);
            if (s->precision == HGM_F64)
                marginal_kernel<double, true><<<last, RED_THREADS, 0, st>>>((const double2 *)s->d, n, mask, 1, M, nullptr, pbest, ibest);
            else
                marginal_kernel<float, true><<<last, RED_THREADS, 0, st>>>((const float2 *)s->d, n, mask, 1, M, nullptr, pbest, ibest);
        }
    }
    count_launch();
    if (last) {
        marginal_final<<<1, RED_THREADS, 0, st>>>(pbest, ibest, (int)last, out);
        count_launch();
    }
    return check("argmax launch");
}

int marginal_probs(State *s, uint64_t mask, double *host_out, void *stream) {
    if (ensure_ctx()) return HGM_ERR_CUDA;
    cudaStream_t st = pick(stream);
    if (!st) return HGM_ERR_CUDA;
    const int n = s->qubits;
    if (n < 64 && (mask >> n)) return fail(HGM_ERR_INVALID, "mask beyond state bits");
    const int m = __builtin_popcountll(mask);
    if (m > 26) return fail(HGM_ERR_UNSUPPORTED, "marginal over %d bits (at most 26)", m);
    const long long M = 1ll << m;
    long long units = 0;
    // sums and values within the scratch; a distribution too large for that is
    // over enough high bits
    const int nch = marginal_chunks(n, mask, (long long)(MARGINAL_SCRATCH / sizeof(double)) - M, &units);
    const unsigned g = (unsigned)(units < (1 << 16) ? units : (1 << 16));
    // the chunks' partial sums, then the values: from the context's scratch when
    // they fit (freeing a stream-ordered allocation at every call's
    // synchronisation returns its pages to the driver)
    const long long n_sums = nch > 1 ? M * nch : 0;
    const size_t need = (size_t)(n_sums + M) * sizeof(double);
    std::lock_guard<std::mutex> lk(g_reduce_mu);
    double *sums = g_ctx.marginal;
    cudaError_t e = cudaSuccess;
    if (need > MARGINAL_SCRATCH) {
        e = cudaMallocAsync(&sums, need, st);
        if (e != cudaSuccess) return fail(HGM_ERR_NOMEM, "marginal output: %s", cudaGetErrorString(e));
    }
    double *d_out = sums + n_sums;
    if (s->precision == HGM_F64)
        marginal_kernel<double, false><<<g, RED_THREADS, 0, st>>>((const double2 *)s->d, n, mask, nch, M, sums, nullptr, nullptr);
    else
        marginal_kernel<float, false><<<g, RED_THREADS, 0, st>>>((const float2 *)s->d, n, mask, nch, M, sums, nullptr, nullptr);
    count_launch();
    if (nch > 1) {
        marginal_chunks_kernel<false><<<chunks_grid(M), RED_THREADS, 0, st>>>(sums, M, nch, chunk_group(M), d_out, nullptr, nullptr);
        count_launch();
    }
    int rc = check("marginal probabilities launch");
    if (!rc) {
        e = cudaMemcpyAsync(host_out, d_out, (size_t)M * sizeof(double), cudaMemcpyDeviceToHost, st);
        if (e == cudaSuccess) e = cudaStreamSynchronize(st);
        if (e != cudaSuccess) rc = fail(HGM_ERR_CUDA, "marginal probabilities: %s", cudaGetErrorString(e));
    }
    if (need > MARGINAL_SCRATCH) cudaFreeAsync(sums, st);
    return rc;
}

int launch_argmax_async(State *s, uint64_t mask, double *pbest, long long *ibest, double *sums, int64_t n_sums,
                        double *out, void *stream) {
    return queue_marginal(s, mask, pbest, ibest, sums, n_sums, out, (cudaStream_t)stream);
}

int marginal_argmax(State *s, uint64_t mask, int64_t *arg, double *prob, void *stream) {
    cudaStream_t st = pick(stream);
    if (!st) return HGM_ERR_CUDA;
    std::lock_guard<std::mutex> lk(g_reduce_mu);
    const int rc = queue_marginal(s, mask, g_ctx.partials, g_ctx.partial_idx, g_ctx.marginal, MARG_SUMS, g_ctx.host_result, st);
    if (rc) return rc;
    cudaError_t e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) return fail(HGM_ERR_CUDA, "marginal argmax: %s", cudaGetErrorString(e));
    if (prob) *prob = g_ctx.host_result[0];
    if (arg) *arg = (int64_t)g_ctx.host_result[1];
    return HGM_OK;
}


// ---------------------------------------------------------------------------
// Allocation-free FP64 norm (hgm_norm_noalloc)
// ---------------------------------------------------------------------------
// Some callers cannot allocate device memory: code embedded in a host
// framework that owns every device allocation (a plugin handed pre-allocated
// buffers), or code running while a CUDA graph is being captured elsewhere
// in the process, where a cudaMalloc would be illegal or would synchronise.
// Such a caller should queue it on a stream created non-blocking: the legacy
// default stream (stream NULL) synchronises with blocking streams, and a
// launch there while one of them captures invalidates that capture.
// This variant of the FP64 norm reduction keeps its per-block partial sums in
// a file-scope device array, so it allocates nothing: the caller passes the
// state and a device location for the result.
//
// Limits and sharing:
//   * the array holds NOALLOC_PARTIALS = 2*1184 doubles (18.5 KiB) on every
//     GPU that loads this library, for the life of the process;
//   * the reduction grid is capped at 1184 blocks (one partial each) for any
//     state size, so the array never limits the size; the qubit range
//     1..34 is the engine's own state range (hgm_state_create), and more
//     qubits are rejected with HGM_ERR_UNSUPPORTED;
//   * the result is exactly one double at d_out: the final step writes
//     d_out[0] and nothing after it;
//   * every call shares the array; each call writes every partial it reads
//     before reading it, so nothing needs clearing, but calls that overlap
//     on the GPU (different streams, or different host threads) race on it
//     and must be serialised by the caller;
//   * the array's device address is looked up once per device, on the first
//     call with that device current (cudaGetSymbolAddress); make that first
//     call before any stream capture.
constexpr int NOALLOC_PARTIALS = 2 * RED_BLOCKS;
static __device__ __align__(256) double g_noalloc_partials[NOALLOC_PARTIALS];

namespace {
std::mutex g_noalloc_mu;
double *g_noalloc_ptr[64] = {};
}  // namespace

static int noalloc_scratch(double **out) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return fail(HGM_ERR_CUDA, "cudaGetDevice: %s", cudaGetErrorString(e));
    if (dev < 0 || dev >= 64) return fail(HGM_ERR_UNSUPPORTED, "device %d beyond 64", dev);
    std::lock_guard<std::mutex> lk(g_noalloc_mu);
    if (!g_noalloc_ptr[dev]) {
        void *p = nullptr;
        e = cudaGetSymbolAddress(&p, g_noalloc_partials);
        if (e != cudaSuccess) return fail(HGM_ERR_CUDA, "cudaGetSymbolAddress: %s", cudaGetErrorString(e));
        g_noalloc_ptr[dev] = reinterpret_cast<double *>(p);
    }
    *out = g_noalloc_ptr[dev];
    return HGM_OK;
}

}  // namespace hgm

using namespace hgm;

extern "C" int hgm_norm_noalloc(const void *d_state, int qubits, int precision, double *d_out, void *stream) {
    if (!d_state || !d_out) return fail(HGM_ERR_INVALID, "null state or output pointer");
    if (precision != HGM_F64 && precision != HGM_F32) return fail(HGM_ERR_INVALID, "bad precision");
    if (qubits < 1 || qubits > 34)
        return fail(HGM_ERR_UNSUPPORTED, "qubits=%d outside 1..34, the engine's state range", qubits);
    double *partials = nullptr;
    int rc = noalloc_scratch(&partials);
    if (rc) return rc;
    cudaStream_t st = (cudaStream_t)stream;  // NULL: the legacy default stream
    const long long N = 1ll << qubits;
    const unsigned g = grid_for(N);
    if (precision == HGM_F64)
        reduce_kernel<double, double, RED_NORM><<<g, RED_THREADS, 0, st>>>((const double2 *)d_state, nullptr, N, 0,
                                                                            partials);
    else
        reduce_kernel<float, float, RED_NORM><<<g, RED_THREADS, 0, st>>>((const float2 *)d_state, nullptr, N, 0,
                                                                          partials);
    reduce_final<RED_NORM><<<1, RED_THREADS, 0, st>>>(partials, (int)g, d_out, 1);  // one double, nothing after it
    count_launch(2);
    return check("hgm_norm_noalloc launch");
}

namespace hgm {
}  // namespace hgm

using namespace hgm;

extern "C" {

int64_t hgm_kernel_launches(void) { return g_launches.load(); }

int hgm_timer_start(void) {
    if (ensure_ctx()) return HGM_ERR_CUDA;
    cudaError_t e = cudaEventRecord(g_ctx.t0, g_ctx.stream);
    return e == cudaSuccess ? HGM_OK : fail(HGM_ERR_CUDA, "event record: %s", cudaGetErrorString(e));
}

int hgm_timer_stop(double *ms) {
    if (ensure_ctx()) return HGM_ERR_CUDA;
    cudaEventRecord(g_ctx.t1, g_ctx.stream);
    cudaError_t e = cudaEventSynchronize(g_ctx.t1);
    if (e != cudaSuccess) return fail(HGM_ERR_CUDA, "event sync: %s", cudaGetErrorString(e));
    float f = 0;
    cudaEventElapsedTime(&f, g_ctx.t0, g_ctx.t1);
    if (ms) *ms = f;
    return HGM_OK;
}

}  // extern "C"
