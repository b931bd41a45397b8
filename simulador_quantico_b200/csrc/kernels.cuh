// Device code of the state-vector engine (sm_100a).
//
// Pass kernel ("register tile" design)
// ------------------------------------
// One CTA owns a tile of 2^K amplitudes, K = 5 + R + W: every thread keeps
// NR = 2^R amplitudes in registers (R = 5 for FP32, 4 for FP64), a warp
// holds 2^(5+R) and the CTA 2^W warps.  The tile is the set of state
// indices that agree on every index bit outside the pass's K tile bits;
// local tile bit q is index bit tb[q].  Which local bits are the lane,
// warp and register bits of a thread is the current phase's layout, chosen by
// the planner (struct Lay): any R local bits can be the register bits.
//
// What a tile goes through -- gates, phase blocks, transposes -- comes as one
// stream of 16-byte units (hgm_internal.h, "device stream"), copied into
// shared memory a window ahead (fetch_stream, finish_tile).
//
// A gate whose target is a register bit of the current layout is applied
// entirely in registers.  Switching layout is a transpose through shared
// memory; when both layouts keep the warp bits in place it stays inside
// each warp (__syncwarp), otherwise it crosses warps (__syncthreads).  The
// load and store layouts put thread bits 0..low_bits-1 on the lowest index
// bits of the state, so each warp instruction moves whole 128-byte runs.
// Shared memory is padded (below); the planner only builds layouts
// whose accesses are free of bank conflicts under that padding.
//
// State loads and stores bypass L1 (ld/st .cg): every amplitude is touched
// once per pass, and a tile written by one CTA may be read by another CTA of
// the same persistent kernel in the next pass, which L2 keeps coherent.
//
// The state is read once and written once per pass (the reference's
// "load a tile, apply the whole gate batch, write back once",
// src/core/kernel.cu:68-128), so a pass moves 2*S bytes of HBM traffic.
#pragma once

#include <cuda_runtime.h>

#include "hgm_internal.h"

namespace hgm {

// Register budget per thread.  The FP32 tile (32 float2) and the FP64 tile
// (16 double2) both hold 64 data registers.  128 lets 4 CTAs of 4 warps share
// an SM; the pass kernel is latency-bound (26-qubit layered passes: FP64 -13%, FP32 -2%, QFT
// -12% against a 168-register cap with 3 CTAs per SM; five CTAs of 96 registers
// spill: 26-qubit FP32 layered 13.3 -> 14.2 ms, FP64 searches a third slower).
#ifndef HGM_MAXREG_F32
#define HGM_MAXREG_F32 128
#endif
#ifndef HGM_MAXREG_F64
#define HGM_MAXREG_F64 128
#endif
// Shared-memory carveout for the pass kernels, in percent (-1: driver's
// choice).  The L1 left over holds the loads in flight; forcing the maximum
// shared carveout measured 30% slower streaming passes.
#ifndef HGM_SMEM_CARVEOUT
#define HGM_SMEM_CARVEOUT -1
#endif
// Programmatic dependent launch.  A kernel launched behind another one on its
// stream (launch_behind, kernels.cu) starts while that one's last blocks run,
// fetches what does not depend on it -- the plan's records -- and waits here
// until it is complete and its writes are visible.  Every block that touches a
// state or a plan's scratch waits first.
__device__ __forceinline__ void wait_for_kernel_before() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
// Lets the kernel behind this one start once every block has got here.
__device__ __forceinline__ void let_next_kernel_start() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

template <typename Real, int R>
constexpr int pass_max_regs() {
    return sizeof(Real) == 8 ? HGM_MAXREG_F64 : HGM_MAXREG_F32;
}

template <typename Real>
struct V2;
template <>
struct V2<double> {
    using T = double2;
};
template <>
struct V2<float> {
    using T = float2;
};

// Shared-memory slot of local index j in a transpose: j + (j >> R) (lower.cpp
// slot).  The padding keeps every layout's warp accesses free of bank conflicts
// (a lane stride of 2^R elements becomes 2^R + 1) and, unlike an XOR swizzle,
// it is additive over a layout's disjoint lane/warp and register bits, so the
// slot of register r is the thread's base slot plus r times a constant.

// Shared memory of one tile's transposes, in amplitudes.
template <int R, int W>
__host__ __device__ constexpr int tile_smem_elems() {
    return (1 << (5 + R + W)) + (1 << (5 + W));
}

// Offset (in amplitudes) of a thread's register-0 amplitude and the R
// register-bit strides in the state, for a layout given by the global index
// bit of each role (thread bits 0..4+W, then register bits), read as one
// 16-byte word: byte by byte, the loads alone took several hundred cycles of
// a small state's pass.
template <int R, int W>
__device__ __forceinline__ void thread_geometry(const int8_t (&gb)[MAX_LAYOUT_ROLES], uint32_t thr, uint64_t &off,
                                                uint64_t (&rs)[R]) {
    const uint4 v = *reinterpret_cast<const uint4 *>(gb);
    auto bit = [&](int k) {
        const uint32_t w = k < 4 ? v.x : k < 8 ? v.y : k < 12 ? v.z : v.w;
        return (w >> (8 * (k & 3))) & 63u;
    };
    off = 0;
#pragma unroll
    for (int t = 0; t < 5 + W; t++) off |= (uint64_t)((thr >> t) & 1) << bit(t);
#pragma unroll
    for (int q = 0; q < R; q++) rs[q] = (uint64_t)1 << bit(5 + W + q);
}

template <int R, int r>
__device__ __forceinline__ uint64_t reg_offset(const uint64_t (&rs)[R]) {
    uint64_t o = 0;
#pragma unroll
    for (int q = 0; q < R; q++)
        if (r & (1 << q)) o += rs[q];
    return o;
}

template <int r>
struct Unroll {
    template <typename F>
    __device__ __forceinline__ static void run(F &f) {
        Unroll<r - 1>::run(f);
        f.template go<r - 1>();
    }
};
template <>
struct Unroll<0> {
    template <typename F>
    __device__ __forceinline__ static void run(F &) {}
};

template <typename A2, int R>
struct LoadF {
    A2 (&a)[1 << R];
    const A2 *__restrict__ p;
    const uint64_t (&rs)[R];
    template <int r>
    __device__ __forceinline__ void go() {
        a[r] = __ldcg(p + reg_offset<R, r>(rs));
    }
};
// p is register 0's place and rs the steps with the relabeled bits' signs
// turned (store_tile).
template <typename A2, int R>
struct StoreF {
    const A2 (&a)[1 << R];
    A2 *__restrict__ p;
    const uint64_t (&rs)[R];
    template <int r>
    __device__ __forceinline__ void go() {
        __stcg(p + (int64_t)reg_offset<R, r>(rs), a[r]);
    }
};

// ---- in-place amplitude updates --------------------------------------------
// Every update of a register amplitude goes through these inline-PTX
// primitives.  Their amplitude operands are tied ("+"), so each result is
// written into the register that held the input and the amplitudes keep their
// registers from one gate to the next.  Written as plain expressions, the
// compiler left each result in a fresh register and copied it back wherever
// the op loop's dispatch paths merge; those copies outnumbered the
// floating-point instructions of the pass kernel.  Negated coefficients come
// in as operands (PTX fma has no negated-operand form).
#define HGM_INPLACE_PRIMITIVES(REAL, SFX, C)                                                                      \
    /* (x, y) <- M (x, y), complex M = m[0..7] (row-major re/im), n_k = -m_k */                                 \
    __device__ __forceinline__ void ip_dense(REAL &xr, REAL &xi, REAL &yr, REAL &yi, const REAL(&m)[8], REAL n1, \
                                             REAL n3, REAL n5, REAL n7) {                                        \
        asm("{\n\t.reg ." SFX " t0, t1, t2, t3;\n\t"                                                              \
            "mul.rn." SFX " t0, %4, %0;\n\tmul.rn." SFX " t1, %4, %1;\n\t"                                          \
            "mul.rn." SFX " t2, %8, %0;\n\tmul.rn." SFX " t3, %8, %1;\n\t"                                          \
            "fma.rn." SFX " t0, %12, %1, t0;\n\tfma.rn." SFX " t1, %5, %0, t1;\n\t"                                 \
            "fma.rn." SFX " t2, %14, %1, t2;\n\tfma.rn." SFX " t3, %9, %0, t3;\n\t"                                 \
            "fma.rn." SFX " t0, %6, %2, t0;\n\tfma.rn." SFX " t1, %7, %2, t1;\n\t"                                  \
            "fma.rn." SFX " t2, %10, %2, t2;\n\tfma.rn." SFX " t3, %11, %2, t3;\n\t"                                \
            "fma.rn." SFX " %0, %13, %3, t0;\n\tfma.rn." SFX " %1, %6, %3, t1;\n\t"                                 \
            "fma.rn." SFX " %2, %15, %3, t2;\n\tfma.rn." SFX " %3, %10, %3, t3;\n\t}"                               \
            : "+" C(xr), "+" C(xi), "+" C(yr), "+" C(yi)                                                         \
            : C(m[0]), C(m[1]), C(m[2]), C(m[3]), C(m[4]), C(m[5]), C(m[6]), C(m[7]), C(n1), C(n3), C(n5),      \
              C(n7));                                                                                            \
    }                                                                                                            \
    /* (x, y) <- M (x, y), real M = (m00, m01, m10, m11) */                                                      \
    __device__ __forceinline__ void ip_real(REAL &xr, REAL &xi, REAL &yr, REAL &yi, REAL m00, REAL m01,         \
                                            REAL m10, REAL m11) {                                                \
        asm("{\n\t.reg ." SFX " t0, t1, t2, t3;\n\t"                                                              \
            "mul.rn." SFX " t0, %4, %0;\n\tmul.rn." SFX " t1, %6, %0;\n\t"                                          \
            "mul.rn." SFX " t2, %4, %1;\n\tmul.rn." SFX " t3, %6, %1;\n\t"                                          \
            "fma.rn." SFX " %0, %5, %2, t0;\n\tfma.rn." SFX " %2, %7, %2, t1;\n\t"                                  \
            "fma.rn." SFX " %1, %5, %3, t2;\n\tfma.rn." SFX " %3, %7, %3, t3;\n\t}"                                 \
            : "+" C(xr), "+" C(xi), "+" C(yr), "+" C(yi)                                                         \
            : C(m00), C(m01), C(m10), C(m11));                                                                   \
    }                                                                                                            \
    /* x <- x * (fr + i fi), nfi = -fi */                                                                        \
    __device__ __forceinline__ void ip_cmul(REAL &xr, REAL &xi, REAL fr, REAL fi, REAL nfi) {                  \
        asm("{\n\t.reg ." SFX " t0, t1;\n\t"                                                                      \
            "mul.rn." SFX " t0, %2, %0;\n\tmul.rn." SFX " t1, %3, %0;\n\t"                                          \
            "fma.rn." SFX " %0, %4, %1, t0;\n\tfma.rn." SFX " %1, %2, %1, t1;\n\t}"                                 \
            : "+" C(xr), "+" C(xi)                                                                               \
            : C(fr), C(fi), C(nfi));                                                                             \
    }
HGM_INPLACE_PRIMITIVES(double, "f64", "d")
HGM_INPLACE_PRIMITIVES(float, "f32", "f")
#undef HGM_INPLACE_PRIMITIVES

// amplitude a <- a * f (complex factor f)
template <typename A2>
__device__ __forceinline__ void ip_cmul2(A2 &a, A2 f) {
    ip_cmul(a.x, a.y, f.x, f.y, -f.y);
}

// y already scaled (lower.cpp make_rot): x <- x + u y, then y <- y + t x.  Two
// multiply-adds a component, in place: no temporary to copy back, and half of
// a general real 2x2's four operations.
__device__ __forceinline__ void ip_rot(double &xr, double &xi, double &yr, double &yi, double u, double t) {
    asm("fma.rn.f64 %0, %4, %2, %0;\n\tfma.rn.f64 %1, %4, %3, %1;\n\t"
        "fma.rn.f64 %2, %5, %0, %2;\n\tfma.rn.f64 %3, %5, %1, %3;"
        : "+d"(xr), "+d"(xi), "+d"(yr), "+d"(yi)
        : "d"(u), "d"(t));
}
// sqrt(2) H: x <- x + y, then y <- x - 2 y.
__device__ __forceinline__ void ip_had(double &xr, double &xi, double &yr, double &yi) {
    xr += yr;
    xi += yi;
    yr = fma(-2.0, yr, xr);
    yi = fma(-2.0, yi, xi);
}
// ---- gate application on register bits -----------------------------------

template <typename Real, typename A2>
__device__ __forceinline__ A2 cmul(A2 a, Real mr, Real mi) {
    A2 o;
    o.x = a.x * mr - a.y * mi;
    o.y = a.x * mi + a.y * mr;
    return o;
}

// Each body handles the NR/2 register pairs (or NR registers) of one target
// bit.  Without register-bit controls (CTRL = false, the common case) the
// body is one basic block, so the FMAs of all pairs interleave; with
// controls (CTRL = true) each pair is guarded by its own branch, which keeps
// that rarer variant's register footprint small.
#define HGM_PAIR_GUARD(r) \
    if (CTRL && (((uint32_t)(r) & cm) != cv)) continue;

template <typename Real, typename A2, int R, int T, bool CTRL>
__device__ __forceinline__ void reg_dense(A2 (&a)[1 << R], const Real (&m)[8], uint32_t cm, uint32_t cv) {
    const Real n1 = -m[1], n3 = -m[3], n5 = -m[5], n7 = -m[7];
#pragma unroll
    for (int r = 0; r < (1 << R); r++) {
        if (r & (1 << T)) continue;
        const int r1 = r | (1 << T);
        HGM_PAIR_GUARD(r)
        ip_dense(a[r].x, a[r].y, a[r1].x, a[r1].y, m, n1, n3, n5, n7);
    }
}

// FP32 real 2x2 on packed (re, im) pairs: one f32x2 multiply and one f32x2
// fused multiply-add per output amplitude instead of two of each (the same
// IEEE operations per component, so the results are bit-identical); the
// coefficients come in duplicated, (m, m), built once per gate.
__device__ __forceinline__ void ip_real_x2(float &xr, float &xi, float &yr, float &yi, unsigned long long c00,
                                           unsigned long long c01, unsigned long long c10, unsigned long long c11) {
    asm("{\n\t.reg .b64 X, Y, P, Q;\n\t"
        "mov.b64 X, {%0, %1};\n\tmov.b64 Y, {%2, %3};\n\t"
        "mul.rn.f32x2 P, %4, X;\n\tmul.rn.f32x2 Q, %6, X;\n\t"
        "fma.rn.f32x2 P, %5, Y, P;\n\tfma.rn.f32x2 Q, %7, Y, Q;\n\t"
        "mov.b64 {%0, %1}, P;\n\tmov.b64 {%2, %3}, Q;\n\t}"
        : "+f"(xr), "+f"(xi), "+f"(yr), "+f"(yi)
        : "l"(c00), "l"(c01), "l"(c10), "l"(c11));
}
__device__ __forceinline__ unsigned long long dup_f32(float v) {
    unsigned long long d;
    asm("mov.b64 %0, {%1, %1};" : "=l"(d) : "f"(v));
    return d;
}

template <typename Real, typename A2, int R, int T, bool CTRL>
__device__ __forceinline__ void reg_real(A2 (&a)[1 << R], const Real (&m)[8], uint32_t cm, uint32_t cv) {
    if constexpr (sizeof(Real) == 4) {
        const unsigned long long c00 = dup_f32(m[0]), c01 = dup_f32(m[2]), c10 = dup_f32(m[4]), c11 = dup_f32(m[6]);
#pragma unroll
        for (int r = 0; r < (1 << R); r++) {
            if (r & (1 << T)) continue;
            const int r1 = r | (1 << T);
            HGM_PAIR_GUARD(r)
            ip_real_x2(a[r].x, a[r].y, a[r1].x, a[r1].y, c00, c01, c10, c11);
        }
    } else {
#pragma unroll
        for (int r = 0; r < (1 << R); r++) {
            if (r & (1 << T)) continue;
            const int r1 = r | (1 << T);
            HGM_PAIR_GUARD(r)
            ip_real(a[r].x, a[r].y, a[r1].x, a[r1].y, m[0], m[2], m[4], m[6]);
        }
    }
}

template <typename Real, typename A2, int R, int T, bool CTRL>
__device__ __forceinline__ void reg_diag(A2 (&a)[1 << R], const Real (&m)[8], uint32_t cm, uint32_t cv) {
    const Real n1 = -m[1], n7 = -m[7];
#pragma unroll
    for (int r = 0; r < (1 << R); r++) {
        HGM_PAIR_GUARD(r)
        if (r & (1 << T)) ip_cmul(a[r].x, a[r].y, m[6], m[7], n7);
        else ip_cmul(a[r].x, a[r].y, m[0], m[1], n1);
    }
}

template <typename Real, typename A2, int R, int T, bool CTRL>
__device__ __forceinline__ void reg_phase(A2 (&a)[1 << R], const Real (&m)[8], uint32_t cm, uint32_t cv) {
    const Real n7 = -m[7];
#pragma unroll
    for (int r = 0; r < (1 << R); r++) {
        if (!(r & (1 << T))) continue;
        HGM_PAIR_GUARD(r)
        ip_cmul(a[r].x, a[r].y, m[6], m[7], n7);
    }
}

template <typename Real, typename A2, int R, int T, bool CTRL>
__device__ __forceinline__ void reg_anti(A2 (&a)[1 << R], const Real (&m)[8], uint32_t cm, uint32_t cv) {
#pragma unroll
    for (int r = 0; r < (1 << R); r++) {
        if (r & (1 << T)) continue;
        const int r1 = r | (1 << T);
        HGM_PAIR_GUARD(r)
        const A2 x = a[r], y = a[r1];
        a[r] = cmul<Real>(y, m[2], m[3]);
        a[r1] = cmul<Real>(x, m[4], m[5]);
    }
}

// Controlled swaps select instead of branching: two selects per component
// are cheaper than a branch per pair.
template <typename A2, int R, int T, bool CTRL>
__device__ __forceinline__ void reg_swap(A2 (&a)[1 << R], uint32_t cm, uint32_t cv) {
#pragma unroll
    for (int r = 0; r < (1 << R); r++) {
        if (r & (1 << T)) continue;
        const int r1 = r | (1 << T);
        const A2 x = a[r], y = a[r1];
        if (CTRL) {
            const bool p = ((uint32_t)r & cm) == cv;
            a[r].x = p ? y.x : x.x;
            a[r].y = p ? y.y : x.y;
            a[r1].x = p ? x.x : y.x;
            a[r1].y = p ? x.y : y.y;
        } else {
            a[r] = y;
            a[r1] = x;
        }
    }
}

// Diagonal gate whose target bit is not a register bit: the factor is the
// same for all of a thread's registers that satisfy the register controls.
template <typename Real, typename A2, int R, bool CTRL>
__device__ __forceinline__ void reg_scale(A2 (&a)[1 << R], Real fr, Real fi, uint32_t cm, uint32_t cv) {
    const Real nfi = -fi;
#pragma unroll
    for (int r = 0; r < (1 << R); r++) {
        HGM_PAIR_GUARD(r)
        ip_cmul(a[r].x, a[r].y, fr, fi, nfi);
    }
}

// Kind dispatch as a chain of independent bit tests (not a switch): each
// body updates the registers in place and merges with the path that skips
// it, the shape under which the registers keep their places (a switch here
// became a jump table and cost a hundred register copies per gate).
template <typename Real>
__device__ __forceinline__ void load_matrix(const Real *__restrict__ src, Real (&m)[8]);
template <typename Real>
__device__ __forceinline__ void load_matrix_flip(const Real *__restrict__ src, Real (&m)[8], bool flip);
template <typename Real, typename A2>
__device__ __forceinline__ A2 load_c(const Real *__restrict__ p);

// LEAN: the pass kernel's lean build (plans without controlled dense, real
// or anti-diagonal gates on register bits; Plan::lean) leaves those bodies out.
template <typename Real, typename A2, int R, int T, bool CTRL, bool LEAN>
__device__ __forceinline__ void reg_kind_c(uint32_t kbit, A2 (&a)[1 << R], const Real *__restrict__ mp, uint32_t cm,
                                           uint32_t cv, bool flip) {
    // each body loads its own matrix, so no matrix is live across the chain
    if (!LEAN && (kbit & (1u << K_DENSE))) {
        Real m[8];
        load_matrix_flip<Real>(mp, m, flip);
        reg_dense<Real, A2, R, T, CTRL>(a, m, cm, cv);
    }
    if (!LEAN && (kbit & (1u << K_REAL))) {
        Real m[8];
        load_matrix_flip<Real>(mp, m, flip);
        reg_real<Real, A2, R, T, CTRL>(a, m, cm, cv);
    }
    if (kbit & (1u << K_DIAG)) {
        Real m[8];
        load_matrix_flip<Real>(mp, m, flip);
        reg_diag<Real, A2, R, T, CTRL>(a, m, cm, cv);
    }
    if (kbit & (1u << K_PHASE)) {
        Real m[8];
        load_matrix<Real>(mp, m);
        reg_phase<Real, A2, R, T, CTRL>(a, m, cm, cv);
    }
    if (!LEAN && (kbit & (1u << K_ANTI))) {
        Real m[8];
        load_matrix_flip<Real>(mp, m, flip);
        reg_anti<Real, A2, R, T, CTRL>(a, m, cm, cv);
    }
    if (kbit & (1u << K_SWAP)) reg_swap<A2, R, T, CTRL>(a, cm, cv);
}

// Target dispatch, the same way: one bit test per register bit.
template <typename Real, typename A2, int R, int T, bool LEAN>
struct RegTarget {
    __device__ __forceinline__ static void run(uint32_t tbit, uint32_t kbit, A2 (&a)[1 << R],
                                               const Real *__restrict__ mp, uint32_t cm, uint32_t cv, bool flip) {
        // one instantiation, with the per-pair control test: gates without
        // register controls (cm = 0, every pair passes) are rare here, since
        // uncontrolled dense gates go out as layers and uncontrolled X gates
        // relabel, and a second copy of every body cost instruction-cache
        // misses
        if constexpr (LEAN) {
            if (tbit & (1u << T)) reg_kind_c<Real, A2, R, T, true, LEAN>(kbit, a, mp, cm, cv, flip);
            RegTarget<Real, A2, R, T + 1, LEAN>::run(tbit, kbit, a, mp, cm, cv, flip);
        } else {
            among<0, R>(tbit, kbit, a, mp, cm, cv, flip);
        }
    }
    // One of the targets LO..HI-1, by halves: in the full build, whose bodies are
    // long, jumping over each target's bodies in turn waits for instructions, and
    // so does passing every other op's body first (finish_tile tests its S_GATE
    // first).  24 qubits FP32, 90 gates of one control: dense 1190 -> 1067 us, real
    // 682 -> 631, anti 894 -> 801; 26 qubits, 120 gates of every kind 3.70 -> 3.33 ms.
    template <int LO, int HI>
    __device__ __forceinline__ static void among(uint32_t tbit, uint32_t kbit, A2 (&a)[1 << R],
                                                 const Real *__restrict__ mp, uint32_t cm, uint32_t cv, bool flip) {
        if constexpr (HI - LO == 1) {
            reg_kind_c<Real, A2, R, LO, true, LEAN>(kbit, a, mp, cm, cv, flip);
        } else {
            constexpr int MID = (LO + HI) / 2;
            if (tbit < (1u << MID)) among<LO, MID>(tbit, kbit, a, mp, cm, cv, flip);
            else among<MID, HI>(tbit, kbit, a, mp, cm, cv, flip);
        }
    }
};
template <typename Real, typename A2, int R, bool LEAN>
struct RegTarget<Real, A2, R, R, LEAN> {
    __device__ __forceinline__ static void run(uint32_t, uint32_t, A2 (&)[1 << R], const Real *__restrict__,
                                               uint32_t, uint32_t, bool) {}
};

// Gate data sits in the stream window in shared memory: 16-byte loads of the
// same address by every lane.
template <>
__device__ __forceinline__ void load_matrix<double>(const double *__restrict__ src, double (&m)[8]) {
    const double2 *p = reinterpret_cast<const double2 *>(src);
#pragma unroll
    for (int k = 0; k < 4; k++) {
        const double2 v = p[k];
        m[2 * k] = v.x;
        m[2 * k + 1] = v.y;
    }
}
template <>
__device__ __forceinline__ void load_matrix<float>(const float *__restrict__ src, float (&m)[8]) {
    const float4 *p = reinterpret_cast<const float4 *>(src);
#pragma unroll
    for (int k = 0; k < 2; k++) {
        const float4 v = p[k];
        m[4 * k] = v.x;
        m[4 * k + 1] = v.y;
        m[4 * k + 2] = v.z;
        m[4 * k + 3] = v.w;
    }
}

// Loads a gate matrix; with `flip` set, the matrix with both bit values of
// its target exchanged (X M X: m00 <-> m11, m01 <-> m10), for registers whose
// labels have that bit swapped (register relabeling, below).
template <typename Real>
__device__ __forceinline__ void load_matrix_flip(const Real *__restrict__ src, Real (&m)[8], bool flip) {
    // entry k of the swapped matrix is entry 3 - k = k ^ 3 of the stored one
    const int fx = flip ? 3 : 0;
#pragma unroll
    for (int k = 0; k < 4; k++) {
        const typename V2<Real>::T v = load_c<Real, typename V2<Real>::T>(src + 2 * (k ^ fx));
        m[2 * k] = v.x;
        m[2 * k + 1] = v.y;
    }
}

// A layer: uncontrolled gates on a set of register bits (mask), lowest bit
// first, one straight-line block per active bit (a uniform branch skips
// inactive bits); the gates' data follow the header in the stream.

// Complex 2x2s (S_DENSE) and real ones (S_REAL).
template <typename Real, typename A2, int R, int T>
struct DenseStep {
    __device__ __forceinline__ static void run(A2 (&a)[1 << R], const Real *__restrict__ d, uint32_t mask, uint32_t xr) {
        if (mask & (1u << T)) {
            Real m[8];
            load_matrix_flip<Real>(d, m, (xr >> T) & 1u);
            reg_dense<Real, A2, R, T, false>(a, m, 0u, 0u);
            d += 8;
        }
        DenseStep<Real, A2, R, T + 1>::run(a, d, mask, xr);
    }
};
template <typename Real, typename A2, int R>
struct DenseStep<Real, A2, R, R> {
    __device__ __forceinline__ static void run(A2 (&)[1 << R], const Real *__restrict__, uint32_t, uint32_t) {}
};

// four values from the stream
__device__ __forceinline__ void load4(const float *__restrict__ p, float (&v)[4]) {
    const float4 x = *reinterpret_cast<const float4 *>(p);
    v[0] = x.x; v[1] = x.y; v[2] = x.z; v[3] = x.w;
}
__device__ __forceinline__ void load4(const double *__restrict__ p, double (&v)[4]) {
    const double2 x = reinterpret_cast<const double2 *>(p)[0], y = reinterpret_cast<const double2 *>(p)[1];
    v[0] = x.x; v[1] = x.y; v[2] = y.x; v[3] = y.y;
}

// HAD: the matrix [[1, 1], [1, -1]], no data (a Hadamard layer in a warp with
// relabeled registers, which the in-place form below does not take).
template <typename Real, typename A2, int R, int T>
struct RealStep {
    __device__ __forceinline__ static void run(A2 (&a)[1 << R], const Real *__restrict__ d, uint32_t mask, uint32_t xr,
                                               bool had) {
        if (mask & (1u << T)) {
            Real v[4] = {1, 1, 1, -1}, m[8];
            if (!had) load4(d, v);
            const bool f = (xr >> T) & 1u;
            m[0] = f ? v[3] : v[0];
            m[2] = f ? v[2] : v[1];
            m[4] = f ? v[1] : v[2];
            m[6] = f ? v[0] : v[3];
            reg_real<Real, A2, R, T, false>(a, m, 0u, 0u);
            d += 4;
        }
        RealStep<Real, A2, R, T + 1>::run(a, d, mask, xr, had);
    }
};
template <typename Real, typename A2, int R>
struct RealStep<Real, A2, R, R> {
    __device__ __forceinline__ static void run(A2 (&)[1 << R], const Real *__restrict__, uint32_t, uint32_t, bool) {}
};

template <typename Real, typename A2, int R, int T>
struct HadStep {
    __device__ __forceinline__ static void run(A2 (&a)[1 << R], uint32_t mask) {
        if (mask & (1u << T)) {
#pragma unroll
            for (int r = 0; r < (1 << R); r++)
                if (!(r & (1 << T))) ip_had(a[r].x, a[r].y, a[r | (1 << T)].x, a[r | (1 << T)].y);
        }
        HadStep<Real, A2, R, T + 1>::run(a, mask);
    }
};
template <typename Real, typename A2, int R>
struct HadStep<Real, A2, R, R> {
    __device__ __forceinline__ static void run(A2 (&)[1 << R], uint32_t) {}
};

template <typename Real, typename A2>
__device__ __forceinline__ A2 cmul2(A2 a, A2 b);

// Multiplies the registers whose bit T is 1 by f (a phase diag(1, f)).
template <typename Real, typename A2, int R, int T>
__device__ __forceinline__ void reg_half_phase(A2 (&a)[1 << R], A2 f) {
    const Real nfi = -f.y;
#pragma unroll
    for (int r = 0; r < (1 << R); r++)
        if (r & (1 << T)) ip_cmul(a[r].x, a[r].y, f.x, f.y, nfi);
}

// Gates Rm diag(1, p), Rm real: on each active register bit T the phase on the
// registers whose bit T is 1, then the real part.
//   FP32 (S_SPLIT): the real 2x2, 2 packed operations an amplitude; 4 with the
//     phase, against the complex matrix's 8.
//   FP64 (S_ROT, lower.cpp make_rot): a rotation in place, its factor left
//     out; 4 + 4 operations a pair against 16 of a complex 2x2 and 12 of the
//     phase and a real 2x2 (S_SPLIT in FP64: gates without that form).
// Seen through a swapped label (xr bit T set) the gate is
//   X Rm diag(1, p) X = p (X Rm X) diag(1, p*),
// so the phase stays on the same registers, conjugated, the real matrix is
// read bit-swapped (a rotation by the opposite angle) and p joins the thread's
// factor `pend`, which the layer multiplies into all registers at its end.
// One gate's data as loaded: m00, m01, m10, m11, p; S_ROT t, u, p.
template <typename Real, bool ROT>
struct SplitRec;
template <>
struct SplitRec<float, false> {
    float4 m;
    float2 p;
    __device__ __forceinline__ void load(const float *__restrict__ d) {
        m = *reinterpret_cast<const float4 *>(d);
        p = *reinterpret_cast<const float2 *>(d + 4);
    }
    static constexpr int words = 8;
};
template <>
struct SplitRec<double, false> {
    double4 m;
    double2 p;
    __device__ __forceinline__ void load(const double *__restrict__ d) {
        const double2 a = reinterpret_cast<const double2 *>(d)[0], b = reinterpret_cast<const double2 *>(d)[1];
        m = make_double4(a.x, a.y, b.x, b.y);
        p = reinterpret_cast<const double2 *>(d)[2];
    }
    static constexpr int words = 8;
};
template <>
struct SplitRec<double, true> {
    double2 tu, p;
    __device__ __forceinline__ void load(const double *__restrict__ d) {
        tu = reinterpret_cast<const double2 *>(d)[0];
        p = reinterpret_cast<const double2 *>(d)[1];
    }
    static constexpr int words = 4;
};

template <typename Real, typename A2, int R, int T, bool ROT>
struct SplitStep {
    __device__ __forceinline__ static void run(A2 (&a)[1 << R], const Real *__restrict__ d, uint32_t mask, uint32_t xr,
                                               A2 &pend, SplitRec<Real, ROT> &cur) {
        if (mask & (1u << T)) {
            const bool flip = (xr >> T) & 1u;
            SplitRec<Real, ROT> c = cur;
            if constexpr (sizeof(Real) == 8) c.load(d);
            d += SplitRec<Real, ROT>::words;
            // FP32: the next gate's data, while this one's arithmetic runs
            // (after the last gate: the units behind the op, not used), 1.2%
            // of a layered pass; in FP64 the eight registers cost 1%
            if constexpr (sizeof(Real) == 4) cur.load(d);
            A2 p = c.p;
            if constexpr (!ROT) {
                if constexpr (sizeof(Real) == 4) {
                    // one rounding order whatever the compiler makes of the
                    // surrounding code
                    const Real px = __fmaf_rn(pend.x, p.x, -__fmul_rn(pend.y, p.y));
                    const Real py = __fmaf_rn(pend.x, p.y, __fmul_rn(pend.y, p.x));
                    pend.x = flip ? px : pend.x;
                    pend.y = flip ? py : pend.y;
                } else if (flip) {
                    pend = cmul2<Real>(pend, p);
                }
                p.y = flip ? -p.y : p.y;
                Real m[8];
                m[0] = flip ? c.m.w : c.m.x;
                m[2] = flip ? c.m.z : c.m.y;
                m[4] = flip ? c.m.y : c.m.z;
                m[6] = flip ? c.m.x : c.m.w;
                reg_half_phase<Real, A2, R, T>(a, p);
                reg_real<Real, A2, R, T, false>(a, m, 0u, 0u);
            } else {
                double t = c.tu.x, u = c.tu.y;
                if (flip) {  // a branch: FP64 products and selects for every gate took 3%
                    // p itself: the stored phase carries 1 + t^2 = 1 / (1 + u t)
                    const double k = t * u + 1.0;
                    A2 q;
                    q.x = p.x * k;
                    q.y = p.y * k;
                    pend = cmul2<Real>(pend, q);
                    t = -t;
                    u = -u;
                    p.y = -p.y;
                }
                reg_half_phase<Real, A2, R, T>(a, p);
#pragma unroll
                for (int r = 0; r < (1 << R); r++)
                    if (!(r & (1 << T))) ip_rot(a[r].x, a[r].y, a[r | (1 << T)].x, a[r | (1 << T)].y, u, t);
            }
        }
        SplitStep<Real, A2, R, T + 1, ROT>::run(a, d, mask, xr, pend, cur);
    }
};
template <typename Real, typename A2, int R, bool ROT>
struct SplitStep<Real, A2, R, R, ROT> {
    __device__ __forceinline__ static void run(A2 (&)[1 << R], const Real *__restrict__, uint32_t, uint32_t, A2 &,
                                               SplitRec<Real, ROT> &) {}
};

template <typename Real, typename A2, int R, bool ROT>
__device__ __forceinline__ void apply_split_layer(A2 (&a)[1 << R], const Real *__restrict__ d, uint32_t mask,
                                                  uint32_t xr) {
    A2 pend;
    pend.x = 1;
    pend.y = 0;
    SplitRec<Real, ROT> cur;
    if constexpr (sizeof(Real) == 4) cur.load(d);
    SplitStep<Real, A2, R, 0, ROT>::run(a, d, mask, xr, pend, cur);
    // every thread of the warp reaches this point (ops are uniform)
    if (__any_sync(0xffffffffu, (xr & mask) != 0u)) {
#pragma unroll
        for (int r = 0; r < (1 << R); r++) ip_cmul2(a[r], pend);
    }
}

// Phase block: diagonal gates with at most one control, combined per thread
// into a scalar f, per-register-bit factors g[b] (bit 1) and h[b] (bit 0) and
// an optional host-built 2^R table (gates whose target and control are both
// register bits); each register is then multiplied once per involved bit.
// A term applies when its controls on non-tile and thread bits hold; a term
// whose target is not a register bit contributes d1 or d0 according to this
// thread's value of that bit.
template <typename Real, typename A2>
__device__ __forceinline__ A2 load_c(const Real *__restrict__ p);
template <>
__device__ __forceinline__ double2 load_c<double, double2>(const double *__restrict__ p) {
    return *reinterpret_cast<const double2 *>(p);
}
template <>
__device__ __forceinline__ float2 load_c<float, float2>(const float *__restrict__ p) {
    return *reinterpret_cast<const float2 *>(p);
}

// A product term of a phase block (S_TERMS): thread controls and target,
// non-tile controls, the diagonal's two entries.
template <typename Real>
constexpr int product_term_bytes() {
    return 32 + 4 * (int)sizeof(Real);
}
template <typename Real, typename A2>
struct ProductTerm {
    A2 f0, f1;
    bool ok;
    int tp;
    __device__ __forceinline__ ProductTerm(const unsigned char *__restrict__ t, uint64_t base, uint32_t thr) {
        const uint4 th = *reinterpret_cast<const uint4 *>(t);
        const ulonglong2 gl = reinterpret_cast<const ulonglong2 *>(t)[1];
        const Real *m = reinterpret_cast<const Real *>(t + 32);
        f0 = load_c<Real, A2>(m);
        f1 = load_c<Real, A2>(m + 2);
        ok = ((base & gl.x) == gl.y) && ((thr & th.x) == th.y);
        tp = (int)th.z;
    }
};

// Factor of one term for this thread: d0 or d1 of its diagonal gate by the
// value of its target (a thread or non-tile bit), or 1 when its controls on
// thread and non-tile bits do not hold.  Branch-free: the conditions differ
// between threads of a warp.
template <typename Real, typename A2>
__device__ __forceinline__ A2 term_factor(const unsigned char *__restrict__ t, uint64_t base, uint32_t thr) {
    const ProductTerm<Real, A2> q(t, base, thr);
    const uint32_t bv = q.tp >= TPOS_GLOBAL   ? (uint32_t)(base >> (q.tp - TPOS_GLOBAL)) & 1u
                        : q.tp >= TPOS_THREAD ? (thr >> (q.tp - TPOS_THREAD)) & 1u
                                              : 0u;
    A2 f = bv ? q.f1 : q.f0;
    f.x = q.ok ? f.x : (Real)1;
    f.y = q.ok ? f.y : (Real)0;
    return f;
}

template <typename Real, typename A2>
__device__ __forceinline__ A2 cmul2(A2 a, A2 b) {
    A2 o;
    o.x = a.x * b.x - a.y * b.y;
    o.y = a.x * b.y + a.y * b.x;
    return o;
}

// acc times the factors of terms t[0..n), two terms per step (two chains, so
// that one term's loads overlap the other's arithmetic).
template <typename Real, typename A2>
__device__ __forceinline__ A2 term_product(const unsigned char *__restrict__ t, int n, uint64_t base, uint32_t thr,
                                           A2 acc) {
    constexpr int B = product_term_bytes<Real>();
    A2 acc2;
    acc2.x = 1;
    acc2.y = 0;
    int i = 0;
#pragma unroll 1
    for (; i + 1 < n; i += 2) {
        const A2 fa = term_factor<Real, A2>(t + i * B, base, thr), fb = term_factor<Real, A2>(t + (i + 1) * B, base, thr);
        acc = cmul2<Real>(acc, fa);
        acc2 = cmul2<Real>(acc2, fb);
    }
    if (i < n) acc = cmul2<Real>(acc, term_factor<Real, A2>(t + i * B, base, thr));
    return cmul2<Real>(acc, acc2);
}

// D terms (a diagonal gate on register bit b, controls elsewhere): h takes
// d0, g takes d1, where the controls hold.
template <typename Real, typename A2>
__device__ __forceinline__ void term_diag_product(const unsigned char *__restrict__ t, int n, uint64_t base,
                                                  uint32_t thr, A2 &h, A2 &g) {
#pragma unroll 1
    for (int i = 0; i < n; i++) {
        ProductTerm<Real, A2> q(t + i * product_term_bytes<Real>(), base, thr);
        q.f0.x = q.ok ? q.f0.x : (Real)1;
        q.f0.y = q.ok ? q.f0.y : (Real)0;
        q.f1.x = q.ok ? q.f1.x : (Real)1;
        q.f1.y = q.ok ? q.f1.y : (Real)0;
        h = cmul2<Real>(h, q.f0);
        g = cmul2<Real>(g, q.f1);
    }
}

// A phase block's 2^R table: complex factors by register label, register r
// holding label r ^ xr.  When no lane of the warp has a relabeled register
// (xr == 0, as in the QFT's phase passes), the labels are the register numbers
// and every entry sits at a constant offset: two entries per 16-byte load in
// FP32 and no address arithmetic.
template <typename Real, typename A2, int R>
__device__ __forceinline__ void apply_table(A2 (&a)[1 << R], const Real *__restrict__ z, uint32_t xr) {
    if (__all_sync(0xffffffffu, xr == 0u)) {
        if constexpr (sizeof(Real) == 4) {
#pragma unroll
            for (int r = 0; r < (1 << R); r += 2) {
                const float4 f = *reinterpret_cast<const float4 *>(z + 2 * r);
                ip_cmul2(a[r], make_float2(f.x, f.y));
                ip_cmul2(a[r + 1], make_float2(f.z, f.w));
            }
        } else {
#pragma unroll
            for (int r = 0; r < (1 << R); r++) ip_cmul2(a[r], load_c<Real, A2>(z + 2 * r));
        }
        return;
    }
#pragma unroll
    for (int r = 0; r < (1 << R); r++) ip_cmul2(a[r], load_c<Real, A2>(z + 2 * (r ^ xr)));
}

// Byte K of the 16 phase-block term counts, kept packed in four words.
template <int K>
__device__ __forceinline__ int count_byte(const uint4 &c) {
    const uint32_t w = K < 4 ? c.x : K < 8 ? c.y : K < 12 ? c.z : c.w;
    return (int)((w >> (8 * (K & 3))) & 0xffu);
}

// Register bit B of a phase block: when the block marks B active, folds the
// G[B], H[B] and D[B] terms into g (factor of the registers whose bit B is 1)
// and h (bit B is 0), starting from `carry` (the block's F factor, handed to
// the first active bit and reset), and multiplies them into the registers
// with one sweep.  Inactive bits cost nothing but the pointer step.
template <typename Real, typename A2, int R, int B>
struct PhaseBits {
    __device__ __forceinline__ static void run(A2 (&a)[1 << R], const unsigned char *__restrict__ t,
                                               const uint4 &cnt, uint32_t act, A2 &carry, uint64_t base,
                                               uint32_t thr, uint32_t xr) {
        constexpr int TB = product_term_bytes<Real>();
        const int ng = count_byte<1 + B>(cnt), nh = count_byte<1 + R + B>(cnt), nd = count_byte<1 + 2 * R + B>(cnt);
        if (act & (1u << B)) {
            A2 g = term_product<Real, A2>(t, ng, base, thr, carry);
            A2 h = term_product<Real, A2>(t + ng * TB, nh, base, thr, carry);
            carry.x = 1;
            carry.y = 0;
            term_diag_product<Real, A2>(t + (ng + nh) * TB, nd, base, thr, h, g);
            // g belongs to the registers whose label has bit B set
            const bool flip = (xr >> B) & 1u;
            const A2 g1 = flip ? h : g, h1 = flip ? g : h;
#pragma unroll
            for (int r = 0; r < (1 << R); r++) ip_cmul2(a[r], ((r >> B) & 1) ? g1 : h1);
        }
        PhaseBits<Real, A2, R, B + 1>::run(a, t + (ng + nh + nd) * TB, cnt, act, carry, base, thr, xr);
    }
};
template <typename Real, typename A2, int R>
struct PhaseBits<Real, A2, R, R> {
    __device__ __forceinline__ static void run(A2 (&)[1 << R], const unsigned char *__restrict__, const uint4 &,
                                               uint32_t, A2 &, uint64_t, uint32_t, uint32_t) {}
};

// ---- phase blocks of compact phase terms (head flag PB_ANGLES) ------------
// Each term adds a0 or a1 turns to its category's phase where its control
// holds; the index bits it tests are those of the thread's register-0
// amplitude, ix = tile base | the thread bits placed at their index bits
// (head bytes 16..23).  A category's factor is exp(2 pi i * turns), one
// sincospi per category instead of a complex multiply per term.
// The words of one compact term.  A linear term (cbit == PB_LINEAR) keeps its
// index mask where a0 (and, in FP32, a1) sit and its scale in pad2 (FP32) or
// a1 (FP64).
template <typename Real>
struct TermWords;
template <>
struct TermWords<float> {
    uint32_t head;
    float a0, a1, scale;
    uint64_t mask;
    __device__ __forceinline__ TermWords(const unsigned char *p) {
        const uint4 v = *reinterpret_cast<const uint4 *>(p);
        head = v.x;
        a0 = __uint_as_float(v.y);
        a1 = __uint_as_float(v.z);
        mask = ((uint64_t)v.z << 32) | v.y;
        scale = __uint_as_float(v.w);
    }
};
template <>
struct TermWords<double> {
    uint32_t head;
    double a0, a1, scale;
    uint64_t mask;
    __device__ __forceinline__ TermWords(const unsigned char *p) {
        const uint4 v = *reinterpret_cast<const uint4 *>(p);
        const double2 w = reinterpret_cast<const double2 *>(p)[1];
        head = v.x;
        a0 = __hiloint2double((int)v.w, (int)v.z);
        a1 = w.x;
        mask = ((uint64_t)v.w << 32) | v.z;
        scale = w.x;
    }
};

// Turns of a linear term at index ix: scale times the masked index as an
// integer, or bit-reversed (brev64 * 2^-63: index bit b weighs 2^-b).
template <typename Real>
__device__ __forceinline__ Real linear_turns(const TermWords<Real> &t, uint64_t ix, bool rev) {
    const unsigned long long x = ix & t.mask;
    const Real v = rev ? (Real)__brevll(x) * (Real)1.0842021724855044e-19 : (Real)x;
    return t.scale * v;
}

// Term k of the block whose terms start at rec0, for a category that adds
// a0 / a1 turns by the value of the term's target: the turns it adds at ix
// (0 where its control does not hold).
template <typename Real>
__device__ __forceinline__ Real term_turns(const unsigned char *__restrict__ rec0, int k, uint64_t ix) {
    const TermWords<Real> t(rec0 + k * sizeof(PhaseTerm<Real>));
    const int cbit = (int)(int8_t)(t.head & 0xffu), cval = (int)((t.head >> 8) & 0xffu);
    const int tbit = (int)(int8_t)((t.head >> 16) & 0xffu);
    const uint32_t tv = tbit < 0 ? 0u : (uint32_t)((ix >> (tbit & 63)) & 1u);
    if (cbit == PB_LINEAR) return (tbit < 0 || tv) ? linear_turns<Real>(t, ix, cval & 1) : (Real)0;
    const bool c = cbit < 0 || (int)((ix >> (cbit & 63)) & 1u) == cval;
    return c ? (tv ? t.a1 : t.a0) : (Real)0;
}

// Term k of a D category (a diagonal on the category's register bit): adds
// its d0 turns to h and its d1 turns to g where its control holds.
template <typename Real>
__device__ __forceinline__ void dterm_turns(const unsigned char *__restrict__ rec0, int k, uint64_t ix, Real &h,
                                            Real &g) {
    const TermWords<Real> t(rec0 + k * sizeof(PhaseTerm<Real>));
    const int cbit = (int)(int8_t)(t.head & 0xffu), cval = (int)((t.head >> 8) & 0xffu);
    if (cbit == PB_LINEAR) {
        const int tbit = (int)(int8_t)((t.head >> 16) & 0xffu);
        if (tbit < 0 || ((ix >> (tbit & 63)) & 1u)) g += linear_turns<Real>(t, ix, cval & 1);
        return;
    }
    const bool c = cbit < 0 || (int)((ix >> (cbit & 63)) & 1u) == cval;
    h += c ? t.a0 : (Real)0;
    g += c ? t.a1 : (Real)0;
}

template <typename Real>
__device__ __forceinline__ Real turns_sum(const unsigned char *__restrict__ rec0, int k0, int n, uint64_t ix, Real acc) {
    Real acc2 = 0;
    int k = 0;
#pragma unroll 1
    for (; k + 1 < n; k += 2) {
        acc += term_turns<Real>(rec0, k0 + k, ix);
        acc2 += term_turns<Real>(rec0, k0 + k + 1, ix);
    }
    if (k < n) acc += term_turns<Real>(rec0, k0 + k, ix);
    return acc + acc2;
}

template <typename A2, typename Real>
__device__ __forceinline__ A2 cis_turns(Real t) {
    const Real r = t - rint(t);
    A2 f;
    if constexpr (sizeof(Real) == 4) sincospif(2.0f * r, &f.y, &f.x);
    else sincospi(2.0 * r, &f.y, &f.x);
    return f;
}

template <typename Real, typename A2, int R, int B>
struct PhaseBitsAngles {
    __device__ __forceinline__ static void run(A2 (&a)[1 << R], const unsigned char *__restrict__ rec0, int k,
                                               const uint4 &cnt, uint32_t act, Real &carry, uint64_t ix, uint32_t xr) {
        const int ng = count_byte<1 + B>(cnt), nh = count_byte<1 + R + B>(cnt), nd = count_byte<1 + 2 * R + B>(cnt);
        if (act & (1u << B)) {
            Real g = turns_sum<Real>(rec0, k, ng, ix, carry);
            Real h = turns_sum<Real>(rec0, k + ng, nh, ix, carry);
            carry = 0;
#pragma unroll 1
            for (int i = 0; i < nd; i++) dterm_turns<Real>(rec0, k + ng + nh + i, ix, h, g);
            // g belongs to the registers whose label has bit B set
            const bool flip = (xr >> B) & 1u;
            const A2 gf = cis_turns<A2>(g), hf = cis_turns<A2>(h);
            const A2 g1 = flip ? hf : gf, h1 = flip ? gf : hf;
#pragma unroll
            for (int r = 0; r < (1 << R); r++) ip_cmul2(a[r], ((r >> B) & 1) ? g1 : h1);
        }
        PhaseBitsAngles<Real, A2, R, B + 1>::run(a, rec0, k + ng + nh + nd, cnt, act, carry, ix, xr);
    }
};
template <typename Real, typename A2, int R>
struct PhaseBitsAngles<Real, A2, R, R> {
    __device__ __forceinline__ static void run(A2 (&)[1 << R], const unsigned char *__restrict__, int, const uint4 &,
                                               uint32_t, Real &, uint64_t, uint32_t) {}
};

// Byte k (runtime) of the 16 phase-block term counts.
__device__ __forceinline__ int count_byte_at(const uint4 &c, int k) {
    const uint32_t w = k < 4 ? c.x : k < 8 ? c.y : k < 12 ? c.z : c.w;
    return (int)((w >> (8 * (k & 3))) & 0xffu);
}

// A gated block's sweep (PB_GATED, no relabeled register in the warp): the
// registers whose bit B is 1 times their table entry, if there is a table, and
// c.  (A fifth of a QFT's blocks have none: 27 qubits FP32 3.04 -> 2.98 ms, 26
// qubits FP64 2.81 -> 2.71 against multiplying by a table of ones.)
template <typename Real, typename A2, int R, int B>
struct GatedSweep {
    __device__ __forceinline__ static void run(int b, A2 (&a)[1 << R], A2 c, const Real *__restrict__ z, bool table) {
        if (b == B) {
            if (table) {
#pragma unroll
                for (int r = 0; r < (1 << R); r++)
                    if (r & (1 << B)) ip_cmul2(a[r], load_c<Real, A2>(z + 2 * r));
            }
#pragma unroll
            for (int r = 0; r < (1 << R); r++)
                if (r & (1 << B)) ip_cmul2(a[r], c);
            return;
        }
        GatedSweep<Real, A2, R, B + 1>::run(b, a, c, z, table);
    }
};
template <typename Real, typename A2, int R>
struct GatedSweep<Real, A2, R, R> {
    __device__ __forceinline__ static void run(int, A2 (&)[1 << R], A2, const Real *__restrict__, bool) {}
};

// S_PHASES: `op` is the op's head in the stream window, hdr its first unit.
// tix: the thread bits at their index bits.  KEEP: computed by the first block
// after a layout change (PB_FRESH) and kept for the others (60 of 500
// instructions a block; 27-qubit FP32 QFT 2.98 -> 2.89 ms, 26-qubit FP64 2.71 ->
// 2.61).  The chained kernels compute it for each block: kept, its registers
// cost their layered circuits 1%.
template <typename Real, typename A2, int R, int W, bool KEEP>
__device__ __forceinline__ void apply_phase_block_angles(A2 (&a)[1 << R], const unsigned char *__restrict__ op,
                                                         const uint4 hdr, uint64_t base, uint32_t thr, uint32_t xr,
                                                         uint64_t &tix) {
    const uint32_t flags = hdr.y, act = hdr.z;
    const Real *__restrict__ table = reinterpret_cast<const Real *>(op + 16 * hdr.w);
    const uint4 cnt = reinterpret_cast<const uint4 *>(op)[1];
    if (!KEEP || (flags & PB_FRESH)) {
        const uint2 tg = reinterpret_cast<const uint2 *>(op)[4];
        tix = 0;
#pragma unroll
        for (int t = 0; t < 5 + W; t++) {
            const uint32_t g = ((t < 4 ? tg.x : tg.y) >> (8 * (t & 3))) & 63u;
            tix |= (uint64_t)((thr >> t) & 1u) << g;
        }
    }
    const uint64_t ix = base | tix;
    const unsigned char *rec0 = op + 48;
    if ((flags & PB_GATED) && __all_sync(0xffffffffu, xr == 0u)) {
        // only G[b] terms, then D[b] terms (the walk order with every other
        // category empty); one factor for the registers whose bit b is 1
        const int b = (int)((flags >> PB_GATE_SHIFT) & 7u);
        const int ng = count_byte_at(cnt, 1 + b), nd = count_byte_at(cnt, 1 + 2 * R + b);
        Real g = turns_sum<Real>(rec0, 0, ng, ix, (Real)0), h = 0;
#pragma unroll 1
        for (int i = 0; i < nd; i++) dterm_turns<Real>(rec0, ng + i, ix, h, g);
        GatedSweep<Real, A2, R, 0>::run(b, a, cis_turns<A2>(g), table, (flags & PB_HAS_TABLE) != 0u);
        return;
    }
    const int nf = count_byte<0>(cnt);
    Real carry = turns_sum<Real>(rec0, 0, nf, ix, (Real)0);
    PhaseBitsAngles<Real, A2, R, 0>::run(a, rec0, nf, cnt, act, carry, ix, xr);
    if ((act & PB_F_ACTIVE) && !(act & ((1u << R) - 1u))) {
        const A2 f = cis_turns<A2>(carry);
#pragma unroll
        for (int r = 0; r < (1 << R); r++) ip_cmul2(a[r], f);
    }
    if (flags & PB_HAS_TABLE) apply_table<Real, A2, R>(a, table, xr);
}

// S_TERMS: the F terms fold into one per-thread factor; each active register
// bit costs one sweep of the registers (PhaseBits); the F factor rides on the
// first active bit's sweep, or gets a sweep of its own when no bit is active;
// the thread-independent 2^R table, if any, is one more sweep.
template <typename Real, typename A2, int R>
__device__ __forceinline__ void apply_phase_block(A2 (&a)[1 << R], const unsigned char *__restrict__ op, const uint4 hdr,
                                                  uint64_t base, uint32_t thr, uint32_t xr) {
    const uint32_t act = hdr.z;   // active register bits, PB_F_ACTIVE: F terms
    const uint4 cnt = reinterpret_cast<const uint4 *>(op)[1];  // 16 count bytes
    const unsigned char *__restrict__ t = op + 48;
    A2 carry;
    carry.x = 1;
    carry.y = 0;
    const int nf = count_byte<0>(cnt);
    carry = term_product<Real, A2>(t, nf, base, thr, carry);
    PhaseBits<Real, A2, R, 0>::run(a, t + nf * product_term_bytes<Real>(), cnt, act, carry, base, thr, xr);
    if ((act & PB_F_ACTIVE) && !(act & ((1u << R) - 1u))) {
#pragma unroll
        for (int r = 0; r < (1 << R); r++) ip_cmul2(a[r], carry);
    }
    if (hdr.y & PB_HAS_TABLE) apply_table<Real, A2, R>(a, reinterpret_cast<const Real *>(op + 16 * hdr.w), xr);
}

// One relabeling X gate (a K_XSET entry): flips the thread's label bit where
// its control holds.
__device__ __forceinline__ uint32_t xset_flip(uint32_t w, uint64_t base, uint32_t thr) {
    const uint32_t t = w & 0xffu, ck = (w >> 8) & 0xffu, cb = (w >> 16) & 0xffu, cv = w >> 24;
    const uint32_t v = ck == XSET_CTRL_THREAD   ? (thr >> cb) & 1u
                       : ck == XSET_CTRL_GLOBAL ? (uint32_t)(base >> cb) & 1u
                                                : cv;
    return (uint32_t)(v == cv) << t;
}

// X on register bit T where label bit C is 1 or 0 (S_CSWAP, one control: the
// CNOTs of a layered circuit): per thread one predicate, q on the registers
// whose bit C is 0 and !q on the others, so a pair costs its four selects.
template <typename A2, int R, int T, int C>
struct CSwap {
    __device__ __forceinline__ static void run(uint32_t c, A2 (&a)[1 << R], bool q) {
        if constexpr (C < R) {
            if constexpr (C != T) {
                if (c == C) {
#pragma unroll
                    for (int r = 0; r < (1 << R); r++) {
                        if (r & (1 << T)) continue;
                        const int r1 = r | (1 << T);
                        const bool p = (r & (1 << C)) ? !q : q;
                        const A2 x = a[r], y = a[r1];
                        a[r].x = p ? y.x : x.x;
                        a[r].y = p ? y.y : x.y;
                        a[r1].x = p ? x.x : y.x;
                        a[r1].y = p ? x.y : y.y;
                    }
                }
            }
            CSwap<A2, R, T, C + 1>::run(c, a, q);
        }
    }
};
template <typename A2, int R, int T>
__device__ __forceinline__ void controlled_swap(uint32_t t, uint32_t c, A2 (&a)[1 << R], bool q) {
    if constexpr (T < R) {
        if (t == T) CSwap<A2, R, T, 0>::run(c, a, q);
        else controlled_swap<A2, R, T + 1>(t, c, a, q);
    }
}

// Any other record (S_GATE).
template <typename Real, typename A2, int R, bool LEAN>
__device__ __forceinline__ void apply_gate(A2 (&a)[1 << R], const unsigned char *__restrict__ op, const uint4 hdr,
                                           uint64_t base, uint32_t thr, uint32_t &xr) {
    const int kind = (int)(hdr.y & 0xffu), tpos = (int)(hdr.y >> 8);
    const uint2 th = reinterpret_cast<const uint2 *>(op)[2];             // cm_thr, cv_thr
    const ulonglong2 gl = reinterpret_cast<const ulonglong2 *>(op)[2];   // cm_glob, cv_glob
    if ((base & gl.x) != gl.y) return;
    if ((thr & th.x) != th.y) return;
    const Real *m = reinterpret_cast<const Real *>(op + 48);
    const uint32_t cm = hdr.z, cv = hdr.w ^ (xr & hdr.z);
    if (tpos < R) {
        if (kind == K_SWAP && cm == 0) {
            xr ^= 1u << tpos;
            return;
        }
        // a phase gate seen through a swapped label is diag(d1, 1): run it as
        // a diagonal gate on the bit-swapped matrix
        const bool flip = (xr >> tpos) & 1u;
        const int k = (kind == K_PHASE && flip) ? K_DIAG : kind;
        RegTarget<Real, A2, R, 0, LEAN>::run(1u << tpos, 1u << k, a, m, cm, cv, flip);
        return;
    }
    // diagonal gate on a thread bit or a non-tile index bit
    const int bv = tpos >= TPOS_GLOBAL ? (int)((base >> (tpos - TPOS_GLOBAL)) & 1)
                                       : (int)((thr >> (tpos - TPOS_THREAD)) & 1);
    if (kind == K_PHASE && !bv) return;
    const A2 f = load_c<Real, A2>(m + (bv ? 6 : 0));
    reg_scale<Real, A2, R, true>(a, f.x, f.y, cm, cv);
}

// ---- the stream in shared memory ---------------------------------------------

constexpr int STREAM_WINDOW_BYTES = STREAM_WINDOW_UNITS * 16;
// Bytes of a pass's window (at most STREAM_WINDOW_BYTES).
template <int W>
__host__ __device__ __forceinline__ constexpr int window_bytes(const TileArgs &ta) {
    if constexpr (W == 0) return (int)ta.ld_tstep[7];
    else return STREAM_WINDOW_BYTES;
}

// Shared memory of a CTA: the transpose buffer, then two stream windows, then
// room for the loads ahead of the last op (a header, a gate's data; not used).
template <typename Real, int R, int W>
__host__ __device__ constexpr int tile_smem_bytes() {
    return tile_smem_elems<R, W>() * (int)sizeof(typename V2<Real>::T);
}
template <typename Real, int R, int W>
__host__ __device__ constexpr int cta_smem_bytes() {
    return tile_smem_bytes<Real, R, W>() + 2 * STREAM_WINDOW_BYTES + 32;
}

// Starts the CTA's copy of `units` units into shared memory (cached in L1: the
// SM's other CTAs run the same pass).
__device__ __forceinline__ void fetch_units(unsigned char *dst, const uint4 *__restrict__ src, int units) {
    const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
    for (int i = threadIdx.x; i < units; i += blockDim.x)
        asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"(d + 16u * i), "l"(src + i) : "memory");
}
__device__ __forceinline__ void fetch_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// Starts copying a pass's first two windows; every earlier reader of the
// windows must be done.
template <int W>
__device__ __forceinline__ void fetch_stream(unsigned char *win, const TileArgs &ta) {
    const uint4 *src = reinterpret_cast<const uint4 *>(ta.stream);
    fetch_units(win, src, ta.units0);
    if (ta.units1) fetch_units(win + window_bytes<W>(ta), src + ta.units0, ta.units1);
}

// ---- layout transposes through shared memory --------------------------------

// Moves the registers from the current layout (thread base `tb`, byte steps in
// the op) to the next.  Register r holds label r ^ xr (register relabeling,
// below): its slot is the thread's base plus the steps of the bits of r ^ xr,
// i.e. the base moved by the steps of xr plus the steps of r with those bits
// negated.
template <typename A2, int R, int W>
__device__ __forceinline__ void transpose(A2 (&a)[1 << R], unsigned char *sm, const unsigned char *__restrict__ op,
                                          const uint4 hdr, uint32_t thr, uint32_t &tb, uint32_t xr) {
    {
        const uint4 f = reinterpret_cast<const uint4 *>(op)[1];
        const uint32_t all[5] = {f.x, f.y, f.z, f.w, hdr.z};
        uint32_t wb = tb, s[R];
        if (hdr.y & STREAM_SYNC_BEFORE) __syncthreads();
        else __syncwarp();
#pragma unroll
        for (int q = 0; q < R; q++) {
            const bool fl = (xr >> q) & 1u;
            wb += fl ? all[q] : 0u;
            s[q] = fl ? 0u - all[q] : all[q];
        }
#pragma unroll
        for (int r = 0; r < (1 << R); r++) {
            uint32_t o = wb;
#pragma unroll
            for (int q = 0; q < R; q++)
                if (r & (1 << q)) o += s[q];
            *reinterpret_cast<A2 *>(sm + o) = a[r];
        }
    }
    const uint4 t = reinterpret_cast<const uint4 *>(op)[2], b0 = reinterpret_cast<const uint4 *>(op)[3],
                b1 = reinterpret_cast<const uint4 *>(op)[4];
    const uint32_t u[5] = {t.x, t.y, t.z, t.w, hdr.w};
    const uint32_t bs[8] = {b0.x, b0.y, b0.z, b0.w, b1.x, b1.y, b1.z, b1.w};
    tb = 0;
#pragma unroll
    for (int b = 0; b < 5 + W; b++) tb += ((thr >> b) & 1u) * bs[b];
    if (hdr.y & STREAM_SYNC_CROSS) __syncthreads();
    else __syncwarp();
#pragma unroll
    for (int r = 0; r < (1 << R); r++) {
        uint32_t o = tb;
#pragma unroll
        for (int q = 0; q < R; q++)
            if (r & (1 << q)) o += u[q];
        a[r] = *reinterpret_cast<const A2 *>(sm + o);
    }
}

// Index of tile `t`: deposit the bits of t into the non-tile index bits, one
// run of consecutive non-tile bits at a time (uniform across the CTA).
__device__ __forceinline__ uint64_t tile_base(uint64_t t, const TileArgs &ta) {
    const ulonglong2 pos = *reinterpret_cast<const ulonglong2 *>(ta.run_pos),
                     len = *reinterpret_cast<const ulonglong2 *>(ta.run_len);
    uint64_t base = 0, p = pos.x, l = len.x;
    for (int i = 0; i < ta.nruns; i++) {
        if (i == 8) {
            p = pos.y;
            l = len.y;
        }
        const int n = (int)(l & 63u);
        base |= (t & ((1ull << n) - 1ull)) << (p & 63u);
        t >>= n;
        p >>= 8;
        l >>= 8;
    }
    return base;
}

template <typename Real, int R, int W>
__device__ __forceinline__ void load_tile(typename V2<Real>::T (&a)[1 << R],
                                          const typename V2<Real>::T *__restrict__ state, const TileArgs &ta,
                                          uint64_t base, uint32_t thr) {
    using A2 = typename V2<Real>::T;
    uint64_t off, rs[R];
    thread_geometry<R, W>(ta.ld_gbit, thr, off, rs);
    LoadF<A2, R> f{a, state + (base | off), rs};
    Unroll<1 << R>::run(f);
}

template <typename Real, int R, int W>
__device__ __forceinline__ void store_tile(const typename V2<Real>::T (&a)[1 << R],
                                           typename V2<Real>::T *__restrict__ state, const TileArgs &ta,
                                           uint64_t base, uint32_t xr) {
    using A2 = typename V2<Real>::T;
    // The thread index is re-read so the store geometry is recomputed here
    // instead of being held in registers through every phase.
    uint32_t thr;
    asm volatile("mov.u32 %0, %%tid.x;" : "=r"(thr));
    uint64_t off, rs[R];
    thread_geometry<R, W>(ta.st_gbit, thr, off, rs);
    // register r goes to the place of label r ^ xr: start at the relabeled
    // bits' steps and take those steps back where r has the bit
    uint64_t idx = base | off;
#pragma unroll
    for (int q = 0; q < R; q++)
        if ((xr >> q) & 1u) {
            idx += rs[q];
            rs[q] = 0ull - rs[q];
        }
    StoreF<A2, R> f{a, state + idx, rs};
    Unroll<1 << R>::run(f);
}

// Applies a pass's stream to a tile already in registers (loaded in the
// pass's load layout) and stores it.  The first windows' copy (fetch_stream)
// has been started.
//
// Register relabeling: a thread keeps `xr`, and register r holds the
// amplitude whose register label is r ^ xr.  An X on a register bit whose
// controls (if any) lie on thread or non-tile bits -- most CNOTs of a pass --
// only flips a bit of xr.  Gates on a register bit whose xr bit is set use
// the bit-swapped matrix, register-bit control values are read through xr,
// and the next transpose or the store puts every amplitude where its label
// says (xr is then 0 again).
//
// LEAN (Plan::lean): the build for plans whose phase blocks are all compact
// terms, with no controlled dense, real or anti-diagonal gate on a register
// bit, no complex layer and, in FP64, no S_SPLIT.  Leaving those bodies out of the kernel
// -- code the benchmark circuits never run -- made 26-qubit FP32 layered
// passes 5% and QFT passes 9% faster (fewer instruction-fetch stalls), so
// each plan runs the smallest build it can.
//
// ctl: renormalisation (the plain pass kernel passes ta's own; the chained
// kernel sets it per position in the pass sequence, in shared memory, where it
// costs the tile no registers).  The scale is read through L2: in a chained
// run it was accumulated by other CTAs of the same launch.
// KEEP_IX: apply_phase_block_angles.
template <typename Real, int R, int W, bool LEAN, bool KEEP_IX>
__device__ __forceinline__ void finish_tile(typename V2<Real>::T (&a)[1 << R], typename V2<Real>::T *__restrict__ state,
                                            const TileArgs &ta, uint64_t base, unsigned char *sm,
                                            const PassCtl &ctl) {
    using A2 = typename V2<Real>::T;
    constexpr bool F64 = sizeof(Real) == 8;
    const uint32_t thr = threadIdx.x, lane = thr & 31;
    unsigned char *win = sm + tile_smem_bytes<Real, R, W>();
    if (ctl.flags & PASS_SCALE) {
        const Real s = (Real)rsqrt(__ldcg(ctl.scale_in));
#pragma unroll
        for (int r = 0; r < (1 << R); r++) {
            a[r].x *= s;
            a[r].y *= s;
        }
    }
    uint32_t tb = 0;
#pragma unroll
    for (int b = 0; b < 5 + W; b++) tb += ((thr >> b) & 1u) * ta.ld_tstep[b];
    uint32_t xr = 0;            // register relabeling
    uint64_t tix = 0;           // thread bits at their index bits (phase blocks)
    uint32_t pc = 0;            // byte offset in the two windows
    uint32_t next = ta.units0 + ta.units1;  // first unit not fetched yet
    fetch_wait();
    __syncthreads();
    // each op's header is loaded while the op before it runs (3.5% of an FP64
    // layered pass, 1.2% FP32)
    uint4 nh = *reinterpret_cast<const uint4 *>(win);
    for (;;) {
        const unsigned char *op = win + pc;
        uint4 hdr = nh;
        // every lane has the same header; after the reduction the compiler
        // knows it and branches without convergence barriers (a 26-qubit
        // layered pass: 200 instructions a warp fewer, 1.5% faster)
        hdr.x = __reduce_or_sync(0xffffffffu, hdr.x);
        hdr.y = __reduce_or_sync(0xffffffffu, hdr.y);
        const uint32_t kind = hdr.x & 0xffu;
        const Real *data = reinterpret_cast<const Real *>(op + 16);
        pc += (hdr.x >> 8) << 4;
        nh = *reinterpret_cast<const uint4 *>(win + pc);
        if (!LEAN && kind == S_GATE) {
            apply_gate<Real, A2, R, LEAN>(a, op, hdr, base, thr, xr);
        } else if (kind == (F64 ? S_ROT : S_SPLIT)) {
            const uint32_t mask = hdr.y & 0xffu;
            apply_split_layer<Real, A2, R, F64>(a, data, mask, xr);
            if (F64) xr ^= hdr.y >> 8;
        } else if (kind == S_REAL || (F64 && kind == S_HAD)) {
            const bool had = F64 && kind == S_HAD;
            if (had && !__any_sync(0xffffffffu, (xr & hdr.y) != 0u)) {
                if constexpr (F64) HadStep<Real, A2, R, 0>::run(a, hdr.y);
            } else {
                RealStep<Real, A2, R, 0>::run(a, data, hdr.y, xr, had);
            }
        } else if (kind == S_TRANS) {
            transpose<A2, R, W>(a, sm, op, hdr, thr, tb, xr);
            xr = 0;
        } else if (kind == S_XSET) {
            const int n = (int)hdr.y;
            xr ^= xset_flip(hdr.z, base, thr);
            if (n > 1) xr ^= xset_flip(hdr.w, base, thr);
#pragma unroll 1
            for (int j = 2; j < n; j++) xr ^= xset_flip(reinterpret_cast<const uint32_t *>(op)[2 + j], base, thr);
        } else if (kind == S_CSWAP) {
            const uint32_t c = hdr.y >> 16;
            controlled_swap<A2, R, 0>(hdr.y & 0xffffu, c, a, ((xr >> c) & 1u) == hdr.z);
        } else if (kind == S_PHASES) {
            apply_phase_block_angles<Real, A2, R, W, KEEP_IX>(a, op, hdr, base, thr, xr, tix);
        } else if (F64 && kind == S_SCALE) {
            const Real f = (Real)__hiloint2double((int)hdr.w, (int)hdr.z);
#pragma unroll
            for (int r = 0; r < (1 << R); r++) {
                a[r].x *= f;
                a[r].y *= f;
            }
        } else if (LEAN && kind == S_GATE) {
            apply_gate<Real, A2, R, LEAN>(a, op, hdr, base, thr, xr);
        } else if (kind == S_NEXT) {
            // the next window has been fetched; this one makes room for the
            // window after it
            fetch_wait();
            __syncthreads();
            const int wb = window_bytes<W>(ta);
            const bool first = pc <= (uint32_t)wb;
            if (hdr.y)
                fetch_units(win + (first ? 0 : wb), reinterpret_cast<const uint4 *>(ta.stream) + next,
                            (int)hdr.y);
            next += hdr.y;
            pc = first ? wb : 0;
            nh = *reinterpret_cast<const uint4 *>(win + pc);
        } else if (F64 && !LEAN && kind == S_SPLIT) {
            apply_split_layer<Real, A2, R, false>(a, data, hdr.y, xr);
        } else if (!LEAN && kind == S_DENSE) {
            DenseStep<Real, A2, R, 0>::run(a, data, hdr.y, xr);
        } else if (!LEAN && kind == S_TERMS) {
            apply_phase_block<Real, A2, R>(a, op, hdr, base, thr, xr);
        } else {
            break;  // S_END
        }
    }
    store_tile<Real, R, W>(a, state, ta, base, xr);
    if (ctl.flags & PASS_NORM) {
        double acc = 0.0;
#pragma unroll
        for (int r = 0; r < (1 << R); r++) acc += (double)a[r].x * a[r].x + (double)a[r].y * a[r].y;
#pragma unroll
        for (int o = 16; o; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
        if (lane == 0) atomicAdd(ctl.norm_out, acc);
    }
}

// ---- permutation pass -----------------------------------------------------------

// Sub-tile u of a permutation pass (hgm_internal.h PASS_PERMUTE), NT threads:
// u, permuted inside, to the place of its partner v and v to that of u; u's
// holder does both, v's nothing.  Loads and stores are runs of 128 bytes and
// more; the bits change places in shared memory (slot s + s / 16: lanes that
// write 2^4 slots apart miss each other's banks), both sub-tiles at once, so
// that few amplitudes are held in registers: inlined in the chained kernels
// beside the tile code, sixteen of them cost 190-430 bytes of spills.
constexpr int PERM_SLOTS = (1 << PERM_BITS) + (1 << (PERM_BITS - 4));  // a sub-tile's slots
template <typename Real, int NT>
__device__ __forceinline__ void permute_subtile(typename V2<Real>::T *__restrict__ state, const TileArgs &ta, uint64_t u,
                                                typename V2<Real>::T *sm, const PassCtl &ctl) {
    using A2 = typename V2<Real>::T;
    constexpr int PER = (1 << PERM_BITS) / NT;
    const uint32_t tid = threadIdx.x;
    const uint64_t base = tile_base(u, ta);
    uint64_t other = base;
    const unsigned char *pair = reinterpret_cast<const unsigned char *>(ta.ld_tstep);
    for (int k = 0; k < ta.pairs; k++) {
        const int a = pair[2 * k], b = pair[2 * k + 1];
        const uint64_t x = ((other >> a) ^ (other >> b)) & 1ull;
        other ^= (x << a) | (x << b);
    }
    if (other < base) return;
    // place in the state and slot after the permutation of local index j
    auto place = [&](uint32_t j) {
        uint64_t o = 0;
#pragma unroll
        for (int q = 0; q < PERM_BITS; q++) o |= (uint64_t)((j >> q) & 1u) << ta.ld_gbit[q];
        return o;
    };
    auto slot = [&](uint32_t j) {
        uint32_t v = 0;
#pragma unroll
        for (int q = 0; q < PERM_BITS; q++) v |= ((j >> q) & 1u) << ta.st_gbit[q];
        return v + (v >> 4);
    };
    const uint64_t at = place(tid);
    const uint32_t to = slot(tid);
    const Real scale = (ctl.flags & PASS_SCALE) ? (Real)rsqrt(__ldcg(ctl.scale_in)) : (Real)1;
    double acc = 0.0;
    const int sides = other != base ? 2 : 1;
#pragma unroll 1
    for (int side = 0; side < sides; side++) {
        const A2 *__restrict__ src = state + ((side ? other : base) | at);
        A2 v[PER];
#pragma unroll
        for (int i = 0; i < PER; i++) v[i] = __ldcg(src + place(i * NT));
        if (ctl.flags & (PASS_SCALE | PASS_NORM)) {
#pragma unroll
            for (int i = 0; i < PER; i++) {
                v[i].x *= scale;
                v[i].y *= scale;
                acc += (double)v[i].x * v[i].x + (double)v[i].y * v[i].y;
            }
        }
#pragma unroll
        for (int i = 0; i < PER; i++) sm[side * PERM_SLOTS + to + slot(i * NT)] = v[i];
    }
    __syncthreads();
#pragma unroll 1
    for (int side = 0; side < sides; side++) {
        A2 *__restrict__ dst = state + ((side ? base : other) | at);
#pragma unroll
        for (int i = 0; i < PER; i++) {
            const uint32_t j = i * NT + tid;
            __stcg(dst + place(i * NT), sm[side * PERM_SLOTS + j + (j >> 4)]);
        }
    }
    __syncthreads();
    if (ctl.flags & PASS_NORM) {
#pragma unroll
        for (int o = 16; o; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
        if ((tid & 31) == 0) atomicAdd(ctl.norm_out, acc);
    }
}

// Runs one pass over tile `tile`.  Shared by the plain pass kernel and the
// chained and batched persistent kernels; the first windows' copy has been
// started.  PERM: the pass may be a permutation pass (the pass kernel's are
// launches of their own).
template <typename Real, int R, int W, bool LEAN, bool PERM>
__device__ __forceinline__ void run_tile(typename V2<Real>::T *__restrict__ state, const TileArgs &ta, uint64_t tile,
                                         unsigned char *sm, const PassCtl &ctl) {
    using A2 = typename V2<Real>::T;
    if constexpr (W >= PERM_WARP_BITS && PERM) {
        if (ta.flags & PASS_PERMUTE) {
            constexpr int SUB = 5 + R + W - PERM_BITS;  // sub-tiles a tile, as a power of two
            static_assert(2 * PERM_SLOTS <= tile_smem_elems<R, W>(), "two sub-tiles fit the transpose buffer");
            for (uint64_t k = 0; k < (1ull << SUB); k++)
                permute_subtile<Real, 32 << W>(state, ta, (tile << SUB) | k, reinterpret_cast<A2 *>(sm), ctl);
            return;
        }
    }
    const uint64_t base = tile_base(tile, ta);
    A2 a[1 << R];
    load_tile<Real, R, W>(a, state, ta, base, threadIdx.x);
    finish_tile<Real, R, W, LEAN, !PERM>(a, state, ta, base, sm, ctl);
}

}  // namespace hgm
