// Lowering: a plan's passes -> the device stream the kernels run.
//
// The planner's records (hgm_internal.h DevOp) say what a pass does; this
// file writes it in the form that costs the pass kernel least:
//   * one linear stream per pass, ops and transposes in the order they run,
//     16 to 32 bytes a gate instead of 80 to 112, so that a window of it fits
//     beside the transpose buffer in shared memory;
//   * FP64 rotations, Hadamards and other invertible gates without their common
//     factor (cos or 1/sqrt 2), which leaves half the operations of the real 2x2
//     out; the factors multiply into one S_SCALE at the plan's end (or when they
//     leave [2^-200, 2^200]; amplitudes above 2^823 would overflow meanwhile).
//     28 qubits, 10 layers, FP64: 67.0 -> 50.1 ms with the stream; 26-qubit
//     search, 32 iterations: 78.7 -> 60.2 ms.  FP32 keeps the plain form: its
//     results are, bit by bit, those of the records, but for phase blocks larger
//     than a window, which run as several;
//   * the swaps that end a circuit (a QFT's qubit reversal), where they fill
//     passes of their own, as one permutation pass: it reads and writes the
//     state once at memory speed, whatever the pairs, where CNOTs need the
//     bits of a pair in one tile (27-qubit FP32 QFT:
//     4.65 -> 3.31 ms, three passes of CNOTs and some of three others gone).
#include <cmath>
#include <cstring>
#include <initializer_list>

#include "hgm_internal.h"

namespace hgm {

namespace {

struct Rot {
    long double kappa;  // factor left out: a plan multiplies hundreds of them
    double t, u, pr, pi;
    bool x;         // an X follows
};

// Writes a real orthogonal matrix (up to a factor) with a phase before it,
//   M = Rm diag(1, p),   Rm = h [[c, -d s], [s, d c]],  d = +-1,
// as kappa X^x R(t) diag(1, e p) with |t| <= 1, e = +-1 and
// R(t) = [[1, -t], [t, 1]]: t = s / c, or (with an X behind) c / s.  The
// kernel runs R(t) diag(1, e p) in place with two multiply-adds a component,
//   y' = ((1 + t^2) e p) y,   x1 = x + u y',   y1 = y' + t x1,
//   u = -t / (1 + t^2),
// the factor 1 + t^2 riding on the phase.  m: Rm row-major.  False when Rm is
// not of that form (a gate that is not unitary up to a factor).
bool make_rot(const double *m, double p_re, double p_im, Rot &r) {
    double big = 0.0;
    for (int k = 0; k < 4; k++) big = std::max(big, std::abs(m[k]));
    const double d = m[0] * m[3] - m[1] * m[2] >= 0.0 ? 1.0 : -1.0;
    const double tol = 4e-15 * big;
    if (!(std::abs(m[3] - d * m[0]) <= tol && std::abs(m[2] + d * m[1]) <= tol)) return false;
    const double c = 0.5 * (m[0] + d * m[3]), s = 0.5 * (m[2] - d * m[1]);
    if (!std::isfinite(c) || !std::isfinite(s) || (c == 0.0 && s == 0.0)) return false;
    r.x = std::abs(s) > std::abs(c);
    const double num = r.x ? c : s, den = r.x ? s : c, e = r.x ? -d : d;
    r.t = num / den;
    const long double sq = 1.0L + (long double)r.t * r.t;
    // from the rounded t, so that kappa sqrt(1 + t^2) is Rm's own factor
    r.kappa = std::copysign(std::hypot((long double)c, (long double)s) / std::sqrt(sq), (long double)den);
    r.u = (double)(-r.t / sq);
    r.pr = (double)(e * p_re * sq);
    r.pi = (double)(e * p_im * sq);
    return true;
}

// Any other invertible real matrix in the same form: rows exchanged if the
// first column's larger entry a is below, then with t = c / a, s = det / a^2
// and u = (b / a) / s,
//   M = a X^x [[1, s u], [t, s (1 + t u)]] diag(1, p),
// run as above with s in the phase's place of e (1 + t^2).  |t| <= 1 bounds the
// growth as row pivoting does.  Not a form that survives a relabeled bit: only
// for bits that no thread has relabeled.  False for (nearly) singular matrices
// and for those whose second column is far larger than the first: s and s u, by
// which amplitudes grow before a is applied, stay below 2^20.
bool make_lift(const double *m, double p_re, double p_im, Rot &r) {
    r.x = std::abs(m[2]) > std::abs(m[0]);
    const long double a = m[r.x ? 2 : 0], b = m[r.x ? 3 : 1], c = m[r.x ? 0 : 2], d = m[r.x ? 1 : 3];
    const long double s = (a * d - b * c) / (a * a);
    r.kappa = a;
    r.t = (double)(c / a);
    r.u = (double)(b / a / s);
    r.pr = (double)(s * p_re);
    r.pi = (double)(s * p_im);
    return std::isfinite(r.t) && std::isfinite(r.u) && std::isfinite(r.pr) && std::isfinite(r.pi) &&
           std::abs(r.u) <= 0x1p20 && std::abs(s) <= 0x1p20 && std::abs(b / a) <= 0x1p20;
}

// The factor a of a [[1, 1], [1, -1]], or 0.  An a within the roundings of H, or
// of a few H fused, of 1/sqrt 2 stands for that: a search multiplies thousands
// of them, and the double's error alone, 5e-17 each, made most of the 1.4e-13 of
// 26 qubits x 32 iterations (now 4e-16).
long double hadamard_factor(const double *m) {
    const double a = 0.25 * (m[0] + m[1] + m[2] - m[3]), tol = 4e-16 * std::abs(a);
    const bool ok = std::isfinite(a) && std::abs(m[0] - a) <= tol && std::abs(m[1] - a) <= tol &&
                    std::abs(m[2] - a) <= tol && std::abs(m[3] + a) <= tol;
    const long double h = std::copysign(std::sqrt(0.5L), (long double)a);
    return !ok ? 0.0L : std::abs(a - h) <= 0x1p-51L ? h : a;
}

// The words of an op other than a phase block, without an allocation for each
// (planning a 17-qubit search 2.48 -> 2.23 ms FP32, 2.97 -> 2.58 FP64).  The largest, five gates of
// 16 words behind a header.
struct Words {
    uint32_t w[96];
    size_t n = 0;
    Words() {}
    Words(std::initializer_list<uint32_t> v) {
        for (uint32_t x : v) w[n++] = x;
    }
    void push_back(uint32_t x) { w[n++] = x; }
    uint32_t &operator[](size_t i) { return w[i]; }
    const uint32_t &operator[](size_t i) const { return w[i]; }
    size_t size() const { return n; }
    const uint32_t *begin() const { return w; }
    const uint32_t *end() const { return w + n; }
};
static_assert(4 + PB_MAX_R * 16 <= 96, "an op of the largest layer");

template <typename Real>
struct Lowering {
    Plan *plan;
    const cplx global;
    const int R, W;
    long double scale = 1.0;  // factors left out and not yet applied
    // the current pass: its windows' units
    std::vector<uint32_t> out;
    std::vector<uint32_t> window;
    std::vector<size_t> windows;   // units of each finished window
    const size_t CAP;              // one unit less than a window: S_NEXT or S_END

    int split_gates = 0, phase_gates = 0;  // gates of split layers; of them, phase gates with a real one behind
    uint32_t relabeled = 0;  // register bits that some thread may have relabeled in this layout
    bool fresh = true;       // no phase block of compact terms in this layout yet
    bool drop_swaps = false; // the marked records are left to a permutation pass

    Lowering(Plan *p, cplx gl)
        : plan(p), global(gl), R(p->reg_bits), W(p->warp_bits),
          CAP((W == 0 && p->qubits > 5 + R ? SHORT_WINDOW_UNITS : STREAM_WINDOW_UNITS) - 1) {}

    bool same_warps(int a, int b) const {
        for (int w = 0; w < W; w++)
            if (plan->layouts[a].pos[5 + w] != plan->layouts[b].pos[5 + w]) return false;
        return true;
    }
    // whether the layout may store the state (planner LayoutMaker::coalesced)
    bool coalesced(int l) const {
        for (int i = 0; i < plan->low_bits && i < 5; i++)
            if (plan->layouts[l].pos[i] != i) return false;
        return true;
    }
    static int records(const DevOp<Real> &d) {
        if (d.kind == K_PHASE_BLOCK) return 1 + d.tpos;
        if (d.kind == K_LAYER || d.kind == K_LAYER_REAL || d.kind == K_LAYER_SPLIT) return 1 + __builtin_popcount(d.cm_reg);
        return 1;
    }
    // whether every op of the record belongs to the final swaps
    static bool swap_record(const DevOp<Real> &d) {
        return d.kind == K_XSET ? d.pad1 == (1u << d.tpos) - 1u : d.kind == K_SWAP && d.pad1;
    }
    bool only_swaps(const DevPhase &ph, const DevOp<Real> *ops) const {
        for (int i = ph.op_begin; i < ph.op_end; i += records(ops[i]))
            if (!swap_record(ops[i])) return false;
        return true;
    }
    bool only_swaps(const PassArgs &pa, const DevOp<Real> *ops) const {
        for (int p = pa.phase_begin; p < pa.phase_end; p++)
            if (!only_swaps(plan->phases[p], ops)) return false;
        return true;
    }

    template <typename V>
    static void put_real(V &v, Real x) {
        uint32_t w[2] = {0, 0};
        memcpy(w, &x, sizeof(Real));
        v.push_back(w[0]);
        if (sizeof(Real) == 8) v.push_back(w[1]);
    }
    template <typename V>
    static void put_u64(V &v, uint64_t x) {
        v.push_back((uint32_t)x);
        v.push_back((uint32_t)(x >> 32));
    }

    // Ends the current window with S_NEXT (its w1 is set when the windows are known).
    void flush(uint32_t kind) {
        window.insert(window.end(), {kind | (1u << 8), 0u, 0u, 0u});
        windows.push_back(window.size() / 4);
        out.insert(out.end(), window.begin(), window.end());
        window.clear();
    }
    // Adds one op (whole units; word 0's unit count is set here).
    template <typename V>
    void add(uint32_t kind, V &&op) {
        while (op.size() % 4) op.push_back(0);
        const size_t units = op.size() / 4;
        op[0] = kind | (uint32_t)(units << 8);
        if (window.size() / 4 + units > CAP) flush(S_NEXT);
        window.insert(window.end(), op.begin(), op.end());
    }
    void add_scale() {
        if (scale == 1.0) return;  // FP32: always
        Words op = {0u, 0u};
        put_real(op, (Real)scale);
        add(S_SCALE, op);
        scale = 1.0;
    }
    void left_out(long double kappa) {
        scale *= kappa;
        const long double a = std::abs(scale);
        if (!(a < 0x1p200L && a > 0x1p-200L)) add_scale();
    }

    // byte offset in the transpose buffer of local index j (kernels.cuh)
    uint32_t slot(uint32_t j) const { return (j + (j >> R)) * (uint32_t)(2 * sizeof(Real)); }
    uint32_t reg_step(const Lay &l, int q) const { return q < R ? slot(1u << l.pos[5 + W + q]) : 0u; }
    uint32_t thread_step(const Lay &l, int b) const { return b < 5 + W ? slot(1u << l.pos[b]) : 0u; }

    void transpose(int from, int to, bool before, bool cross) {
        const Lay &f = plan->layouts[from], &t = plan->layouts[to];
        Words op = {0u, (before ? STREAM_SYNC_BEFORE : 0u) | (cross ? STREAM_SYNC_CROSS : 0u),
                                    reg_step(f, 4), reg_step(t, 4)};
        for (int q = 0; q < 4; q++) op.push_back(reg_step(f, q));
        for (int q = 0; q < 4; q++) op.push_back(reg_step(t, q));
        for (int b = 0; b < 8; b++) op.push_back(thread_step(t, b));
        add(S_TRANS, op);
        fresh = true;
        relabeled = 0;
    }

    void gate(const DevOp<Real> &d) {
        if (d.kind == K_SWAP && d.tpos < R && !d.cm_thr && !d.cm_glob && __builtin_popcount(d.cm_reg) == 1) {
            add(S_CSWAP, Words{0u, (uint32_t)d.tpos | (uint32_t)__builtin_ctz(d.cm_reg) << 16, d.cv_reg ? 1u : 0u, 0u});
            return;
        }
        Words op = {0u, (uint32_t)d.kind | ((uint32_t)d.tpos << 8), d.cm_reg, d.cv_reg,
                                    d.cm_thr, d.cv_thr, 0u, 0u};
        put_u64(op, d.cm_glob);
        put_u64(op, d.cv_glob);
        if (d.kind != K_SWAP)
            for (int k = 0; k < 8; k++) put_real(op, d.m[k]);
        add(S_GATE, op);
        if (d.kind == K_SWAP && d.tpos < R && !d.cm_reg) relabeled |= 1u << d.tpos;
    }

    // A layer of real or split gates: mats[k] is the record of the k-th bit of the mask.
    void layer(const DevOp<Real> &head, const DevOp<Real> *mats) {
        const uint32_t mask = head.cm_reg;
        const int n = __builtin_popcount(mask);
        const bool split = head.kind == K_LAYER_SPLIT;
        if (sizeof(Real) == 4) {
            Words op = {0u, mask, 0u, 0u};
            for (int i = 0; i < n; i++) {
                for (int j = 0; j < 4; j++) put_real(op, mats[i].m[split ? j : 2 * j]);
                if (split)
                    for (Real v : {mats[i].m[4], mats[i].m[5], (Real)0, (Real)0}) put_real(op, v);
            }
            add(split ? S_SPLIT : S_REAL, op);
            return;
        }
        // Each gate of a split layer in place where it has that form.  Where
        // one has not, it takes the phase and the real 2x2 (S_SPLIT, or a phase
        // gate and the real form on the lean build, run()), and the real gates of
        // the layer the real form.
        int bit[PB_MAX_R], at = 0;
        for (int b = 0; b < R; b++)
            if ((mask >> b) & 1u) bit[at++] = b;
        Rot form[PB_MAX_R];
        uint32_t in_place = 0, turned = 0;  // gates with that form; with a phase
        for (int i = 0; i < n && split; i++) {
            const Real *m = mats[i].m;
            const double rm[4] = {(double)m[0], (double)m[1], (double)m[2], (double)m[3]}, pr = m[4], pi = m[5];
            if (make_rot(rm, pr, pi, form[i]) || (!((relabeled >> bit[i]) & 1u) && make_lift(rm, pr, pi, form[i])))
                in_place |= 1u << bit[i];
            if (pr != 1.0 || pi != 0.0) turned |= 1u << bit[i];
        }
        if (in_place != mask) in_place &= turned;
        Words rot{0u, 0u, 0u, 0u}, had{0u, 0u, 0u, 0u}, real{0u, 0u, 0u, 0u}, general{0u, 0u, 0u, 0u};
        long double left = 1.0, left_had = 1.0;
        for (int i = 0; i < n; i++) {
            const Real *m = mats[i].m;
            const uint32_t b = 1u << bit[i];
            const double rm[4] = {(double)m[0], (double)m[split ? 1 : 2], (double)m[split ? 2 : 4], (double)m[split ? 3 : 6]};
            if (in_place & b) {
                const Rot &r = form[i];
                rot[1] |= b | (r.x ? b << 8 : 0u);
                for (double v : {r.t, r.u, r.pr, r.pi}) put_real(rot, (Real)v);
                left *= r.kappa;
            } else if ((turned & b) && !plan->lean) {
                general[1] |= b;
                for (double v : {rm[0], rm[1], rm[2], rm[3], (double)m[4], (double)m[5], 0.0, 0.0}) put_real(general, (Real)v);
            } else {
                if (turned & b) {
                    DevOp<Real> d;
                    memset(&d, 0, sizeof d);
                    d.kind = K_PHASE;
                    d.tpos = bit[i];
                    d.m[0] = (Real)1;
                    d.m[6] = m[4];
                    d.m[7] = m[5];
                    gate(d);
                    phase_gates++;
                }
                if (const long double a = hadamard_factor(rm); a != 0.0L) {
                    had[1] |= b;
                    left_had *= a;
                } else {
                    real[1] |= b;
                    for (double v : rm) put_real(real, (Real)v);
                }
            }
        }
        if (split) split_gates += n;
        if (rot[1]) {
            add(S_ROT, rot);
            relabeled |= rot[1] >> 8;
            left_out(left);
        }
        if (general[1]) add(S_SPLIT, general);
        if (had[1]) {
            add(S_HAD, had);
            left_out(left_had);
        }
        if (real[1]) add(S_REAL, real);
    }

    // The parts of a phase block: its terms by category in the kernel's walk
    // order (F, then G, H, D of each register bit), `per` units each, and its
    // table.  A block too large for a window goes out as several (each a
    // block of its own: factors multiply), the table with the last.
    int phase_block(const DevOp<Real> *rec) {
        const DevOp<Real> &head = rec[0];
        const bool angles = head.cm_reg & PB_ANGLES;
        uint8_t counts[16];
        memcpy(counts, head.m, 16);
        std::vector<int> order = {0};
        for (int b = 0; b < R; b++)
            for (int c : {1 + b, 1 + R + b, 1 + 2 * R + b}) order.push_back(c);
        const int total_terms = [&] {
            int t = 0;
            for (int c : order) t += counts[c];
            return t;
        }();
        // the terms' words, in walk order
        constexpr int per = pb_terms_per_record<Real>();
        const int tu = angles ? (int)sizeof(PhaseTerm<Real>) / 16 : 2 + (sizeof(Real) == 8 ? 2 : 1);
        std::vector<std::vector<uint32_t>> terms;
        for (int k = 0; k < total_terms; k++) {
            std::vector<uint32_t> t;
            if (angles) {
                t.resize(sizeof(PhaseTerm<Real>) / 4);
                memcpy(t.data(), reinterpret_cast<const unsigned char *>(rec + 1 + k / per) + (k % per) * sizeof(PhaseTerm<Real>),
                       sizeof(PhaseTerm<Real>));
            } else {
                const DevOp<Real> &d = rec[1 + k];
                t = {d.cm_thr, d.cv_thr, (uint32_t)d.tpos2, 0u};
                put_u64(t, d.cm_glob);
                put_u64(t, d.cv_glob);
                for (int j : {0, 1, 6, 7}) put_real(t, d.m[j]);
            }
            terms.push_back(t);
        }
        const int nrec = head.tpos;
        // a table of ones (a QFT block's on its lowest register bit) is left out
        bool table = false;
        for (int r = 0; (head.cm_reg & PB_HAS_TABLE) && r < (1 << R); r++) {
            const DevOp<Real> &z = rec[1 + nrec - (1 << R) / 4 + r / 4];
            table = table || z.m[2 * (r & 3)] != (Real)1 || z.m[2 * (r & 3) + 1] != (Real)0;
        }
        const int tab_units = table ? (int)((size_t(1) << R) * 2 * sizeof(Real) / 16) : 0;
        const int fit = ((int)CAP - 3 - tab_units) / tu;
        int done = 0;
        do {
            const int take = std::min(fit, total_terms - done);
            const bool last = done + take == total_terms;
            uint8_t cnt[16] = {0};
            uint32_t act = 0;
            int at = 0;
            for (int c : order) {
                for (int j = 0; j < counts[c]; j++, at++) {
                    if (at < done || at >= done + take) continue;
                    cnt[c]++;
                    act |= c == 0 ? PB_F_ACTIVE : 1u << ((c - 1) % R);
                }
            }
            uint32_t flags = head.cm_reg;
            if (!(last && done == 0)) flags &= ~PB_GATED;
            const bool tab = last && table;
            if (!tab) flags &= ~PB_HAS_TABLE;
            if (angles && fresh) {
                flags |= PB_FRESH;
                fresh = false;
            }
            std::vector<uint32_t> op = {0u, flags, act, tab ? (uint32_t)(3 + take * tu) : 0u};
            op.resize(12);
            memcpy(&op[4], cnt, 16);
            memcpy(&op[8], reinterpret_cast<const unsigned char *>(head.m) + 16, 8);
            for (int k = done; k < done + take; k++) op.insert(op.end(), terms[k].begin(), terms[k].end());
            if (tab)
                for (int r = 0; r < (1 << R); r++) {
                    const DevOp<Real> &z = rec[1 + nrec - (1 << R) / 4 + r / 4];
                    put_real(op, z.m[2 * (r & 3)]);
                    put_real(op, z.m[2 * (r & 3) + 1]);
                }
            add(angles ? S_PHASES : S_TERMS, op);
            done += take;
        } while (done < total_terms);
        return 1 + nrec;
    }

    void pass(const PassArgs &pa, const DevOp<Real> *ops, size_t n_ops, bool last_pass) {
        out.clear();
        window.clear();
        windows.clear();
        fresh = true;
        relabeled = 0;
        int cur = pa.load_layout;
        bool prev_cross = false;
        auto go_to = [&](int layout) {
            if (layout == cur) return;
            const bool cross = !same_warps(cur, layout);
            transpose(cur, layout, prev_cross || cross, cross);
            prev_cross = cross;
            cur = layout;
        };
        for (int p = pa.phase_begin; p < pa.phase_end; p++) {
            const DevPhase &ph = plan->phases[p];
            if (drop_swaps && only_swaps(ph, ops)) continue;
            go_to(ph.layout);
            for (int i = ph.op_begin; i < ph.op_end;) {
                const DevOp<Real> &d = ops[i];
                if (drop_swaps && swap_record(d)) {
                    i++;
                } else if (d.kind == K_PHASE_BLOCK) {
                    i += phase_block(ops + i);
                } else if (d.kind == K_LAYER_REAL || d.kind == K_LAYER_SPLIT) {
                    layer(d, ops + i + 1);
                    i += 1 + __builtin_popcount(d.cm_reg);
                } else if (d.kind == K_LAYER) {
                    const int k = __builtin_popcount(d.cm_reg);
                    Words op = {0u, d.cm_reg, 0u, 0u};
                    for (int j = 0; j < k; j++)
                        for (int e = 0; e < 8; e++) put_real(op, ops[i + 1 + j].m[e]);
                    add(S_DENSE, op);
                    i += 1 + k;
                } else if (d.kind == K_XSET) {
                    Words op = {0u, 0u};
                    for (int k = 0; k < d.tpos; k++) {
                        if (drop_swaps && ((d.pad1 >> k) & 1u)) continue;
                        uint32_t w;
                        memcpy(&w, reinterpret_cast<const unsigned char *>(d.m) + 4 * k, 4);
                        op.push_back(w);
                        op[1]++;
                        relabeled |= 1u << (w & 0xffu);
                    }
                    add(S_XSET, op);
                    i++;
                } else if (last_pass && i + 1 == (int)n_ops && global != 1.0) {
                    // the plan's scalar takes the factors left out with it
                    DevOp<Real> e = d;
                    e.m[0] = e.m[6] = (Real)(global.real() * scale);
                    e.m[1] = e.m[7] = (Real)(global.imag() * scale);
                    scale = 1.0;
                    gate(e);
                    i++;
                } else {
                    gate(d);
                    i++;
                }
            }
        }
        if (last_pass) add_scale();
        if (!(drop_swaps && coalesced(cur))) go_to(pa.store_layout);
        flush(S_END);

        TileArgs t;
        memset(&t, 0, sizeof t);
        t.stream = reinterpret_cast<const void *>(plan->stream.size() * 4);
        t.units0 = (int32_t)windows[0];
        t.units1 = windows.size() > 1 ? (int32_t)windows[1] : 0;
        // every S_NEXT names the units of the window after the one it enters
        size_t end = 0;
        for (size_t w = 0; w < windows.size(); w++) {
            end += windows[w];
            if (w + 2 < windows.size()) out[4 * (end - 1) + 1] = (uint32_t)windows[w + 2];
        }
        plan->stream.insert(plan->stream.end(), out.begin(), out.end());
        t.n = pa.n;
        t.k = pa.k;
        t.nruns = pa.nruns;
        static_assert(TILE_RUNS <= MAX_FREE_RUNS && 5 + PB_MAX_R + 3 + 1 <= TILE_RUNS, "runs of the largest tile");
        memcpy(t.run_pos, pa.run_pos, sizeof t.run_pos);
        memcpy(t.run_len, pa.run_len, sizeof t.run_len);
        memcpy(t.ld_gbit, pa.ld_gbit, sizeof t.ld_gbit);
        for (int k = 0; k < 5 + W + R; k++) t.st_gbit[k] = pa.tb[plan->layouts[cur].pos[k]];
        t.pass = (int32_t)(&pa - plan->passes.data());
        for (int b = 0; b < 8; b++) t.ld_tstep[b] = thread_step(plan->layouts[pa.load_layout], b);
        if (W == 0) t.ld_tstep[7] = (uint32_t)(CAP + 1) * 16u;
        plan->tiles.push_back(t);
    }

    // The permutation pass for `swaps`; false when its sub-tile cannot be
    // chosen: the low index bits (128-byte runs) with their partners, then
    // pairs, then bits that stay, PERM_BITS in all.
    bool permutation(const std::vector<std::pair<int, int>> &swaps, TileArgs &t) const {
        const int n = plan->qubits, low = sizeof(Real) == 8 ? 3 : 4;
        if (n < PERM_BITS || W < PERM_WARP_BITS) return false;
        int to[64];
        for (int b = 0; b < n; b++) to[b] = b;
        for (const auto &p : swaps) {
            to[p.first] = p.second;
            to[p.second] = p.first;
        }
        uint64_t in = 0;
        for (int b = 0; b < low; b++) in |= (uint64_t(1) << b) | (uint64_t(1) << to[b]);
        for (int want_pair = 1; want_pair >= 0; want_pair--)
            for (int b = 0; b < n; b++) {
                const uint64_t m = (uint64_t(1) << b) | (uint64_t(1) << to[b]);
                if ((in & m) || (to[b] != b) != (want_pair == 1)) continue;
                if (__builtin_popcountll(in | m) <= PERM_BITS) in |= m;
            }
        if (__builtin_popcountll(in) != PERM_BITS) return false;
        memset(&t, 0, sizeof t);
        int local[64], k = 0;
        for (int b = 0; b < n; b++)
            if ((in >> b) & 1) {
                t.ld_gbit[k] = (int8_t)b;
                local[b] = k++;
            }
        for (int q = 0; q < PERM_BITS; q++) t.st_gbit[q] = (int8_t)local[to[t.ld_gbit[q]]];
        for (int g = 0; g < n;) {
            if ((in >> g) & 1) {
                g++;
                continue;
            }
            int e = g;
            while (e < n && !((in >> e) & 1)) e++;
            if (t.nruns == TILE_RUNS) return false;
            t.run_pos[t.nruns] = (int8_t)g;
            t.run_len[t.nruns++] = (int8_t)(e - g);
            g = e;
        }
        int8_t *pair = reinterpret_cast<int8_t *>(t.ld_tstep);
        for (const auto &p : swaps) {
            if ((in >> p.first) & 1) continue;
            if (2 * (t.pairs + 1) > (int)sizeof t.ld_tstep) return false;
            pair[2 * t.pairs] = (int8_t)p.first;
            pair[2 * t.pairs + 1] = (int8_t)p.second;
            t.pairs++;
        }
        t.n = n;
        t.k = 5 + R + W;
        t.flags = PASS_PERMUTE;
        t.pass = -1;
        return true;
    }

    void run(const std::vector<std::pair<int, int>> &swaps) {
        const DevOp<Real> *ops = reinterpret_cast<const DevOp<Real> *>(plan->ops_bytes.data());
        const size_t n_ops = plan->ops_bytes.size() / sizeof(DevOp<Real>);
        // one permutation pass instead of the swaps when that saves a pass of
        // theirs: 15 qubits and up for a QFT.  Below, every pass has gates to
        // run, and the swaps ride along at less than a pass's fixed cost.
        TileArgs perm;
        size_t passes = plan->passes.size(), first = passes;
        while (first > 0 && only_swaps(plan->passes[first - 1], ops)) first--;
        drop_swaps = first < passes && first > 0 && global == 1.0 && !swaps.empty() && permutation(swaps, perm);
        if (drop_swaps) passes = first;
        const auto all = [&] {
            for (size_t p = 0; p < passes; p++) pass(plan->passes[p], ops, n_ops, p + 1 == passes);
        };
        all();
        // The lean build has no S_SPLIT in FP64: the branch alone cost layered
        // circuits 0.4%, while a phase gate costs a fifth of a gate of a
        // layer, and the full build a twentieth of the whole.  26 qubits, six
        // layers of gates with phases: a quarter of them not unitary 7.2 ms, all
        // 7.5 (8.8 and 9.8 where one such gate put its layer in the real form).
        if (plan->lean && 4 * phase_gates > split_gates) {
            plan->lean = false;
            plan->stream.clear();
            plan->tiles.clear();
            scale = 1.0;
            all();
        }
        if (drop_swaps) plan->tiles.push_back(perm);
    }
};

}  // namespace

void lower_plan(Plan *plan, cplx global, const std::vector<std::pair<int, int>> &swaps) {
    plan->stream.clear();
    plan->tiles.clear();
    if (plan->precision == HGM_F64) Lowering<double>(plan, global).run(swaps);
    else Lowering<float>(plan, global).run(swaps);
}

}  // namespace hgm
