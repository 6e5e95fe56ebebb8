// pcg_common.cuh — per-cell PCG phases on the base level, shared by the graph
// kernels (solver.cu) and the V-cycle (vcycle.cu).
//
// Restates Apic::solve_pcg (src/apic.rs:1865-1956) and apply_matrix_and_dot
// (:1823-1863).  Each phase visits the base fluid cells through the segment
// list (one warp per non-zero 32-cell mask word) and returns this thread's
// contribution to the phase's reduction; callers reduce deterministically.
#pragma once

#include <cuda_runtime.h>

#include "apic_device.cuh"
#include "apic_internal.h"

namespace apic {
namespace pcg {

#define APIC_BASE_LOOP(B, nseg, warp, nwarps)                                                          \
    const uint32_t lane_ = threadIdx.x & 31;                                                           \
    for (uint32_t s_ = (warp), nxt_ = seg_first((B).seg, (nseg), (warp), 0xFFFFFFFFu); s_ < (nseg);    \
         s_ += (nwarps))                                                                               \
        if (uint32_t word_ = seg_step((B).seg, (nseg), s_ + (nwarps), nxt_); ((B).fluid[word_] >> lane_) & 1u)

// The same loop over every lane of a segment inside the grid: the body runs
// without waiting for the mask word, so its loads issue at once, and tests
// fluid_ before it stores or accumulates.  All reads of a cell in [0, cells)
// and of its neighbours stay inside the padded arrays.
#define APIC_BASE_ALL(B, nseg, warp, nwarps) APIC_BASE_ALL_W0(B, nseg, warp, nwarps, 0xFFFFFFFFu)
// w0: the warp's first segment word when the caller loaded it early (before
// waiting on the previous kernel), else 0xFFFFFFFF.
#define APIC_BASE_ALL_W0(B, nseg, warp, nwarps, w0)                                                  \
    const uint32_t lane_ = threadIdx.x & 31;                                                         \
    for (uint32_t s_ = (warp), nxt_ = seg_first((B).seg, (nseg), (warp), (w0)); s_ < (nseg);        \
         s_ += (nwarps))                                                                             \
        if (const uint32_t word_ = seg_step((B).seg, (nseg), s_ + (nwarps), nxt_),                   \
            raw_ = word_ * 32 + lane_;                                                               \
            raw_ < (B).cells)                                                                        \
            if (const bool fluid_ = (((B).fluid[word_] >> lane_) & 1u) != 0u; true)

// pressure = 0 at fluid cells (src/apic.rs:1872-1883).
__device__ __forceinline__ void ph_clear_pressure(const Level& B, uint32_t nseg, uint32_t warp, uint32_t nwarps,
                                                  float* p) {
    APIC_BASE_LOOP(B, nseg, warp, nwarps) { p[word_ * 32 + lane_] = 0.0f; }
}

// s = z; returns r.z (src/apic.rs:1887-1888).  Dot products sum the FP32
// products in double-float (F2, apic_device.cuh).
__device__ __forceinline__ F2 ph_start(const Level& B, uint32_t nseg, uint32_t warp, uint32_t nwarps, float* s) {
    F2 acc{0.0f, 0.0f};
    APIC_BASE_ALL(B, nseg, warp, nwarps) {
        const uint32_t c = raw_ + B.w;
        const float z = B.err[c], r = B.res[c];
        if (!fluid_) continue;
        s[c] = z;
        acc = f2_add(acc, r * z);
    }
    return acc;
}

// ---- graph-path forms with the search update folded in -----------------------
// The search direction of an iteration, s' = z + beta s (:1945-1954), is not
// written by a kernel of its own: the SpMV evaluates it at the five stencil
// points from z and the previous s, and the update kernel, the last to read
// the previous s, stores it.  Both round exactly as the separate update would.
// With beta_valid == 0 (first iteration of a solve) s already holds z.

// s' at padded index q.
__device__ __forceinline__ float search_at(const float* z, const float* s, float beta, bool beta_valid, uint32_t q) {
    return beta_valid ? z[q] + (beta * s[q]) : s[q];
}

// Ap' = A s' at raw cell `raw` of the grid (the FMA chain of :1833-1846); *sc:
// s' there.
__device__ __forceinline__ float apply_search(const Level& B, uint32_t raw, const float* s, float beta,
                                              bool beta_valid, float* s_here) {
    const long long W = B.w, q = raw;
    const float* z = B.err;
    const uint32_t c = raw + B.w;
    const bool fr = fluid_raw(B.fluid, q + 1, B.cells), fl = fluid_raw(B.fluid, q - 1, B.cells);
    const bool fu = fluid_raw(B.fluid, q + W, B.cells), fd = fluid_raw(B.fluid, q - W, B.cells);
    const float sc = search_at(z, s, beta, beta_valid, c);
    const float sr = search_at(z, s, beta, beta_valid, c + 1), sl = search_at(z, s, beta, beta_valid, c - 1);
    const float su = search_at(z, s, beta, beta_valid, c + uint32_t(W));
    const float sd = search_at(z, s, beta, beta_valid, c - uint32_t(W));
    const float pxc = B.px[c], pxl = B.px[c - 1], pyc = B.py[c], pyd = B.py[c - W];
    float v = B.diag[c] * sc;
    float t = __fmaf_rn(pxc, sr, v);
    v = fr ? t : v;
    t = __fmaf_rn(pxl, sl, v);
    v = fl ? t : v;
    t = __fmaf_rn(pyc, su, v);
    v = fu ? t : v;
    t = __fmaf_rn(pyd, sd, v);
    v = fd ? t : v;
    *s_here = sc;
    return v;
}

// Ap' over the segments; returns s'.Ap'.
__device__ __forceinline__ F2 ph_spmv_search(const Level& B, uint32_t nseg, uint32_t warp, uint32_t nwarps,
                                             const float* s, float beta, bool beta_valid, float* ap,
                                             uint32_t w0 = 0xFFFFFFFFu) {
    F2 acc{0.0f, 0.0f};
    APIC_BASE_ALL_W0(B, nseg, warp, nwarps, w0) {
        float sc;
        const float v = apply_search(B, raw_, s, beta, beta_valid, &sc);
        if (!fluid_) continue;
        ap[raw_ + B.w] = v;
        acc = f2_add(acc, v * sc);
    }
    return acc;
}

// The same on a grid whose rows are whole vectors (w a multiple of four): a
// warp takes four segments, eight lanes each, a lane four cells with 16-byte
// loads.  w0: this lane's first segment word if the caller loaded it early.
// A cell at a time, the SpMV of a large level was bound by its instructions
// (140 per 32 cells, 57% of the issue slots, 2.8 times the DRAM time); now by
// the latency of its loads.  An iteration at 2048^2 (2.1 M fluid cells) 234.7 ->
// 228.4 us.
__device__ __forceinline__ F2 ph_spmv_search4(const Level& B, uint32_t nseg, uint32_t warp, uint32_t nwarps,
                                              const float* s, float beta, bool beta_valid, float* ap,
                                              uint32_t w0 = 0xFFFFFFFFu) {
    F2 acc{0.0f, 0.0f};
    const uint32_t lane = threadIdx.x & 31u, W = B.w;
    const float* z = B.err;
    auto four = [](const float* p) { return *reinterpret_cast<const float4*>(p); };
    auto search4 = [&](uint32_t q) {
        float4 v = four(s + q);
        if (beta_valid) {
            const float4 y = four(z + q);
            v = make_float4(y.x + (beta * v.x), y.y + (beta * v.y), y.z + (beta * v.z), y.w + (beta * v.w));
        }
        return v;
    };
    // mask bits of the four cells from raw on (raw a multiple of four)
    auto bits4 = [&](long long raw) -> uint32_t {
        return raw >= 0 && raw < (long long)B.cells ? (B.fluid[raw >> 5] >> (raw & 31)) & 15u : 0u;
    };
    for (uint32_t q0 = 4u * warp; q0 < nseg; q0 += 4u * nwarps) {
        const uint32_t q = q0 + (lane >> 3);
        if (q >= nseg) continue;
        const uint32_t word = q0 == 4u * warp && w0 != 0xFFFFFFFFu ? w0 : B.seg[q];
        const uint32_t raw = word * 32u + 4u * (lane & 7u), c = raw + W;
        if (raw >= B.cells) continue;
        const uint32_t m = bits4(raw), up = bits4((long long)raw + W), dn = bits4((long long)raw - W);
        const uint32_t side = fluid_raw(B.fluid, (long long)raw - 1, B.cells) |
                              (fluid_raw(B.fluid, (long long)raw + 4, B.cells) << 1);
        const float4 sc = search4(c), su = search4(c + W), sd = search4(c - W);
        const float sl = search_at(z, s, beta, beta_valid, c - 1), sr = search_at(z, s, beta, beta_valid, c + 4);
        const float4 dg = four(B.diag + c), px = four(B.px + c), py = four(B.py + c), pyd = four(B.py + c - W);
        const float pxl = B.px[c - 1];
        const float cs[6] = {sl, sc.x, sc.y, sc.z, sc.w, sr};
        const float xs[5] = {pxl, px.x, px.y, px.z, px.w}, d[4] = {dg.x, dg.y, dg.z, dg.w};
        const float ys[4] = {py.x, py.y, py.z, py.w}, yd[4] = {pyd.x, pyd.y, pyd.z, pyd.w};
        const float us[4] = {su.x, su.y, su.z, su.w}, ds[4] = {sd.x, sd.y, sd.z, sd.w};
        const uint32_t right = (m >> 1) | ((side & 2u) << 2), left = (m << 1) | (side & 1u);
        float v[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            float a = d[k] * cs[k + 1];
            float t = __fmaf_rn(xs[k + 1], cs[k + 2], a);
            a = (right >> k) & 1u ? t : a;
            t = __fmaf_rn(xs[k], cs[k], a);
            a = (left >> k) & 1u ? t : a;
            t = __fmaf_rn(ys[k], us[k], a);
            a = (up >> k) & 1u ? t : a;
            t = __fmaf_rn(yd[k], ds[k], a);
            a = (dn >> k) & 1u ? t : a;
            v[k] = (m >> k) & 1u ? a : 0.0f;
            if ((m >> k) & 1u) acc = f2_add(acc, a * cs[k + 1]);
        }
        if (m) *reinterpret_cast<float4*>(ap + c) = make_float4(v[0], v[1], v[2], v[3]);
    }
    return acc;
}

// (grids without a coarser level; the others update in the base level's down
// kernel, tiles.cuh)  x += alpha s', r = fma(-alpha, Ap, r) (:1910-1928), s = s'; and on red
// cells the preconditioner's first sweep from zero error, which needs only
// the cell's new residual: z = 0 + omega (r / diag - 0) (smooth_level
// :487-507 with every neighbour still zero).  Returns max|r| and sum r^2.
__device__ __forceinline__ void ph_update_search(const Level& B, uint32_t nseg, uint32_t warp, uint32_t nwarps,
                                                 float alpha, float beta, bool beta_valid, float* x, int x_padded,
                                                 float* s, const float* ap, float* max_r, F2* r2,
                                                 uint32_t w0 = 0xFFFFFFFFu) {
    constexpr float kOmegaSor = 1.2f;
    float mx = 0.0f;
    F2 acc{0.0f, 0.0f};
    APIC_BASE_ALL_W0(B, nseg, warp, nwarps, w0) {
        const uint32_t c = raw_ + B.w;
        const uint32_t xi = x_padded ? c : raw_;
        const float sc = search_at(B.err, s, beta, beta_valid, c);
        const float nx = x[xi] + alpha * sc;
        const float nr = __fmaf_rn(-alpha, ap[c], B.res[c]);
        const float inv = B.inv_diag[c];
        if (!fluid_) continue;
        s[c] = sc;
        x[xi] = nx;
        B.res[c] = nr;
        if (red_at(raw_, B.w, B.wshift))
            B.err[c] = inv != 0.0f ? 0.0f + (kOmegaSor * (nr * inv - 0.0f)) : 0.0f;
        mx = fmaxf(mx, fabsf(nr));
        acc = f2_add(acc, f2_square(nr));
    }
    *max_r = mx;
    *r2 = acc;
}

// gamma' = r.z ends the reference mode's iteration (:1934-1943): beta, or
// the exit when r.z is below SAFTY.  Run by one thread.  (The relative modes
// form beta at the start of the next iteration, where a zero r.z ends the
// solve.)
__device__ __forceinline__ void finish_rz_reference(Ctl* ctl, float ng) {
    constexpr float kSafetyRz = 1e-5f;  // SAFTY, src/apic.rs:8
    if (ng < kSafetyRz) {
        ctl->pcg_done = 1;
        return;
    }
    ctl->beta = ng / ctl->gamma;
    ctl->beta_valid = 1;
    ctl->gamma = ng;
}

// After the residual's exit test: whether the PCG loop goes on (not
// converged, under the iteration cap; dyn_cap reads the remaining budget of a
// refinement).  In the relative modes a continuing loop's next iteration
// forms beta from the r.z parts that this iteration's V-cycle stores
// (beta_valid); the reference mode's k_gamma_exact does that itself.  A loop
// that ends at the cap is marked in pcg_done too: the loop's body holds several
// iterations, and those after the last must do nothing.  Run by thread 0 of
// one block; loop_decision sets the graph's loop condition when set_cond.
__device__ __forceinline__ bool loop_continue(Ctl* ctl, int mode, uint32_t cap, int dyn_cap) {
    const uint32_t c = dyn_cap ? ctl->inner_cap : cap;
    const bool cont = !ctl->pcg_done && ctl->pcg_iters < c;
    if (mode != APIC_SOLVER_REFERENCE) {
        if (cont) ctl->beta_valid = 1;
        else if (!ctl->pcg_done) ctl->pcg_done = kStoppedAtCap;
    }
    return cont;
}
__device__ __forceinline__ void loop_decision(Ctl* ctl, int mode, cudaGraphConditionalHandle h, uint32_t cap,
                                              int dyn_cap, int set_cond) {
    const bool cont = loop_continue(ctl, mode, cap, dyn_cap);
    if (set_cond) cudaGraphSetConditional(h, cont ? 1u : 0u);
}

// The exits that the update leaves to the next kernel: its delta stop, or
// the residual test on its block parts, max|r| < solve_error (reference
// mode, src/apic.rs:1929-1932) or ||r|| <= target * ||b||.  Run by one
// block, after the caller's dependency wait.
__device__ __forceinline__ void residual_exit(Ctl* ctl, const float4* part, uint32_t n, int mode, float solve_error) {
    if (ctl->delta_stop) {  // s.Ap was unusable: no update, no residual parts
        if (threadIdx.x == 0) {
            ctl->pcg_done = 1;
            ctl->res_sel ^= 1u;  // the update left the residual where it was
        }
        return;
    }
    double tot;
    float t;
    sum_max_partials<kSegBlock>(part, n, &tot, &t);
    if (threadIdx.x == 0) {
        if (mode == APIC_SOLVER_REFERENCE) {
            ctl->max_r_bits = __float_as_uint(t);
            if (t < solve_error) ctl->pcg_done = 1;
        } else {
            ctl->rnorm2 = tot;
            if (tot <= ctl->stop2) ctl->pcg_done = 1;
        }
    }
}

// ||r||^2 at which a solve relative to ||b|| has converged; formed once, by
// the thread that sets the target, so that the test in an iteration is a
// comparison (a division and a square root in FP64 took 0.6 us of it).
__device__ __forceinline__ void set_target(Ctl* ctl, double rel) {
    ctl->target_rel = rel;
    ctl->stop2 = ctl->bnorm2 > 0.0 ? rel * rel * ctl->bnorm2 : HUGE_VAL;
}

// Base residual: the buffer that holds it now.
__device__ __forceinline__ const float* cur_res(const Level& B, const Ctl* ctl) {
    return ctl->res_sel && B.res2 ? B.res2 : B.res;
}

// In every CTA of a kernel whose CTAs all go on or all return (a cluster, a
// single CTA): whether the solve is over.  After an update (a.on) each CTA sums
// the residual's parts itself, to the same verdict, and `writer`'s thread 0
// records it and takes the loop decision, also where the update itself ended
// the solve (else the loop would go on without end).  One thread reads
// pcg_done: the writer may set it meanwhile, and a CTA's threads must agree.
__device__ __forceinline__ bool solve_over(Ctl* ctl, const ExitArgs& a, bool writer) {
    if (!a.on) return ctl->pcg_done != 0;
    __shared__ bool s_done;
    uint32_t was_done = 0, delta_stop = 0, iters = 0, cap = 0;
    double stop2 = 0.0, tot;
    float t;
    if (threadIdx.x == 0) {  // (on their way during the sum)
        was_done = ctl->pcg_done;
        delta_stop = ctl->delta_stop;
        iters = ctl->pcg_iters;
        cap = a.dyn_cap ? ctl->inner_cap : a.cap;
        stop2 = ctl->stop2;
    }
    sum_max_partials<kSegBlock>(a.part, a.nparts, &tot, &t);
    if (threadIdx.x == 0) {
        const bool before = was_done != 0, stop = !before && delta_stop != 0;
        bool done = before || stop;
        if (!done && a.mode == APIC_SOLVER_REFERENCE) done = t < a.solve_error;
        else if (!done) done = tot <= stop2;
        // (at the iteration cap every CTA returns, as the decision marks it)
        s_done = done || (a.mode != APIC_SOLVER_REFERENCE && iters >= cap);
        if (writer) {
            if (stop) ctl->res_sel ^= 1u;  // the update left the residual where it was
            else if (!before && a.mode == APIC_SOLVER_REFERENCE) ctl->max_r_bits = __float_as_uint(t);
            else if (!before) ctl->rnorm2 = tot;
            if (done && !before) ctl->pcg_done = 1;
            loop_decision(ctl, a.mode, a.h, a.cap, a.dyn_cap, a.set_cond);
        }
    }
    __syncthreads();
    return s_done;
}

// r.z after the preconditioner (:1936).
__device__ __forceinline__ F2 ph_rz(const Level& B, uint32_t nseg, uint32_t warp, uint32_t nwarps) {
    F2 acc{0.0f, 0.0f};
    APIC_BASE_ALL(B, nseg, warp, nwarps) {
        const uint32_t c = raw_ + B.w;
        const float rz = B.res[c] * B.err[c];
        if (fluid_) acc = f2_add(acc, rz);
    }
    return acc;
}

// ---- FP64 refinement (APIC_SOLVER_REL_MIXED) ---------------------------------

// b64 = res, p64 = 0; returns ||b||^2.
// warm: keep p64 as the previous solve left it (the initial guess of the
// refinement), else start from zero.
__device__ __forceinline__ double ph_mixed_init(const Level& B, uint32_t nseg, uint32_t warp, uint32_t nwarps,
                                                double* b64, double* p64, int warm) {
    double bb = 0;
    APIC_BASE_ALL(B, nseg, warp, nwarps) {
        const uint32_t c = raw_ + B.w;
        const double b = double(B.res[c]);
        if (!fluid_) continue;
        b64[c] = b;
        if (!warm) p64[c] = 0.0;
        bb += b * b;
    }
    return bb;
}

// r64 = b64 - A p64 in FP64; flags bit 0: res = float(r64), bit 1: x = 0.
// Returns ||r64||^2.
__device__ __forceinline__ double ph_true_residual(const Level& B, uint32_t nseg, uint32_t warp, uint32_t nwarps,
                                                   const double* b64, const double* p64, float* x, int flags) {
    double rr = 0;
    const uint32_t W = B.w;
    // every load is issued before the fluid tests (all neighbours of a cell
    // inside the grid lie inside the padded arrays); non-fluid neighbours
    // are dropped by selects, which adds exactly what skipping them adds
    APIC_BASE_ALL(B, nseg, warp, nwarps) {
        const uint32_t c = raw_ + W;
        const long long raw = raw_;
        const float dg = B.diag[c], pxc = B.px[c], pxl = B.px[c - 1], pyc = B.py[c], pyd = B.py[c - W];
        const double pc = p64[c], pr = p64[c + 1], pl = p64[c - 1], pu = p64[c + W], pd = p64[c - W], bc = b64[c];
        const bool fr = fluid_raw(B.fluid, raw + 1, B.cells), fl = fluid_raw(B.fluid, raw - 1, B.cells);
        const bool fu = fluid_raw(B.fluid, raw + W, B.cells), fd = fluid_raw(B.fluid, raw - (long long)W, B.cells);
        double v = double(dg) * pc;
        double t = v + double(pxc) * pr;
        v = fr ? t : v;
        t = v + double(pxl) * pl;
        v = fl ? t : v;
        t = v + double(pyc) * pu;
        v = fu ? t : v;
        t = v + double(pyd) * pd;
        v = fd ? t : v;
        if (!fluid_) continue;
        const double r = bc - v;
        rr += r * r;
        if (flags & 1) B.res[c] = float(r);
        if (flags & 2) x[c] = 0.0f;
    }
    return rr;
}

// A relative solve's start in one pass: b64 = res, pressure = 0 and ||b||^2
// (x), and for refinement (mixed) the true residual of the starting p64
// (ph_true_residual's terms: kept where warm, else zero, whose residual is b),
// x = 0 and its ||r||^2 (y).
__device__ __forceinline__ double2 ph_solve_start(const Level& B, uint32_t nseg, uint32_t warp, uint32_t nwarps,
                                                  double* b64, double* p64, float* x, float* pressure, int warm,
                                                  int mixed) {
    double bb = 0.0, rr = 0.0;
    const uint32_t W = B.w;
    APIC_BASE_ALL(B, nseg, warp, nwarps) {
        const uint32_t c = raw_ + W;
        const long long raw = raw_;
        const float res = B.res[c];
        const double b = double(res);
        double r = b;
        if (warm) {
            const float dg = B.diag[c], pxc = B.px[c], pxl = B.px[c - 1], pyc = B.py[c], pyd = B.py[c - W];
            const double pc = p64[c], pr = p64[c + 1], pl = p64[c - 1], pu = p64[c + W], pd = p64[c - W];
            const bool fr = fluid_raw(B.fluid, raw + 1, B.cells), fl = fluid_raw(B.fluid, raw - 1, B.cells);
            const bool fu = fluid_raw(B.fluid, raw + W, B.cells);
            const bool fd = fluid_raw(B.fluid, raw - (long long)W, B.cells);
            double v = double(dg) * pc;
            double t = v + double(pxc) * pr;
            v = fr ? t : v;
            t = v + double(pxl) * pl;
            v = fl ? t : v;
            t = v + double(pyc) * pu;
            v = fu ? t : v;
            t = v + double(pyd) * pd;
            v = fd ? t : v;
            r = b - v;
        }
        if (!fluid_) continue;
        b64[c] = b;
        pressure[raw_] = 0.0f;
        bb += b * b;
        if (!warm) p64[c] = 0.0;
        if (!mixed) continue;
        rr += r * r;
        if (warm) B.res[c] = float(r);
        x[c] = 0.0f;
    }
    return make_double2(bb, rr);
}

// p64 += x, or (finalize) pressure = float(p64).
__device__ __forceinline__ void ph_accumulate(const Level& B, uint32_t nseg, uint32_t warp, uint32_t nwarps,
                                              double* p64, const float* x, float* pressure, int finalize) {
    APIC_BASE_ALL(B, nseg, warp, nwarps) {
        const uint32_t c = raw_ + B.w;
        const double p = p64[c];
        const float xv = finalize ? 0.0f : x[c];
        if (!fluid_) continue;
        if (!finalize) p64[c] = p + double(xv);
        else pressure[raw_] = float(p);
    }
}

// p64 = pressure (the FP32 pressure the projection uses, for its true residual).
__device__ __forceinline__ void ph_pressure_to64(const Level& B, uint32_t nseg, uint32_t warp, uint32_t nwarps,
                                                 const float* pressure, double* p64) {
    APIC_BASE_LOOP(B, nseg, warp, nwarps) {
        uint32_t raw = word_ * 32 + lane_;
        p64[raw + B.w] = double(pressure[raw]);
    }
}

#undef APIC_BASE_LOOP

}  // namespace pcg
}  // namespace apic
