// vcycle_common.cuh — per-cell V-cycle arithmetic shared by the graph kernels
// (vcycle.cu) and the distributed-shared-memory V-cycle (vcycle_dsm.cu).
//
// Restates MultiGridLevel::smooth_level (src/apic.rs:471-535), restrict
// (:537-594), prolongate (:596-616) and solve_coarse_exact (:618-704).
#pragma once

#include <cuda_runtime.h>

#include "apic_device.cuh"
#include "apic_internal.h"

namespace apic {
namespace vc {

constexpr float kOmega = 1.2f;
// "no preloaded segment word" (phases load seg[warp] themselves)
constexpr uint32_t kNoWord = 0xFFFFFFFFu;
constexpr int kTailThreads = 1024;
constexpr size_t kTailSmemBudget = 200 * 1024;

// ---- per-cell arithmetic shared by the global and the shared-memory kernels

// One SOR update (src/apic.rs:487-507) of padded cell c with raw index raw.
// nb(padded, raw) returns a neighbour's current error; neighbours that are not
// fluid are skipped (their reference contribution is zero).
template <class NB>
__device__ __forceinline__ float sor_cell(const uint32_t* bits, uint32_t w, uint32_t cells, const float* inv_d,
                                          const float* px, const float* py, const float* res, long long raw,
                                          uint32_t c, float old, bool neighbours, NB nb) {
    float inv = inv_d[c];
    if (inv == 0.0f) return old;
    float sum = res[c];
    if (neighbours) {
        const long long W = w;
        if (fluid_raw(bits, raw + 1, cells)) sum = __fmaf_rn(-px[c], nb(c + 1, raw + 1), sum);
        if (fluid_raw(bits, raw + W, cells)) sum = __fmaf_rn(-py[c], nb(c + w, raw + W), sum);
        if (fluid_raw(bits, raw - 1, cells)) sum = __fmaf_rn(-px[c - 1], nb(c - 1, raw - 1), sum);
        if (fluid_raw(bits, raw - W, cells)) sum = __fmaf_rn(-py[c - w], nb(c - w, raw - W), sum);
    }
    float gs = sum * inv;
    return old + (kOmega * (gs - old));
}

// Coarse residual of coarse cell (cx, cy) from its fine children (:549-583).
// E(padded, raw) gives the fine error of a fluid cell.
template <class E>
__device__ __forceinline__ float restrict_cell_fn(const uint32_t* fb, uint32_t fw, uint32_t fcells, const float* fd,
                                                  const float* fpx, const float* fpy, const float* fr, E fe,
                                                  uint32_t cx, uint32_t cy) {
    float sum = 0.0f;
    const long long W = fw;
    for (uint32_t dy = 0; dy < 2; ++dy)
        for (uint32_t dx = 0; dx < 2; ++dx) {
            long long rf = (long long)(cy * 2 + dy) * fw + (cx * 2 + dx);
            if (!fluid_raw(fb, rf, fcells)) continue;
            uint32_t pf = uint32_t(rf) + fw;
            float b = fr[pf];
            float ax = fd[pf] * fe(pf, rf);
            if (fluid_raw(fb, rf + 1, fcells)) ax += fpx[pf] * fe(pf + 1, rf + 1);
            if (fluid_raw(fb, rf + W, fcells)) ax += fpy[pf] * fe(pf + fw, rf + W);
            if (fluid_raw(fb, rf - 1, fcells)) ax += fpx[pf - 1] * fe(pf - 1, rf - 1);
            if (fluid_raw(fb, rf - W, fcells)) ax += fpy[pf - fw] * fe(pf - fw, rf - W);
            sum += b - ax;
        }
    return sum;
}

__device__ __forceinline__ float restrict_cell(const uint32_t* fb, uint32_t fw, uint32_t fcells, const float* fd,
                                               const float* fpx, const float* fpy, const float* fr, const float* fe,
                                               uint32_t cx, uint32_t cy) {
    return restrict_cell_fn(fb, fw, fcells, fd, fpx, fpy, fr, [fe](uint32_t p, long long) { return fe[p]; }, cx, cy);
}

// Branch-free forms of sor_cell / restrict_cell for the sweeps whose
// neighbour values are plain loads.  Every load is issued up front, without
// waiting for the fluid tests: all neighbours of a cell with raw index in
// [0, cells) have padded indices inside [0, cells + 2w), the extent of every
// level array.  Non-fluid neighbours (and children) are then dropped by
// selects, which yields the same floats as skipping them.  nb / fe must be
// safe to call for any such neighbour.
template <class NB>
__device__ __forceinline__ float sor_cell_all(const uint32_t* bits, uint32_t w, uint32_t cells, const float* inv_d,
                                              const float* px, const float* py, const float* res, long long raw,
                                              uint32_t c, float old, bool neighbours, NB nb) {
    const float inv = inv_d[c];
    float sum = res[c];
    if (neighbours) {
        const long long W = w;
        const bool fr = fluid_raw(bits, raw + 1, cells), fu = fluid_raw(bits, raw + W, cells);
        const bool fl = fluid_raw(bits, raw - 1, cells), fd = fluid_raw(bits, raw - W, cells);
        const float pxc = px[c], pyc = py[c], pxl = px[c - 1], pyd = py[c - w];
        const float er = nb(c + 1, raw + 1), eu = nb(c + w, raw + W), el = nb(c - 1, raw - 1), ed = nb(c - w, raw - W);
        float t = __fmaf_rn(-pxc, er, sum);
        sum = fr ? t : sum;
        t = __fmaf_rn(-pyc, eu, sum);
        sum = fu ? t : sum;
        t = __fmaf_rn(-pxl, el, sum);
        sum = fl ? t : sum;
        t = __fmaf_rn(-pyd, ed, sum);
        sum = fd ? t : sum;
    }
    const float gs = sum * inv;
    const float nv = old + (kOmega * (gs - old));
    return inv == 0.0f ? old : nv;
}

// Coarse residual of coarse cell (cx, cy) (any cell of the coarse grid).
__device__ __forceinline__ float restrict_cell_all(const uint32_t* fb, uint32_t fw, uint32_t fcells, const float* fd,
                                                   const float* fpx, const float* fpy, const float* fr,
                                                   const float* fe, uint32_t cx, uint32_t cy) {
    float sum = 0.0f;
    const long long W = fw;
#pragma unroll
    for (uint32_t dy = 0; dy < 2; ++dy)
#pragma unroll
        for (uint32_t dx = 0; dx < 2; ++dx) {
            const long long rf = (long long)(cy * 2 + dy) * fw + (cx * 2 + dx);
            const uint32_t pf = uint32_t(rf) + fw;
            const bool f0 = fluid_raw(fb, rf, fcells);
            const bool fr_ = fluid_raw(fb, rf + 1, fcells), fu = fluid_raw(fb, rf + W, fcells);
            const bool fl = fluid_raw(fb, rf - 1, fcells), fdn = fluid_raw(fb, rf - W, fcells);
            const float b = fr[pf];
            float ax = fd[pf] * fe[pf];
            float t = ax + fpx[pf] * fe[pf + 1];
            ax = fr_ ? t : ax;
            t = ax + fpy[pf] * fe[pf + fw];
            ax = fu ? t : ax;
            t = ax + fpx[pf - 1] * fe[pf - 1];
            ax = fl ? t : ax;
            t = ax + fpy[pf - fw] * fe[pf - fw];
            ax = fdn ? t : ax;
            t = sum + (b - ax);
            sum = f0 ? t : sum;
        }
    return sum;
}


// e + ec, plus ec again `reps` times (the padded base list, :611-615).
__device__ __forceinline__ float prolonged(float e, float ec, uint32_t reps) {
    e = e + ec;
    for (uint32_t k = 0; k < reps; ++k) e = e + ec;
    return e;
}

// ---- the coarsest level's CG -------------------------------------------------

// Sum (double-float) and a vote over the first `nwarps` warps of the CTA,
// returned to each of their threads: a shuffle tree per warp, one barrier of
// those warps, and the same tree over the warps' results in every warp, so
// no second barrier broadcasts it.  sh: one slot per warp; two calls in a row
// must use different slots (the barrier of the second then separates the
// readers of the first from its next writers).  A CG iteration is bound by the latency of
// its two sums.  In FP64, with every warp adding all warps' doubles, GB300's
// FP64 rate bound them: a PCG iteration of a 216^2 scene (27^2 coarsest
// cells) took 70.7 us, of a 488^2 one (61^2) 76.7, and now 48 and 59.  A
// double-float holds 48 bits of a sum that is rounded to 24: over 2700 random
// sums of 9 to 9375 products its rounded value was the FP64 sum's every time.
struct CgSlot {
    float4 w[32];
};
__device__ __forceinline__ void cg_bar(uint32_t nwarps) {
    asm volatile("bar.sync 1, %0;" ::"r"(nwarps * 32u) : "memory");
}
// any: whether it holds in any thread (kAny).
template <bool kAny>
__device__ __forceinline__ float cg_reduce(F2 v, bool& any, CgSlot& sh, uint32_t nwarps) {
    v = warp_sum(v);
    if (kAny) any = __any_sync(0xffffffffu, any);
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (lane == 0) sh.w[warp] = make_float4(v.hi, v.lo, kAny && any ? 1.0f : 0.0f, 0.0f);
    cg_bar(nwarps);
    const float4 q = lane < nwarps ? sh.w[lane] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    v = warp_sum(F2{q.x, q.y});
    if (kAny) any = __any_sync(0xffffffffu, q.z != 0.0f);
    return float(f2_value(v));
}

// The reference solver mode's sums (solve_coarse_exact, :627-629, :660,
// :681-687): the products, staged in fluid order, added one after another by
// one thread.  prod holds `n` products rounded up to a multiple of 8 with
// zeros behind them (a sum that starts at +0 is never -0, so adding +0
// changes nothing).  Loads run two groups ahead of the add chain, whose
// latency is all that is left.
__device__ __forceinline__ float serial_sum8(const float* prod, uint32_t n) {
    float s = 0.0f;
    float a[8], b[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) a[k] = n > 0 ? prod[k] : 0.0f;
    for (uint32_t i = 0; i < n; i += 8) {
#pragma unroll
        for (int k = 0; k < 8; ++k) b[k] = i + 8 < n ? prod[i + 8 + k] : 0.0f;
#pragma unroll
        for (int k = 0; k < 8; ++k) s = s + a[k];
#pragma unroll
        for (int k = 0; k < 8; ++k) a[k] = b[k];
    }
    return s;
}

// The level a CG runs on.  own: diag, px, py and cs lie in this CTA's shared
// memory and may be overwritten.
struct CgArrays {
    const uint32_t* bits;
    uint32_t w, cells;
    float *diag, *px, *py;
    const float* res;
    float *err, *cs, *cap, *cr;
    bool own;
};
constexpr uint32_t kCgMaxK = 10;  // cells per thread held in registers

// Plain CG on the coarsest level (solve_coarse_exact, :618-704) by the first
// `nwarps` warps of a CTA.  Cell k of a thread is threadIdx.x + k * threads.
// exact: the dot products are the reference's serial FP32 sums (reference
// solver mode).
//   K == 1: a cell's coefficients, vectors and the neighbours that count in
//     registers, the directions in cs.
//   K > 1:  the vectors of K cells in registers; diag, px and py (own) are
//     first zeroed wherever the reference skips a term, so the loops run over
//     all cells without a test (a term of zero leaves a sum as it was).
//   K == 0: everything in memory (levels of more than kCgMaxK cells per
//     thread).
struct CgShared {
    CgSlot slot[2];
    float dot;
    uint32_t pre[32 * kCgMaxK];  // exact: fluid cells before each mask word
};
template <int K>
static __device__ __noinline__ void cg_warps(const CgArrays& arrays, CgShared& sh, uint32_t nwarps, bool exact) {
    const CgArrays A = arrays;  // in registers: a barrier makes the compiler read memory again
    const uint32_t threads = nwarps * 32u;
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t W = A.w, cells = A.cells;
    const uint32_t nwords = (cells + 31u) >> 5;
    uint32_t nfl = 0;  // fluid cells of the level
    for (uint32_t k = lane; k < nwords; k += 32) nfl += uint32_t(__popc(A.bits[k]));
    nfl = __reduce_add_sync(0xffffffffu, nfl);
    if (K > 0 && exact) {
        for (uint32_t word = threadIdx.x; word < nwords; word += threads) {
            uint32_t c = 0;
            for (uint32_t k = 0; k < word; ++k) c += uint32_t(__popc(A.bits[k]));
            sh.pre[word] = c;
        }
    }
    // neighbours that count (right, left, up, down), bit 4: the cell is fluid
    auto links = [&](uint32_t r) -> uint32_t {
        if (r >= cells || !bit_at(A.bits, r)) return 0u;
        const long long q = r;
        return 16u | (fluid_raw(A.bits, q + 1, cells) ? 1u : 0u) | (fluid_raw(A.bits, q - 1, cells) ? 2u : 0u) |
               (fluid_raw(A.bits, q + W, cells) ? 4u : 0u) | (fluid_raw(A.bits, q - (long long)W, cells) ? 8u : 0u);
    };
    auto apply = [&](uint32_t c, uint32_t nb, float d, float sc, float pxc, float pxl, float pyc, float pyd) {
        // (all four loads first: they lie inside the padded array)
        const float sr = A.cs[c + 1], sl = A.cs[c - 1], su = A.cs[c + W], sd = A.cs[c - W];
        float v = d * sc;
        float t = __fmaf_rn(pxc, sr, v);
        v = (nb & 1u) ? t : v;
        t = __fmaf_rn(pxl, sl, v);
        v = (nb & 2u) ? t : v;
        t = __fmaf_rn(pyc, su, v);
        v = (nb & 4u) ? t : v;
        t = __fmaf_rn(pyd, sd, v);
        v = (nb & 8u) ? t : v;
        return v;
    };
    // exact sums: the fluid cells' products are staged at cap in fluid order
    auto stage = [&](uint32_t r, float q) {
        const uint32_t word = r >> 5, m = A.bits[word];
        if ((m >> lane) & 1u) A.cap[sh.pre[word] + uint32_t(__popc(m & ((1u << lane) - 1u)))] = q;
    };
    auto serial = [&]() {
        if (nfl + threadIdx.x < ((nfl + 7u) & ~7u)) A.cap[nfl + threadIdx.x] = 0.0f;
        cg_bar(nwarps);
        if (threadIdx.x == 0) sh.dot = serial_sum8(A.cap, nfl);
        cg_bar(nwarps);
        return sh.dot;
    };
    // ... or added up by thread 0 itself where the cells are in memory
    auto serial_cells = [&](const float* a, const float* b) {
        cg_bar(nwarps);
        if (threadIdx.x == 0) {
            float s = 0.0f;
            for (uint32_t r = 0; r < cells; ++r)
                if (bit_at(A.bits, r)) s = s + a[r + W] * b[r + W];
            sh.dot = s;
        }
        cg_bar(nwarps);
        return sh.dot;
    };
    constexpr int KR = K > 0 ? K : 1;
    uint32_t nb = 0;
    float d = 0.0f, pxc = 0.0f, pxl = 0.0f, pyc = 0.0f, pyd = 0.0f;  // K == 1
    float rv[KR], x[KR], av[KR];
#pragma unroll
    for (int k = 0; k < KR; ++k) rv[k] = x[k] = av[k] = 0.0f;
    F2 g{0.0f, 0.0f};
    bool more = false;
    if constexpr (K == 1) {
        if (exact) cg_bar(nwarps);  // sh.pre
        nb = links(threadIdx.x);
        if (nb) {
            const uint32_t c = threadIdx.x + W;
            d = A.diag[c];
            pxc = A.px[c];
            pxl = A.px[c - 1];
            pyc = A.py[c];
            pyd = A.py[c - W];
            rv[0] = A.res[c];
            A.cs[c] = rv[0];
        }
        const float q = rv[0] * rv[0];
        if (exact && nb) stage(threadIdx.x, q);
        g = F2{q, 0.0f};
    } else if constexpr (K > 1) {
        for (uint32_t c = threadIdx.x; c < cells + 2u * W; c += threads) {
            const long long r = (long long)c - W;
            const bool f = fluid_raw(A.bits, r, cells) != 0;
            if (!f || !fluid_raw(A.bits, r + 1, cells)) A.px[c] = 0.0f;
            if (!f || !fluid_raw(A.bits, r + W, cells)) A.py[c] = 0.0f;
            if (!f) A.diag[c] = 0.0f;
            A.cs[c] = f ? A.res[c] : 0.0f;
        }
        cg_bar(nwarps);
#pragma unroll
        for (int k = 0; k < K; ++k) {
            const uint32_t r = threadIdx.x + uint32_t(k) * threads;
            if (r >= cells) continue;
            rv[k] = A.cs[r + W];
            const float q = rv[k] * rv[k];
            if (exact) stage(r, q);
            g = f2_add(g, q);
        }
    } else {
        for (uint32_t r = threadIdx.x; r < cells; r += threads) {
            if (!bit_at(A.bits, r)) continue;
            const uint32_t c = r + W;
            const float q = A.res[c];
            A.err[c] = 0.0f;
            A.cr[c] = q;
            A.cs[c] = q;
            g = f2_add(g, q * q);
        }
    }
    float gamma;
    if (exact)
        gamma = K > 0 ? serial() : serial_cells(A.cr, A.cr);
    else
        gamma = cg_reduce<false>(g, more, sh.slot[0], nwarps);
    const uint32_t max_it = gamma < 1e-12f ? 0u : min(nfl, 100u);
    for (uint32_t it = 0; it < max_it; ++it) {
        // (the directions are visible: a barrier follows their update)
        F2 dsum{0.0f, 0.0f};
        if constexpr (K == 1) {
            float q = 0.0f;
            if (nb) {
                const uint32_t c = threadIdx.x + W;
                const float sc = A.cs[c];
                av[0] = apply(c, nb, d, sc, pxc, pxl, pyc, pyd);
                q = sc * av[0];
                if (exact) stage(threadIdx.x, q);
            }
            dsum = F2{q, 0.0f};
        } else if constexpr (K > 1) {
#pragma unroll
            for (int k = 0; k < K; ++k) {
                const uint32_t r = threadIdx.x + uint32_t(k) * threads;
                if (r >= cells) continue;
                const uint32_t c = r + W;
                const float sc = A.cs[c];
                float v = A.diag[c] * sc;
                v = __fmaf_rn(A.px[c], A.cs[c + 1], v);
                v = __fmaf_rn(A.px[c - 1], A.cs[c - 1], v);
                v = __fmaf_rn(A.py[c], A.cs[c + W], v);
                v = __fmaf_rn(A.py[c - W], A.cs[c - W], v);
                av[k] = v;
                const float q = sc * v;
                if (exact) stage(r, q);
                dsum = f2_add(dsum, q);
            }
        } else {
            for (uint32_t r = threadIdx.x; r < cells; r += threads) {
                const uint32_t n = links(r);
                if (!n) continue;
                const uint32_t c = r + W;
                const float sc = A.cs[c];
                const float v = apply(c, n, A.diag[c], sc, A.px[c], A.px[c - 1], A.py[c], A.py[c - W]);
                A.cap[c] = v;
                dsum = f2_add(dsum, sc * v);
            }
        }
        float delta;
        if (exact)
            delta = K > 0 ? serial() : serial_cells(A.cs, A.cap);
        else
            delta = cg_reduce<false>(dsum, more, sh.slot[1], nwarps);
        if (fabsf(delta) < 1e-5f) break;
        const float alpha = gamma / delta;
        more = false;  // some |r| is not below the exit (max|r| < 1e-6)
        F2 ng{0.0f, 0.0f};
        if constexpr (K > 0) {
#pragma unroll
            for (int k = 0; k < K; ++k) {
                const uint32_t r = threadIdx.x + uint32_t(k) * threads;
                if (r >= cells) continue;
                x[k] = x[k] + alpha * A.cs[r + W];
                rv[k] = rv[k] - alpha * av[k];
                more = more || fabsf(rv[k]) >= 1e-6f;
                const float q = rv[k] * rv[k];
                if (exact) stage(r, q);
                ng = K == 1 ? F2{q, 0.0f} : f2_add(ng, q);
            }
        } else {
            for (uint32_t r = threadIdx.x; r < cells; r += threads) {
                if (!bit_at(A.bits, r)) continue;
                const uint32_t c = r + W;
                A.err[c] = A.err[c] + alpha * A.cs[c];
                const float nr = A.cr[c] - alpha * A.cap[c];
                A.cr[c] = nr;
                more = more || fabsf(nr) >= 1e-6f;
                ng = f2_add(ng, nr * nr);
            }
        }
        // the exit's test and the next r.r in one reduction (the latter is
        // dropped when the former ends the loop)
        float new_gamma = cg_reduce<true>(ng, more, sh.slot[0], nwarps);
        if (!more) break;
        if (exact) new_gamma = K > 0 ? serial() : serial_cells(A.cr, A.cr);
        const float beta = new_gamma / gamma;
        gamma = new_gamma;
        if constexpr (K > 0) {
#pragma unroll
            for (int k = 0; k < K; ++k) {
                const uint32_t r = threadIdx.x + uint32_t(k) * threads;
                if (r >= cells || (K == 1 && !nb)) continue;
                A.cs[r + W] = rv[k] + (beta * A.cs[r + W]);
            }
        } else {
            for (uint32_t r = threadIdx.x; r < cells; r += threads) {
                if (!bit_at(A.bits, r)) continue;
                const uint32_t c = r + W;
                A.cs[c] = A.cr[c] + (beta * A.cs[c]);
            }
        }
        cg_bar(nwarps);
    }
    if constexpr (K > 0) {
#pragma unroll
        for (int k = 0; k < K; ++k) {
            const uint32_t r = threadIdx.x + uint32_t(k) * threads;
            if (r < cells && bit_at(A.bits, r)) A.err[r + W] = x[k];
        }
    }
}

// The same CG for a level of at most 32 cells (a grid whose sides halve down
// to 4 x 4), a cell per lane of one warp, all vectors in registers and the
// neighbours' directions by shuffle.  The sums are FP64 over the lanes (one
// warp's five adds are a shorter chain than the double-float's), or, exact,
// serial over the lanes; a lane that is not fluid adds +0.
static __device__ __noinline__ void cg_one_warp(const CgArrays& A, bool exact) {
    const uint32_t lane = threadIdx.x, W = A.w, cells = A.cells, c = lane + W;
    const uint32_t m = A.bits[0] & (cells < 32u ? (1u << cells) - 1u : 0xffffffffu);
    const bool on = (m >> lane) & 1u;
    auto fluid = [&](uint32_t l) { return on && l < 32u && ((m >> l) & 1u); };
    const bool fr = fluid(lane + 1u), fl = fluid(lane - 1u), fu = fluid(lane + W), fd = fluid(lane - W);
    float d = 0.0f, r = 0.0f, pr = 0.0f, pl = 0.0f, pu = 0.0f, pd = 0.0f, x = 0.0f;
    if (on) {
        d = A.diag[c];
        r = A.res[c];
        pr = fr ? A.px[c] : 0.0f;
        pl = fl ? A.px[c - 1] : 0.0f;
        pu = fu ? A.py[c] : 0.0f;
        pd = fd ? A.py[c - W] : 0.0f;
    }
    auto dot = [&](float q) {
        if (!exact) return float(warp_sum(double(q)));
        float t = 0.0f;
#pragma unroll 8
        for (int l = 0; l < 32; ++l) t = t + __shfl_sync(0xffffffffu, q, l);
        return t;
    };
    float s = r;
    float gamma = dot(r * r);
    const uint32_t max_it = gamma < 1e-12f ? 0u : min(uint32_t(__popc(m)), 100u);
    for (uint32_t it = 0; it < max_it; ++it) {
        const float sr = __shfl_sync(0xffffffffu, s, lane + 1u), sl = __shfl_sync(0xffffffffu, s, lane - 1u);
        const float su = __shfl_sync(0xffffffffu, s, lane + W), sd = __shfl_sync(0xffffffffu, s, lane - W);
        float v = d * s;
        v = fr ? __fmaf_rn(pr, sr, v) : v;
        v = fl ? __fmaf_rn(pl, sl, v) : v;
        v = fu ? __fmaf_rn(pu, su, v) : v;
        v = fd ? __fmaf_rn(pd, sd, v) : v;
        const float delta = dot(s * v);
        if (fabsf(delta) < 1e-5f) break;
        const float alpha = gamma / delta;
        x = x + alpha * s;
        r = r - alpha * v;
        if (!__any_sync(0xffffffffu, fabsf(r) >= 1e-6f)) break;
        const float new_gamma = dot(r * r);
        const float beta = new_gamma / gamma;
        gamma = new_gamma;
        s = r + (beta * s);
    }
    if (on) A.err[c] = x;
}

// A level of up to 32 cells takes one warp, up to 1024 one cell per thread of as many warps as that needs; above, all threads hold 4,
// 6 or 10 cells each; beyond 10240 cells (or without shared-memory copies to
// overwrite) the cells stay in memory.
static __device__ __forceinline__ void cta_coarse_cg(const CgArrays& A, bool exact) {
    __shared__ CgShared sh;
    const uint32_t need = (A.cells + 31u) >> 5, all = blockDim.x >> 5;
    const uint32_t nwarps = need < all ? need : all;
    if ((threadIdx.x >> 5) < nwarps) {
        if (need <= 1u)
            cg_one_warp(A, exact);
        else if (need <= all)
            cg_warps<1>(A, sh, nwarps, exact);
        else if (A.own && need <= 4u * all)
            cg_warps<4>(A, sh, nwarps, exact);
        else if (A.own && need <= 6u * all)
            cg_warps<6>(A, sh, nwarps, exact);
        else if (A.own && need <= kCgMaxK * all)
            cg_warps<int(kCgMaxK)>(A, sh, nwarps, exact);
        else
            cg_warps<0>(A, sh, nwarps, exact);
    }
    __syncthreads();
}

// ---- the coarse tail in shared memory ----------------------------------------
struct TailLevel {
    uint32_t w, h, cells, words, padded;
    int wshift;   // log2 w, or -1 when w is not a power of two
    const uint32_t* fluid;
    const float *diag, *inv, *px, *py;
    float* res;   // global residual (read for the first tail level)
    float* err;   // global error (written back for the first tail level)
    uint32_t o_bits, o_diag, o_inv, o_px, o_py, o_res, o_err;  // shared offsets, 4-byte units
};
struct TailParams {
    int n;                      // tail levels; lv[n - 1] is the coarsest
    int exact;                  // coarsest CG with the reference's serial FP32 sums
    uint32_t o_cs, o_cap, o_cr;  // coarse CG vectors
    TailLevel lv[kMaxLevels];
};

struct SmemLevel {
    uint32_t w, h, cells;
    int wshift;
    uint32_t* bits;
    float *diag, *inv, *px, *py, *res, *err;
};

__device__ __forceinline__ SmemLevel smem_level(uint32_t* sm, const TailLevel& t) {
    float* f = reinterpret_cast<float*>(sm);
    return SmemLevel{t.w,          t.h,          t.cells,      t.wshift,     sm + t.o_bits, f + t.o_diag,
                     f + t.o_inv,  f + t.o_px,   f + t.o_py,   f + t.o_res,  f + t.o_err};
}

// One colour sweep of a shared-memory level (w even: every level that is
// swept has a coarser one).  Thread t visits the colour's cells k = t,
// t + blockDim.x, ... directly, row by row, and skips the cells outside the
// fluid mask (their result is never stored).
__device__ __forceinline__ void cta_sweep(const SmemLevel& L, int color, int init) {
    const float* e = L.err;
    const uint32_t half = L.w >> 1;
    const int hs = L.wshift > 0 ? L.wshift - 1 : -1;
    const uint32_t n = L.h * half;
    for (uint32_t k = threadIdx.x; k < n; k += blockDim.x) {
        uint32_t kk, row;
        raw_xy(k, half, hs, kk, row);
        const uint32_t r = row * L.w + 2u * kk + ((row + uint32_t(color)) & 1u);
        if (!bit_at(L.bits, r)) continue;
        const uint32_t c = r + L.w;
        const float old = init ? 0.0f : e[c];
        L.err[c] = sor_cell_all(L.bits, L.w, L.cells, L.inv, L.px, L.py, L.res, r, c, old, !(init && color == 0),
                                [e](uint32_t p, long long) { return e[p]; });
    }
    __syncthreads();
}



// ---- sweep phases over a level's segment list -------------------------------
// `warp` / `nwarps`: this warp's index in the grid and the grid's warp count.
// Each phase visits every fluid cell of the level once (one warp per segment).

// One colour sweep; init: first sweep after the level's error was zero-filled.
// Every lane of the colour computes (its loads do not wait for the mask word)
// and only fluid cells store.
// w0: this warp's first segment word if the caller loaded it early
// (before waiting on the previous kernel), else kNoWord.
__device__ __forceinline__ void ph_smooth(const Level& L, uint32_t nseg, uint32_t warp, uint32_t nwarps, int color,
                                          int init, uint32_t w0 = kNoWord) {
    const uint32_t lane = threadIdx.x & 31;
    const float* e = L.err;
    for (uint32_t s = warp, nxt = seg_first(L.seg, nseg, warp, w0); s < nseg; s += nwarps) {
        const uint32_t word = nxt;
        nxt = seg_next(L.seg, nseg, s + nwarps);
        const uint32_t raw = word * 32 + lane;
        if (raw >= L.cells || int(!red_at(raw, L.w, L.wshift)) != color) continue;
        const bool fluid = (L.fluid[word] >> lane) & 1u;
        const uint32_t c = raw + L.w;
        const float old = init ? 0.0f : e[c];
        const float v = sor_cell_all(L.fluid, L.w, L.cells, L.inv_diag, L.px, L.py, L.res, raw, c, old,
                                     !(init && color == 0), [e](uint32_t p, long long) { return e[p]; });
        if (fluid) L.err[c] = v;
    }
}

// Asynchronous 4-byte copy global -> shared (cp.async, sm_80+): the copies
// of a whole array set are issued back to back and complete together at
// cp_async_wait_all, so loading costs about one L2 round trip instead of one
// per loop iteration.
__device__ __forceinline__ void cp_async4(void* smem, const void* gmem) {
    const uint32_t sa = static_cast<uint32_t>(__cvta_generic_to_shared(smem));
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(sa), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;\n" ::: "memory"); }
// 16-byte form (both addresses 16-byte aligned), through L2 only.
__device__ __forceinline__ void cp_async16(void* smem, const void* gmem) {
    const uint32_t sa = static_cast<uint32_t>(__cvta_generic_to_shared(smem));
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(sa), "l"(gmem) : "memory");
}

// Start copying every tail level's mask and coefficients into shared memory
// (complete after cp_async_wait_all).  The whole tail region is zeroed first:
// cells outside the fluid mask are never written, and with the stale shared
// memory of earlier kernels left in place the cluster-launched solve reached
// NaN (after other scenes had run in the process; the read that carried it
// was not located), while zeroed memory gives the same results as before.
__device__ __forceinline__ void cta_tail_issue_coeffs(const TailParams& tp, uint32_t* sm) {
    if (tp.n > 0) {
        const uint32_t words = tp.o_cr + tp.lv[tp.n - 1].padded;
        for (uint32_t i = threadIdx.x; i < words; i += blockDim.x) sm[i] = 0u;
        __syncthreads();  // zeroes land before any copy into the same words
    }
    for (int l = 0; l < tp.n; ++l) {
        const TailLevel& t = tp.lv[l];
        SmemLevel L = smem_level(sm, t);
        for (uint32_t i = threadIdx.x; i < t.words; i += blockDim.x) cp_async4(L.bits + i, t.fluid + i);
        for (uint32_t i = threadIdx.x; i < t.padded; i += blockDim.x) {
            cp_async4(L.diag + i, t.diag + i);
            cp_async4(L.inv + i, t.inv + i);
            cp_async4(L.px + i, t.px + i);
            cp_async4(L.py + i, t.py + i);
        }
    }
}

// Copy every tail level's mask and coefficients into shared memory.
__device__ __forceinline__ void cta_tail_load_coeffs(const TailParams& tp, uint32_t* sm) {
    cta_tail_issue_coeffs(tp, sm);
    cp_async_wait_all();
    __syncthreads();
}

// The coarse tail (levels held in shared memory) by one CTA.  load_coeffs:
// copy masks and coefficients first (otherwise they are already resident);
// the first level's residual is always copied in and its error copied out.
// load_coeffs false: the coefficients are resident or their copies were
// issued earlier by this CTA (cta_tail_issue_coeffs); the wait below covers
// those too.  global_io false: the first level's residual is already in
// shared memory and its error stays there (a cluster's other CTAs exchange
// them through distributed shared memory).
__device__ __forceinline__ void cta_tail(const TailParams& tp, uint32_t* sm, bool load_coeffs,
                                         bool global_io = true) {
    if (load_coeffs) cta_tail_issue_coeffs(tp, sm);
    if (global_io) {
        const TailLevel& t = tp.lv[0];
        SmemLevel L = smem_level(sm, t);
        for (uint32_t i = threadIdx.x; i < t.padded; i += blockDim.x) cp_async4(L.res + i, t.res + i);
    }
    cp_async_wait_all();
    __syncthreads();
    for (int l = 0; l + 1 < tp.n; ++l) {
        SmemLevel f = smem_level(sm, tp.lv[l]);
        SmemLevel c = smem_level(sm, tp.lv[l + 1]);
        cta_sweep(f, 0, 1);
        cta_sweep(f, 1, 1);
        for (uint32_t rc = threadIdx.x; rc < c.cells; rc += blockDim.x) {
            if (!bit_at(c.bits, rc)) continue;
            uint32_t cx, cy;
            raw_xy(rc, c.w, c.wshift, cx, cy);
            c.res[rc + c.w] = restrict_cell_all(f.bits, f.w, f.cells, f.diag, f.px, f.py, f.res, f.err, cx, cy);
        }
        __syncthreads();
    }
    {
        SmemLevel L = smem_level(sm, tp.lv[tp.n - 1]);
        float* fs = reinterpret_cast<float*>(sm);
        cta_coarse_cg(CgArrays{L.bits, L.w, L.cells, L.diag, L.px, L.py, L.res, L.err, fs + tp.o_cs, fs + tp.o_cap,
                               fs + tp.o_cr, true},
                      tp.exact != 0);
    }
    for (int l = tp.n - 2; l >= 0; --l) {
        SmemLevel f = smem_level(sm, tp.lv[l]);
        SmemLevel c = smem_level(sm, tp.lv[l + 1]);
        for (uint32_t r = threadIdx.x; r < f.cells; r += blockDim.x)
            if (bit_at(f.bits, r)) {
                uint32_t x, y;
                raw_xy(r, f.w, f.wshift, x, y);
                f.err[r + f.w] = f.err[r + f.w] + c.err[(y >> 1) * c.w + (x >> 1) + c.w];
            }
        __syncthreads();
        cta_sweep(f, 1, 0);
        cta_sweep(f, 0, 0);
    }
    if (!global_io) {
        __syncthreads();
        return;
    }
    const TailLevel& t = tp.lv[0];
    SmemLevel L = smem_level(sm, t);
    for (uint32_t r = threadIdx.x; r < t.cells; r += blockDim.x)
        if (bit_at(L.bits, r)) t.err[r + t.w] = L.err[r + t.w];
}

// Host: tail parameters for levels [first, s.nlevels) laid out in shared memory.
inline TailParams make_tail_params(const Scene& s, int first, uint32_t* words_out) {
    TailParams tp;
    tp.n = s.nlevels - first;
    tp.exact = coarse_cg_exact(s) ? 1 : 0;
    uint32_t off = 0;
    for (int k = 0; k < tp.n; ++k) {
        const Level& v = s.lv[first + k];
        TailLevel& t = tp.lv[k];
        t.w = v.w; t.h = v.h; t.cells = v.cells; t.words = v.words; t.padded = v.padded;
        t.wshift = -1;
        for (int k = 0; k < 31; ++k)
            if ((1u << k) == v.w) t.wshift = k;
        t.fluid = v.fluid; t.diag = v.diag; t.inv = v.inv_diag; t.px = v.px; t.py = v.py;
        t.res = v.res; t.err = v.err;
        t.o_bits = off; off += v.words;
        t.o_diag = off; off += v.padded;
        t.o_inv = off; off += v.padded;
        t.o_px = off; off += v.padded;
        t.o_py = off; off += v.padded;
        t.o_res = off; off += v.padded;
        t.o_err = off; off += v.padded;
    }
    uint32_t cp = s.lv[s.nlevels - 1].padded;
    tp.o_cs = off; off += cp;
    tp.o_cap = off; off += cp;
    tp.o_cr = off; off += cp;
    *words_out = off;
    return tp;
}

}  // namespace vc
}  // namespace apic
