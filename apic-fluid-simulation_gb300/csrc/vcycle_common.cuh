// vcycle_common.cuh — per-cell V-cycle arithmetic shared by the graph kernels
// (vcycle.cu) and the distributed-shared-memory V-cycle (vcycle_dsm.cu).
//
// Restates MultiGridLevel::smooth_level (src/apic.rs:471-535), restrict
// (:537-594), prolongate (:596-616) and solve_coarse_exact (:618-704).
#pragma once

#include <cuda_runtime.h>

#include <cstring>

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
// Every load is issued up front, without waiting for the fluid tests: all
// neighbours of a cell with raw index in [0, cells) have padded indices
// inside [0, cells + 2w), the extent of every level array.  Non-fluid
// neighbours are then dropped by selects, which yields the same floats as
// skipping them.  nb must be safe to call for any such neighbour.
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

// e + ec, plus ec again `reps` times (the padded base list, :611-615).
__device__ __forceinline__ float prolonged(float e, float ec, uint32_t reps) {
    e = e + ec;
    for (uint32_t k = 0; k < reps; ++k) e = e + ec;
    return e;
}

// ---- the coarsest level's CG -------------------------------------------------

// Sum, rounded to FP32, and a vote over the first `nwarps` warps of the CTA,
// returned to each of their threads: a shuffle tree per warp, one barrier of
// those warps, and the same tree over the warps' results in every warp, so
// no second barrier broadcasts it.  sh: one slot per warp; two calls in a row
// must use different slots (the barrier of the second then separates the
// readers of the first from its next writers).  A CG iteration is bound by the latency of
// its two sums.  In FP64, with every warp adding all warps' doubles, GB300's
// FP64 rate bound them: a PCG iteration of a 216^2 scene (27^2 coarsest
// cells) took 70.7 us, of a 488^2 one (61^2) 76.7, and 48 and 59 with
// double-float sums.  A double-float holds 48 bits where FP64 holds 53, so the
// result is checked: where the sum could round to another float within its
// error bound, or is not finite (a double-float overflows to NaN), the terms are
// summed again in FP64: one in some 5000 sums of random squares, one in 100 of
// random terms of both signs, and no rounded sum of 83000 was wrong.  The check
// takes 0.2 us of an iteration with 27^2 coarsest cells (33.5 -> 33.7), 0.8 with
// 61^2 (41.5 -> 42.3) and 2.6 with 125 x 75 (62.0 -> 64.5).
struct CgSlot {
    float4 w[32];
};
__device__ __forceinline__ void cg_bar(uint32_t nwarps) {
    asm volatile("bar.sync 1, %0;" ::"r"(nwarps * 32u) : "memory");
}
// The sum in FP64 of a, or a b, over the cells of each thread (r, r + threads,
// ...: those it wrote itself) that bits holds; every thread of the warps takes part.
static __device__ __noinline__ float cg_sum64(const float* a, const float* b, const uint32_t* bits, uint32_t cells,
                                              double* wide, uint32_t nwarps) {
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    double t = 0.0;
    for (uint32_t r = threadIdx.x; r < cells; r += nwarps * 32u)
        if (bit_at(bits, r)) t += double(b ? a[r] * b[r] : a[r]);
    t = warp_sum(t);
    if (lane == 0) wide[warp] = t;
    cg_bar(nwarps);
    return float(warp_sum(lane < nwarps ? wide[lane] : 0.0));
}
// A thread's terms of a sum: their double-float sum and, where they may have both
// signs, the sum of their magnitudes.
struct CgTerms {
    F2 v{0.0f, 0.0f};
    float mag = 0.0f;
    template <bool kSigned> __device__ __forceinline__ void add(float q) {
        v = f2_add(v, q);
        if (kSigned) mag += fabsf(q);
    }
    template <bool kSigned> __device__ __forceinline__ void set(float q) {
        v = F2{q, 0.0f};
        if (kSigned) mag = fabsf(q);
    }
};
// any: whether it holds in any thread (kAny).  eps: the error bound of a sum, in
// units of its terms' magnitudes (bounded by the largest of a thread's times
// the threads: two votes instead of ten shuffles); sum64(): the sum in FP64.
// exact: only the vote counts.
template <bool kAny, bool kSigned, class Sum64>
__device__ __forceinline__ float cg_reduce(const CgTerms& t, bool& any, CgSlot& sh, uint32_t nwarps, float eps,
                                           bool exact, Sum64 sum64) {
    F2 v = t.v;
    float mag = t.mag;
    if (kSigned) mag = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(mag)));
    v = warp_sum(v);
    if (kAny) any = __any_sync(0xffffffffu, any);
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (lane == 0) sh.w[warp] = make_float4(v.hi, v.lo, kAny && any ? 1.0f : 0.0f, mag);
    cg_bar(nwarps);
    // (up to 8 warps: four copies of their results, three levels of the tree)
    const uint32_t from = nwarps <= 8u ? lane & 7u : lane;
    const float4 q = from < nwarps ? sh.w[from] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    v = F2{q.x, q.y};
    if (kSigned) mag = float(nwarps * 32u) * __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(q.w)));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        if (o > 4 && nwarps <= 8u) continue;
        v = f2_add(v, F2{__shfl_xor_sync(0xffffffffu, v.hi, o), __shfl_xor_sync(0xffffffffu, v.lo, o)});
    }
    if (kAny) any = __any_sync(0xffffffffu, q.z != 0.0f);
    // (the same in every warp: the same values through the same tree)
    const float e = eps * (kSigned ? mag : v.hi), up = v.hi + (v.lo + e), down = v.hi + (v.lo - e);
    if (up == down || exact) return up;
    return sum64();
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

// The level a CG runs on.
struct CgArrays {
    const uint32_t* bits;
    uint32_t w, cells;
    float *diag, *px, *py;
    const float* res;
    float *err, *cs, *cap, *cr;
};
constexpr uint32_t kCgMaxK = 10;  // cells per thread held in registers

// Plain CG on the coarsest level (solve_coarse_exact, :618-704) by the first
// `nwarps` warps of a CTA.  Cell k of a thread is threadIdx.x + k * threads.
// exact: the dot products are the reference's serial FP32 sums (reference
// solver mode).
//   K == 1: a cell's coefficients and vectors in registers, the directions in
//     cs.
//   K > 1:  the vectors of K cells in registers.
//   K == 0: everything in memory (levels of more than kCgMaxK cells per
//     thread).
// The coefficients are zero outside the fluid and so are the directions, so a
// term that the reference skips adds zero.
struct CgShared {
    CgSlot slot[2];
    double wide[32];
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
    auto count = [&] {
        for (uint32_t k = lane; k < nwords; k += 32) nfl += uint32_t(__popc(A.bits[k]));
        nfl = __reduce_add_sync(0xffffffffu, nfl);
    };
    if (exact) {
        count();
        if (K > 0)
            for (uint32_t word = threadIdx.x; word < nwords; word += threads) {
                uint32_t c = 0;
                for (uint32_t k = 0; k < word; ++k) c += uint32_t(__popc(A.bits[k]));
                sh.pre[word] = c;
            }
    }
    auto apply = [&](uint32_t c, float d, float sc, float pxc, float pxl, float pyc, float pyd) {
        float v = d * sc;
        v = __fmaf_rn(pxc, A.cs[c + 1], v);
        v = __fmaf_rn(pxl, A.cs[c - 1], v);
        v = __fmaf_rn(pyc, A.cs[c + W], v);
        return __fmaf_rn(pyd, A.cs[c - W], v);
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
    float d = 0.0f, pxc = 0.0f, pxl = 0.0f, pyc = 0.0f, pyd = 0.0f;  // K == 1
    float rv[KR], x[KR], av[KR];
#pragma unroll
    for (int k = 0; k < KR; ++k) rv[k] = x[k] = av[k] = 0.0f;
    // r.r first: where it is below the exit, as in many V-cycles of a relative
    // solve, nothing else is needed.  The directions are zero outside the
    // fluid and in the padding.
    CgTerms g;
    bool more = false;
    // a double-float add errs by at most 5 * 2^-48 of its operands' magnitudes;
    // a thread adds its cells, the two trees add ten times
    const float eps = float((K > 0 ? uint32_t(K) : cells / threads) + 16u) * 0x1p-45f;
    // (cells in registers put their terms into cap, which only the exact sums use)
    auto rr64 = [&]() {
        if constexpr (K == 0) return cg_sum64(A.cr + W, A.cr + W, A.bits, cells, sh.wide, nwarps);
#pragma unroll
        for (int k = 0; k < K; ++k) {
            const uint32_t r = threadIdx.x + uint32_t(k) * threads;
            if (r < cells) A.cap[r] = rv[k] * rv[k];
        }
        return cg_sum64(A.cap, nullptr, A.bits, cells, sh.wide, nwarps);
    };
    if (exact && K > 0) cg_bar(nwarps);  // sh.pre
    for (uint32_t c = threadIdx.x; c < 2u * W; c += threads) A.cs[c < W ? c : cells + c] = 0.0f;
    if constexpr (K > 0) {
#pragma unroll
        for (int k = 0; k < K; ++k) {
            const uint32_t r = threadIdx.x + uint32_t(k) * threads;
            if (r >= cells) continue;
            rv[k] = bit_at(A.bits, r) ? A.res[r + W] : 0.0f;
            A.cs[r + W] = rv[k];
            const float q = rv[k] * rv[k];
            if (exact) stage(r, q);
            if constexpr (K == 1) g.template set<false>(q);
            else g.template add<false>(q);
        }
    } else {
        for (uint32_t r = threadIdx.x; r < cells; r += threads) {
            const uint32_t c = r + W;
            const float q = bit_at(A.bits, r) ? A.res[c] : 0.0f;
            A.err[c] = 0.0f;
            A.cr[c] = q;
            A.cs[c] = q;
            g.template add<false>(q * q);
        }
    }
    float gamma;
    if (exact)
        gamma = K > 0 ? serial() : serial_cells(A.cr, A.cr);
    else
        gamma = cg_reduce<false, false>(g, more, sh.slot[0], nwarps, eps, exact, rr64);
    uint32_t max_it = 0;
    if (!(gamma < 1e-12f)) {
        if (!exact) count();
        max_it = min(nfl, 100u);
        if (K == 1 && threadIdx.x < cells) {
            const uint32_t c = threadIdx.x + W;
            d = A.diag[c];
            pxc = A.px[c];
            pxl = A.px[c - 1];
            pyc = A.py[c];
            pyd = A.py[c - W];
        }
    }
    for (uint32_t it = 0; it < max_it; ++it) {
        // (the directions are visible: a barrier follows their update)
        CgTerms dsum;
        if constexpr (K == 1) {
            float q = 0.0f;
            if (threadIdx.x < cells) {
                const uint32_t c = threadIdx.x + W;
                const float sc = A.cs[c];
                av[0] = apply(c, d, sc, pxc, pxl, pyc, pyd);
                q = sc * av[0];
                if (exact) stage(threadIdx.x, q);
            }
            dsum.template set<true>(q);
        } else if constexpr (K > 1) {
#pragma unroll
            for (int k = 0; k < K; ++k) {
                const uint32_t r = threadIdx.x + uint32_t(k) * threads;
                if (r >= cells) continue;
                const uint32_t c = r + W;
                const float sc = A.cs[c];
                const float v = apply(c, A.diag[c], sc, A.px[c], A.px[c - 1], A.py[c], A.py[c - W]);
                av[k] = v;
                const float q = sc * v;
                if (exact) stage(r, q);
                dsum.template add<true>(q);
            }
        } else {
            for (uint32_t r = threadIdx.x; r < cells; r += threads) {
                if (!bit_at(A.bits, r)) continue;
                const uint32_t c = r + W;
                const float sc = A.cs[c];
                const float v = apply(c, A.diag[c], sc, A.px[c], A.px[c - 1], A.py[c], A.py[c - W]);
                A.cap[c] = v;
                dsum.template add<true>(sc * v);
            }
        }
        float delta;
        if (exact)
            delta = K > 0 ? serial() : serial_cells(A.cs, A.cap);
        else
            delta = cg_reduce<false, true>(dsum, more, sh.slot[1], nwarps, eps, false, [&]() {
                if constexpr (K == 0) return cg_sum64(A.cs + W, A.cap + W, A.bits, cells, sh.wide, nwarps);
#pragma unroll
                for (int k = 0; k < K; ++k) {
                    const uint32_t r = threadIdx.x + uint32_t(k) * threads;
                    if (r < cells) A.cap[r] = A.cs[r + W] * av[k];
                }
                return cg_sum64(A.cap, nullptr, A.bits, cells, sh.wide, nwarps);
            });
        if (fabsf(delta) < 1e-5f) break;
        const float alpha = gamma / delta;
        more = false;  // some |r| is not below the exit (max|r| < 1e-6)
        CgTerms ng;
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
                if constexpr (K == 1) ng.template set<false>(q);
                else ng.template add<false>(q);
            }
        } else {
            for (uint32_t r = threadIdx.x; r < cells; r += threads) {
                if (!bit_at(A.bits, r)) continue;
                const uint32_t c = r + W;
                A.err[c] = A.err[c] + alpha * A.cs[c];
                const float nr = A.cr[c] - alpha * A.cap[c];
                A.cr[c] = nr;
                more = more || fabsf(nr) >= 1e-6f;
                ng.template add<false>(nr * nr);
            }
        }
        // the exit's test and the next r.r in one reduction (the latter is
        // dropped when the former ends the loop)
        float new_gamma = cg_reduce<true, false>(ng, more, sh.slot[0], nwarps, eps, exact, rr64);
        if (!more) break;
        if (exact) new_gamma = K > 0 ? serial() : serial_cells(A.cr, A.cr);
        const float beta = new_gamma / gamma;
        gamma = new_gamma;
        if constexpr (K > 0) {
#pragma unroll
            for (int k = 0; k < K; ++k) {
                const uint32_t r = threadIdx.x + uint32_t(k) * threads;
                if (r >= cells) continue;
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
        if (!exact) {
            double t = double(q);
            if (cells > 16u) t += __shfl_xor_sync(0xffffffffu, t, 16);  // (else the upper lanes hold zeros)
#pragma unroll
            for (int o = 8; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
            return __shfl_sync(0xffffffffu, float(t), 0);
        }
        float t = 0.0f;
        for (uint32_t l0 = 0; l0 < cells; l0 += 8) {  // (lanes beyond the level hold zeros)
#pragma unroll
            for (uint32_t l = 0; l < 8; ++l) t = t + __shfl_sync(0xffffffffu, q, int(l0 + l));
        }
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

// A level of up to 32 cells takes one warp, up to 1024 one cell per thread of
// as many warps as that needs; above, all threads hold 4, 6 or 10 cells each;
// beyond 10240 cells they stay in memory.
static __device__ __forceinline__ void cta_coarse_cg(const CgArrays& A, bool exact) {
    __shared__ CgShared sh;
    const uint32_t need = (A.cells + 31u) >> 5, all = blockDim.x >> 5;
    const uint32_t nwarps = need < all ? need : all;
    if ((threadIdx.x >> 5) < nwarps) {
        if (need <= 1u)
            cg_one_warp(A, exact);
        else if (need <= all)
            cg_warps<1>(A, sh, nwarps, exact);
        else if (need <= 4u * all)
            cg_warps<4>(A, sh, nwarps, exact);
        else if (need <= 6u * all)
            cg_warps<6>(A, sh, nwarps, exact);
        else if (need <= kCgMaxK * all)
            cg_warps<int(kCgMaxK)>(A, sh, nwarps, exact);
        else
            cg_warps<0>(A, sh, nwarps, exact);
    }
    __syncthreads();
}

// ---- the coarse tail in shared memory ----------------------------------------
struct TailLevel {
    const uint32_t* fluid;
    const float *diag, *inv, *px, *py;
    float* res;   // global residual (read for the first tail level)
    float* err;   // global error (written back for the first tail level)
};
struct TailParams {
    int n;                      // tail levels; lv[n - 1] is the coarsest
    int exact;                  // coarsest CG with the reference's serial FP32 sums
    uint32_t w, h;              // of the first level
    int wshift;                 // log2 w, or -1 when w is not a power of two
    TailLevel lv[kMaxLevels];
};

// One level in the tail's shared memory (32-bit words): mask words, then
// diagonal, inverse diagonal, couplings, residual and error, each `padded`
// long.  A level follows from the one before it by arithmetic alone (sides
// halve, offsets add up): a load of its sizes and offsets from the kernel's
// parameters missed the constant cache at each phase (0.25 us of 0.4).
struct SmemLevel {
    uint32_t w, h, cells, words, padded;
    int wshift;
    uint32_t* bits;
    float *diag, *inv, *px, *py, *res, *err;
};
inline __host__ __device__ uint32_t tail_words(uint32_t cells) { return (cells + 63u) / 64u * 2u; }
inline __host__ __device__ uint32_t tail_padded(uint32_t w, uint32_t cells) { return (cells + 2u * w + 7u) & ~7u; }
__device__ __forceinline__ SmemLevel smem_at(uint32_t* at, uint32_t w, uint32_t h, int wshift) {
    SmemLevel L;
    L.w = w;
    L.h = h;
    L.cells = w * h;
    L.words = tail_words(L.cells);
    L.padded = tail_padded(w, L.cells);
    L.wshift = wshift;
    L.bits = at;
    L.diag = reinterpret_cast<float*>(at + L.words);
    L.inv = L.diag + L.padded;
    L.px = L.inv + L.padded;
    L.py = L.px + L.padded;
    L.res = L.py + L.padded;
    L.err = L.res + L.padded;
    return L;
}
__device__ __forceinline__ SmemLevel smem_first(const TailParams& tp, uint32_t* sm) {
    return smem_at(sm, tp.w, tp.h, tp.wshift);
}
__device__ __forceinline__ SmemLevel smem_coarser(const SmemLevel& f) {
    return smem_at(f.bits + f.words + 6u * f.padded, f.w >> 1, f.h >> 1, f.wshift > 0 ? f.wshift - 1 : -1);
}
__device__ __forceinline__ SmemLevel smem_finer(const SmemLevel& c) {
    const uint32_t w = c.w << 1, h = c.h << 1;
    return smem_at(c.bits - tail_words(w * h) - 6u * tail_padded(w, w * h), w, h, c.wshift >= 0 ? c.wshift + 1 : -1);
}

// ---- phases on levels in shared memory ---------------------------------------
// The coarse levels' coefficients are zero at every cell outside the fluid
// (the multigrid setup writes them so), so on a level held by a CTA (the
// tail, below) or by a cluster in bands of rows (vcycle_dsm.cu) a phase runs
// over all cells without a test.  A neighbour that the reference skips enters
// with a zero coupling, which leaves a sum as it was; a cell whose inverse
// diagonal is zero keeps its old value, as in the reference.  A level takes
// four phases a V-cycle: black sweep (the red one is formed with the residual,
// red_first), restriction; prolongation fused into the black and into the red
// reverse sweep.  What bounds a phase is its instructions (32 warps on four
// schedulers) and then its barrier, so index arithmetic and tests went first.

// The first red sweep of a cell from zero error (its own residual is all it takes).
__device__ __forceinline__ float red_first(float r, float inv) {
    return inv != 0.0f ? 0.0f + (kOmega * (r * inv - 0.0f)) : 0.0f;
}
// One SOR update; er, eu, el, ed: the neighbours' errors in the reference's order.
__device__ __forceinline__ float sor_masked(float inv, float sum, float pxc, float pyc, float pxl, float pyd, float er,
                                            float eu, float el, float ed, float old) {
    sum = __fmaf_rn(-pxc, er, sum);
    sum = __fmaf_rn(-pyc, eu, sum);
    sum = __fmaf_rn(-pxl, el, sum);
    sum = __fmaf_rn(-pyd, ed, sum);
    const float gs = sum * inv;
    const float nv = old + (kOmega * (gs - old));
    return inv == 0.0f ? old : nv;
}
// b - A e (restrict :549-583) of the cells at indexes i (even) and i + 1 of
// arrays with rows of w (even; 8-byte aligned): pairs are read whole, which
// halves the reads and their bank conflicts.
__device__ __forceinline__ float2 left_over(const float* r, const float* d, const float* px, const float* py,
                                            const float* e, int i, int w) {
    auto two = [](const float* p) { return *reinterpret_cast<const float2*>(p); };
    const float2 ec = two(e + i), eu = two(e + i + w), ed = two(e + i - w), dc = two(d + i), rc = two(r + i);
    const float2 pxc = two(px + i), pyc = two(py + i), pyd = two(py + i - w);
    const float el = e[i - 1], er = e[i + 2], pxl = px[i - 1];
    float a0 = dc.x * ec.x, a1 = dc.y * ec.y;
    a0 = a0 + pxc.x * ec.y;
    a1 = a1 + pxc.y * er;
    a0 = a0 + pyc.x * eu.x;
    a1 = a1 + pyc.y * eu.y;
    a0 = a0 + pxl * el;
    a1 = a1 + pxc.x * ec.x;
    a0 = a0 + pyd.x * ed.x;
    a1 = a1 + pyd.y * ed.y;
    return make_float2(rc.x - a0, rc.y - a1);
}
// The errors around a cell under prolongation: its coarse cell's error c0,
// that of the coarse cell beside it in x and in y (the other two neighbours
// lie under c0).
struct CoarseAround {
    float c0, h, v;
};
__device__ __forceinline__ CoarseAround coarse_around(const float* ce, int cc, int cw, bool x_odd, bool y_odd) {
    return CoarseAround{ce[cc], ce[cc + (x_odd ? 1 : -1)], ce[cc + (y_odd ? cw : -cw)]};
}

// k-th cell of one colour of a level with rows of w = 2 * half: its row and column.
__device__ __forceinline__ void colour_cell(uint32_t k, uint32_t half, int hshift, uint32_t color, uint32_t& x,
                                            uint32_t& y) {
    uint32_t kk;
    raw_xy(k, half, hshift, kk, y);
    x = 2u * kk + ((y + color) & 1u);
}

// The tail's phases (padded layout; w even on every level that is swept).
__device__ __forceinline__ void cta_black(const SmemLevel& L) {
    const uint32_t half = L.w >> 1;
    const int hs = L.wshift > 0 ? L.wshift - 1 : -1, w = int(L.w);
    for (uint32_t k = threadIdx.x; k < L.h * half; k += blockDim.x) {
        uint32_t x, y;
        colour_cell(k, half, hs, 1u, x, y);
        const int c = int((y + 1u) * L.w + x);
        L.err[c] = sor_masked(L.inv[c], L.res[c], L.px[c], L.py[c], L.px[c - 1], L.py[c - w], L.err[c + 1],
                              L.err[c + w], L.err[c - 1], L.err[c - w], 0.0f);
    }
    __syncthreads();
}
// Two threads per coarse cell, one per row of its children; the even one adds
// the four in the reference's order.
__device__ __forceinline__ void cta_restrict(const SmemLevel& f, const SmemLevel& c) {
    const uint32_t n = (2u * c.cells + 31u) & ~31u;  // whole warps take part in the shuffles
    const int w = int(f.w);
    for (uint32_t i = threadIdx.x; i < n; i += blockDim.x) {
        const uint32_t q = i >> 1, dy = i & 1u;
        float d0 = 0.0f, d1 = 0.0f;
        uint32_t cx = 0, cy = 0;
        if (q < c.cells) {
            raw_xy(q, c.w, c.wshift, cx, cy);
            const int p = int((2u * cy + dy + 1u) * f.w + 2u * cx);
            const float2 two = left_over(f.res, f.diag, f.px, f.py, f.err, p, w);
            d0 = two.x;
            d1 = two.y;
        }
        const float d2 = __shfl_down_sync(0xffffffffu, d0, 1), d3 = __shfl_down_sync(0xffffffffu, d1, 1);
        if (dy == 0 && q < c.cells) {
            const float sum = (((0.0f + d0) + d1) + d2) + d3;
            const uint32_t p = q + c.w;
            c.res[p] = sum;
            c.err[p] = ((cx + cy) & 1u) == 0u ? red_first(sum, c.inv[p]) : 0.0f;
        }
    }
    __syncthreads();
}
template <int kColor>
__device__ __forceinline__ void cta_up(const SmemLevel& f, const SmemLevel& c) {
    const uint32_t half = f.w >> 1;
    const int hs = f.wshift > 0 ? f.wshift - 1 : -1, w = int(f.w);
    for (uint32_t k = threadIdx.x; k < f.h * half; k += blockDim.x) {
        uint32_t x, y;
        colour_cell(k, half, hs, kColor, x, y);
        const int p = int((y + 1u) * f.w + x), cc = int(((y >> 1) + 1u) * c.w + (x >> 1));
        const bool xo = x & 1u, yo = y & 1u;
        float er = f.err[p + 1], eu = f.err[p + w], el = f.err[p - 1], ed = f.err[p - w], old = f.err[p];
        if (kColor == 1) {
            const CoarseAround a = coarse_around(c.err, cc, int(c.w), xo, yo);
            old = old + a.c0;
            er = er + (xo ? a.h : a.c0);
            el = el + (xo ? a.c0 : a.h);
            eu = eu + (yo ? a.v : a.c0);
            ed = ed + (yo ? a.c0 : a.v);
        } else {
            old = old + c.err[cc];
        }
        f.err[p] = sor_masked(f.inv[p], f.res[p], f.px[p], f.py[p], f.px[p - 1], f.py[p - w], er, eu, el, ed, old);
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
// (complete after cp_async_wait_all), and zero the vectors (their padding is
// read beside the level's edge).
__device__ __forceinline__ void cta_tail_issue_coeffs(const TailParams& tp, uint32_t* sm) {
    SmemLevel L = smem_first(tp, sm);
    for (int l = 0; l < tp.n; ++l) {
        const TailLevel& t = tp.lv[l];
        for (uint32_t i = threadIdx.x; i < L.words; i += blockDim.x) cp_async4(L.bits + i, t.fluid + i);
        for (uint32_t i = threadIdx.x; i < L.padded; i += blockDim.x) {
            cp_async4(L.diag + i, t.diag + i);
            cp_async4(L.inv + i, t.inv + i);
            cp_async4(L.px + i, t.px + i);
            cp_async4(L.py + i, t.py + i);
            L.err[i] = 0.0f;
            if (l > 0) L.res[i] = 0.0f;
        }
        L = smem_coarser(L);
    }
}

// The V-cycle on the tail's levels by one CTA: the first level's residual and
// first red sweep are in shared memory, its final error stays there.
__device__ __forceinline__ void cta_tail_levels(const TailParams& tp, uint32_t* sm) {
    const int n = tp.n;
    SmemLevel f = smem_first(tp, sm);
    for (int l = 0; l + 1 < n; ++l) {
        const SmemLevel c = smem_coarser(f);
        cta_black(f);
        cta_restrict(f, c);
        f = c;
    }
    float* cg = reinterpret_cast<float*>(f.bits + f.words + 6u * f.padded);  // three vectors behind the last level
    cta_coarse_cg(CgArrays{f.bits, f.w, f.cells, f.diag, f.px, f.py, f.res, f.err, cg, cg + f.padded,
                           cg + 2u * f.padded},
                  tp.exact != 0);
    for (int l = n - 2; l >= 0; --l) {
        const SmemLevel c = f;
        f = smem_finer(c);
        cta_up<1>(f, c);
        cta_up<0>(f, c);
    }
}

// The coarse tail by one CTA, from the first level's residual in global
// memory to its error there.  The coefficients' copies were issued before
// (cta_tail_issue_coeffs).
__device__ __forceinline__ void cta_tail(const TailParams& tp, uint32_t* sm) {
    const SmemLevel L = smem_first(tp, sm);
    const float* res = tp.lv[0].res;
    float* err = tp.lv[0].err;
    for (uint32_t i = threadIdx.x; i < L.padded; i += blockDim.x) cp_async4(L.res + i, res + i);
    cp_async_wait_all();
    __syncthreads();
    // (only the fluid cells' residual was written)
    for (uint32_t i = threadIdx.x; i < L.padded; i += blockDim.x) {
        const long long r = (long long)i - L.w;
        if (!fluid_raw(L.bits, r, L.cells)) L.res[i] = 0.0f;
        else if (red_at(uint32_t(r), L.w, L.wshift)) L.err[i] = red_first(L.res[i], L.inv[i]);
    }
    __syncthreads();
    cta_tail_levels(tp, sm);
    for (uint32_t r = threadIdx.x; r < L.cells; r += blockDim.x)
        if (bit_at(L.bits, r)) err[r + L.w] = L.err[r + L.w];
}

// Host: tail parameters for levels [first, s.nlevels), and the 32-bit words
// they take in shared memory (the CG's three vectors last).
inline TailParams make_tail_params(const Scene& s, int first, uint32_t* words_out) {
    TailParams tp;
    std::memset(&tp, 0, sizeof(tp));
    tp.n = s.nlevels - first;
    tp.exact = coarse_cg_exact(s) ? 1 : 0;
    uint32_t off = 0;
    for (int k = 0; k < tp.n; ++k) {
        const Level& v = s.lv[first + k];
        if (k == 0) {
            tp.w = v.w;
            tp.h = v.h;
            tp.wshift = v.wshift;
        }
        tp.lv[k] = TailLevel{v.fluid, v.diag, v.inv_diag, v.px, v.py, v.res, v.err};
        off += tail_words(v.cells) + 6 * tail_padded(v.w, v.cells);
    }
    const Level& last = s.lv[s.nlevels - 1];
    off += 3 * tail_padded(last.w, last.cells);
    *words_out = off;
    return tp;
}

}  // namespace vc
}  // namespace apic
