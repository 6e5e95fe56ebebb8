// solver.cu — multigrid-preconditioned CG pressure solve.
//
// Restates Apic::solve_pcg (src/apic.rs:1865-1956) with its preconditioner
// apply_preconditioner (:1788-1821): one V-cycle of red/black SOR (omega 1.2,
// one pre- and one post-sweep, MultiGridLevel::smooth_level :471-535),
// residual restriction over 2x2 children (:537-594), piecewise-constant
// prolongation (:596-616; on the base level the last fluid cell receives the
// correction once more per duplicate that pads the reference's list to a
// multiple of 8, :1487-1494) and plain CG on the coarsest level
// (solve_coarse_exact :618-704, one CTA here).
//
// The kernels walk the level's segment list or its list of fluid tiles, whose
// lengths live in device memory, and return at once when the device-side
// `pcg_done` flag is set, so an iteration costs no host round trip.  Dot
// products sum FP32 products in double-float (FP64 in the refinement) and are
// reduced deterministically: per-block partials, summed in block order by the
// kernel that needs the total.  The reference's alpha/beta/gamma are FP32 and
// so are they here: the sums are rounded to float before the reference's FP32
// divisions.
//
// Solver modes: APIC_SOLVER_REFERENCE keeps the reference's exits (max|r| <
// solve_error, gamma/delta < 1e-5, 100 iterations).  APIC_SOLVER_REL_FP32
// iterates to ||r||_2 <= tol*||b||_2.  APIC_SOLVER_REL_MIXED wraps FP32 inner
// solves in FP64 iterative refinement on the true residual b - A p.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>

#include "apic_device.cuh"
#include "apic_graph.h"
#include "apic_internal.h"
#include "batch.h"
#include "pcg_common.cuh"
#include "tiles.cuh"

namespace apic {
namespace {

constexpr float kSafety = 1e-5f;  // SAFTY, src/apic.rs:8
constexpr uint32_t kDeltaChunk = 8192;  // apply_matrix_and_dot's par_chunks(8192), src/apic.rs:1857-1859

__device__ __forceinline__ uint32_t gwarp() { return (blockIdx.x * blockDim.x + threadIdx.x) >> 5; }
__device__ __forceinline__ uint32_t gnwarps() { return (gridDim.x * blockDim.x) >> 5; }

// A PCG solve's starting state.
__device__ __forceinline__ void pcg_reset(Ctl* ctl) {
    ctl->pcg_done = 0;
    ctl->pcg_iters = 0;
    ctl->gamma = 0.0f;
    ctl->alpha = 0.0f;
    ctl->beta = 0.0f;
    ctl->beta_valid = 0;
    ctl->delta_stop = 0;
    ctl->rnorm2 = 0.0;
    ctl->res_sel = 0;  // a solve's right-hand side is in the first buffer
}

__global__ void k_pcg_begin(Ctl* ctl) {
    pdl_wait();
    pcg_reset(ctl);
}

// ---- PCG kernels on the base level (phases in pcg_common.cuh) --------------

// Each kernel's work is a body taking the block's coordinates in its scene's
// grid (bk), run by the single-scene kernel with the hardware's and by the
// batch kernel (one launch over many scenes, batch.h) with the scene's.

// Entry of the PCG loop: go on while not converged and under the iteration
// cap (src/apic.rs:1894-1899); dyn_cap reads the remaining budget of a
// refinement.  Inside the loop the same decision is taken by the kernel that
// runs the residual's exit test (pcg::loop_decision) or, in the reference
// mode, by k_gamma_exact.
__device__ __forceinline__ bool pcg_entry(const Ctl* ctl, uint32_t cap, int dyn_cap) {
    const uint32_t c = dyn_cap ? ctl->inner_cap : cap;
    return !ctl->pcg_done && ctl->pcg_iters < c;
}

// The loop that a kernel which ends a solve's setup opens (set 0: none).
struct LoopEntry {
    cudaGraphConditionalHandle h = 0;
    uint32_t cap = 0;
    int dyn_cap = 0;
    int set = 0;
};

// s = z and gamma = r.z (src/apic.rs:1887-1892).
// In the reference mode k_gamma_exact forms gamma and the exit instead.
// True in the one thread that formed gamma.
__device__ __forceinline__ bool kb_pcg_start(Blk bk, const Level& B, float* s, Ctl* ctl, double* partials, int mode) {
    F2 acc = pcg::ph_start(B, ctl->seg_count[0], blk_warp(bk), blk_nwarps(bk), s);
    if (mode == APIC_SOLVER_REFERENCE) return false;
    double tot;
    if (block_sum_last<kSegBlock>(bk, acc, partials, &ctl->red_counter, &tot) && threadIdx.x == 0) {
        float gamma = float(tot);
        ctl->gamma = gamma;
        ctl->dgamma = tot;
        if (!(gamma != 0.0f)) ctl->pcg_done = 1;
        return true;
    }
    return false;
}
__global__ void __launch_bounds__(kSegBlock) k_pcg_start(Level B, float* s, Ctl* ctl, double* partials, int mode,
                                                         LoopEntry loop) {
    pdl_wait();
    if (kb_pcg_start(hw_blk(), B, s, ctl, partials, mode) && loop.set)
        cudaGraphSetConditional(loop.h, pcg_entry(ctl, loop.cap, loop.dyn_cap) ? 1u : 0u);
}

// The relative modes' s' = z + beta s, Ap = A s' and this block's part of delta =
// s'.Ap (apply_matrix_and_dot, src/apic.rs:1823-1863; the search update
// :1945-1954 is folded in).  The update sums the parts.  The previous
// iteration's r.z arrives as the parts its V-cycle stored (rz): every block
// sums them into gamma' and forms beta = gamma' / gamma (:1934-1943); a zero
// r.z ends the solve (the update records it).  Block 0 keeps beta for the
// update.
// (after the dependency wait; w0: this warp's first segment word)
// rz_sum: the parts' sum formed once beforehand (batched solves), else null.
__device__ __forceinline__ void kb_spmv_dot(Blk bk, const Level& B, uint32_t nseg, uint32_t w0, const float* s,
                                            float* ap, Ctl* ctl, float2* part, const float2* rz,
                                            uint32_t nrz, const float* rz_sum = nullptr) {
    const bool done = ctl->pcg_done != 0, bv = ctl->beta_valid != 0;
    float beta = ctl->beta;
    const float gamma = ctl->gamma;
    const float ng = rz_sum ? *rz_sum : sum_partials<kSegBlock>(rz, nrz);
    if (done) return;
    if (bv) {
        if (!(ng != 0.0f)) return;
        beta = ng / gamma;
        if (bk.id == 0 && threadIdx.x == 0) ctl->beta = beta;
    }
    // the buffer this iteration's update writes the residual to (read by the
    // kernels after this one)
    if (bk.id == 0 && threadIdx.x == 0) ctl->res_sel = (ctl->pcg_iters + 1u) & 1u;
    const F2 acc = spmv_segs(B) == 4u ? pcg::ph_spmv_search4(B, nseg, blk_warp(bk), blk_nwarps(bk), s, beta, bv, ap, w0)
                                      : pcg::ph_spmv_search(B, nseg, blk_warp(bk), blk_nwarps(bk), s, beta, bv, ap, w0);
    block_store<kSegBlock>(bk, acc, part);
}
// first: of its loop body (counted).
__global__ void __launch_bounds__(kSegBlock, 5) k_spmv_dot(Level B, const float* s, float* ap, Ctl* ctl, float2* part,
                                                        const float2* rz, uint32_t nrz, int first) {
    // the base segment list is written by the substep's setup: load this
    // warp's first word before waiting on the previous kernel
    const uint32_t nseg = ctl->seg_count[0];
    const uint32_t s0 = spmv_segs(B) == 4u ? 4u * gwarp() + ((threadIdx.x & 31u) >> 3) : gwarp();
    const uint32_t w0 = s0 < nseg ? B.seg[s0] : 0xFFFFFFFFu;
    pdl_wait();
    if (first && blockIdx.x == 0 && threadIdx.x == 0) ctl->pcg_bodies++;
    kb_spmv_dot(hw_blk(), B, nseg, w0, s, ap, ctl, part, rz, nrz);
}

// delta (the sum of k_spmv_dot's parts, formed by every block) gives alpha or
// the exit (src/apic.rs:1899-1906, applied by the next kernel).  False: the
// block has nothing to do.
// rz_sum, sap_sum: the parts' sums formed once beforehand (batched solves).
struct StepArgs {
    const float2* sap;
    uint32_t nsap;
    int mode;
    const float* exact_parts;
    const uint32_t* seg_pre;
    const float2* rz;
    uint32_t nrz;
};
__device__ __forceinline__ bool pcg_alpha(Blk bk, Ctl* ctl, const StepArgs& a, float* alpha_out,
                                          const float* rz_sum = nullptr, const float* sap_sum = nullptr) {
    const bool done = ctl->pcg_done != 0, bv = ctl->beta_valid != 0;
    // this iteration's gamma: from the solve's start, or (relative modes) the
    // previous iteration's r.z parts, which k_spmv_dot summed the same way
    float gamma = ctl->gamma, delta;
    if (a.mode == APIC_SOLVER_REFERENCE) {
        if (done) return false;
        // the chunk sums of k_delta_exact, added in chunk order from zero
        const uint32_t nchunks = (a.seg_pre[ctl->seg_count[0]] + kDeltaChunk - 1) / kDeltaChunk;
        delta = 0.0f;
        for (uint32_t c = 0; c < nchunks; ++c) delta = delta + a.exact_parts[c];
    } else {
        const float2 sums =
            rz_sum ? make_float2(*rz_sum, *sap_sum) : sum_partials<kSegBlock>(a.rz, a.nrz, a.sap, a.nsap);
        if (done) return false;
        delta = sums.y;
        if (bv) {
            gamma = sums.x;
            if (!(gamma != 0.0f)) {
                if (bk.id == 0 && threadIdx.x == 0) ctl->pcg_done = 1;
                return false;
            }
        }
    }
    const bool stop = a.mode == APIC_SOLVER_REFERENCE ? fabsf(delta) < kSafety : (!(delta != 0.0f) || !isfinite(delta));
    const float alpha = gamma / delta;
    // every block reads pcg_done on entry, so the stop is recorded aside and
    // the next kernel turns it into pcg_done
    if (bk.id == 0 && threadIdx.x == 0) {
        ctl->gamma = gamma;
        ctl->pcg_iters++;
        ctl->delta_stop = stop ? 1u : 0u;
        if (!stop) ctl->alpha = alpha;
    }
    *alpha_out = alpha;
    return !stop;
}

// The update (p += alpha s', r = fma(-alpha, Ap, r), s = s', :1907-1932) in
// the base level's down kernel (tiles.cuh), and this block's part of ||r||^2
// and max|r|, whose exit test runs in the next kernel.  Block b takes the
// tiles b, b + n, ...  A tile's constants are read before the wait for the
// previous kernel and its vectors before alpha is formed from the parts.
// sel: the buffer the residual goes to (Ctl::res_sel, which alternates), or -1:
// read it.
__device__ __forceinline__ tile::Update update_args(const Level& B, const Ctl* ctl, float* p, int p_padded, float* s,
                                                    const float* ap, int sel) {
    const bool second = sel >= 0 ? sel != 0 : ctl->res_sel != 0;
    return tile::Update{second ? B.res : B.res2, ap, B.err, s, p, p_padded, second ? B.res2 : B.res};
}
// (after the dependency wait; g: the first tile's constants, if the block has one)
template <bool kAll>
__device__ __forceinline__ void kb_update_down(Blk bk, const Level& B, const Level& C, tile::Shared& sh,
                                               tile::DownRegs& g, uint32_t count, uint32_t id, float* p, int p_padded,
                                               float* s, const float* ap, Ctl* ctl, const StepArgs& a, float4* part,
                                               int sel, const float* rz_sum = nullptr,
                                               const float* sap_sum = nullptr) {
    const float beta = ctl->beta;
    const bool beta_valid = ctl->beta_valid != 0;
    const tile::Update u = update_args(B, ctl, p, p_padded, s, ap, sel);
    if (bk.id < count) tile::down_load<true, kAll>(B, u.res, u, g);
    float alpha;
    if (!pcg_alpha(bk, ctl, a, &alpha, rz_sum, sap_sum)) return;
    float mx = 0.0f;
    F2 acc{0.0f, 0.0f};
    for (uint32_t i = bk.id; i < count; i += bk.n) {
        if (i != bk.id) {
            id = B.tiles[i];
            __syncthreads();  // the tile before this one has been read
            tile::down_load_const<kAll>(B, id, g);
            tile::down_load<true, kAll>(B, u.res, u, g);
        }
        tile::down_tile<true>(sh, B, C, id, g, u, alpha, beta, beta_valid, &acc, &mx);
    }
    block_store<kSegBlock>(bk, acc, mx, part);
}
template <bool kAll>
__global__ void __launch_bounds__(kTileBlock, 4) k_update_down(Level B, Level C, float* p, int p_padded, float* s,
                                                                 const float* ap, Ctl* ctl, StepArgs a, float4* part,
                                                                 int sel) {
    __shared__ tile::Shared sh;
    const uint32_t count = ctl->tile_count[0];
    const uint32_t id = blockIdx.x < count ? B.tiles[blockIdx.x] : 0u;
    tile::DownRegs g;
    if (blockIdx.x < count) tile::down_load_const<kAll>(B, id, g);
    pdl_wait();
    kb_update_down<kAll>(hw_blk(), B, C, sh, g, count, id, p, p_padded, s, ap, ctl, a, part, sel);
}

// The update alone, and the base level's first red sweep (grids without a
// coarser level).
__global__ void __launch_bounds__(kSegBlock) k_pcg_update(Level B, float* p, int p_padded, float* s,
                                                          const float* ap, Ctl* ctl, StepArgs a, float4* part) {
    pdl_wait();
    float alpha;
    if (!pcg_alpha(hw_blk(), ctl, a, &alpha)) return;
    float mx;
    F2 acc;
    pcg::ph_update_search(B, ctl->seg_count[0], gwarp(), gnwarps(), alpha, ctl->beta, ctl->beta_valid != 0, p,
                          p_padded, s, ap, &mx, &acc);
    block_store<kSegBlock>(hw_blk(), acc, mx, part);
}

// Stand-alone exit test (grids without a coarser level).
__global__ void __launch_bounds__(kSegBlock) k_residual_exit(Ctl* ctl, ExitArgs a) {
    pdl_wait();
    if (!ctl->pcg_done) pcg::residual_exit(ctl, a.part, a.nparts, a.mode, a.solve_error);
    if (threadIdx.x == 0) pcg::loop_decision(ctl, a.mode, a.h, a.cap, a.dyn_cap, a.set_cond);
}

// This block's part of gamma' = r.z (src/apic.rs:1934-1943); the next
// iteration's k_spmv_dot and k_pcg_update sum the parts.
__global__ void __launch_bounds__(kSegBlock) k_dot_rz(Level B, Ctl* ctl, float2* part) {
    pdl_wait();
    if (ctl->pcg_done) return;
    F2 acc = pcg::ph_rz(B, ctl->seg_count[0], gwarp(), gnwarps());
    block_store<kSegBlock>(hw_blk(), acc, part);
}

// ---- the reference's FP32 reduction orders (APIC_SOLVER_REFERENCE) --------
//
// Float addition is not associative, so the reference mode forms its two
// Krylov reductions in exactly the reference's order; the solve is then
// bit-identical to the oracle's.

// acc + v[0].x + v[0].y + ... + v[n - 1].w, one addition after another, with
// the loads kAhead vectors ahead of the add chain.
template <uint32_t kAhead>
__device__ __forceinline__ float add_in_order(const float4* v, uint32_t n, float acc) {
    float4 a[kAhead];
#pragma unroll
    for (uint32_t k = 0; k < kAhead; ++k) a[k] = k < n ? v[k] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    uint32_t i = 0;
    for (; i + kAhead <= n; i += kAhead) {
#pragma unroll
        for (uint32_t k = 0; k < kAhead; ++k) {
            const float4 q = a[k];
            a[k] = i + kAhead + k < n ? v[i + kAhead + k] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            acc = acc + q.x;
            acc = acc + q.y;
            acc = acc + q.z;
            acc = acc + q.w;
        }
    }
#pragma unroll
    for (uint32_t k = 0; k < kAhead; ++k) {
        if (i + k >= n) break;
        acc = acc + a[k].x;
        acc = acc + a[k].y;
        acc = acc + a[k].z;
        acc = acc + a[k].w;
    }
    return acc;
}

// gamma = dot_product(residual[W..W+cells], error[W..W+cells]) (:11-29): eight
// lane sums, lane = raw index mod 8, each added in ascending order; then
// wide's reduce_add pairing ((l0 + l2) + (l1 + l3)) + ((l4 + l6) + (l5 + l7));
// then the cells beyond the last full chunk of 8, serially.  The error is
// zero outside the fluid cells (apply_preconditioner zeroes it, :1790-1792,
// and only fluid cells are smoothed or prolonged), and adding a zero product
// leaves a lane sum unchanged (the sums start at +0 and never become -0), so
// only the fluid cells' products count.  One block: warps 1..31 stage the
// products of a batch of segments (32 raw cells each, zero where not fluid)
// in shared memory while threads 0..7 add the previous batch's products of
// their lane in order (two stage buffers); only those eight add chains are
// serial.  A lane's products of a segment (raw cells t, t + 8, t + 16, t + 24)
// lie side by side in its own row of the stage, so a thread takes a segment
// with one 16-byte load and has the next eight in flight: the four dependent
// adds are all that a segment costs (1024^2 grid, 514605 fluid cells: a solve
// of one such pass 402 -> 302 us).
// start: the solve's first gamma (sets gamma and the SAFTY exit,
// :1887-1892), else the iteration's new gamma.
constexpr int kGammaThreads = 1024;
constexpr uint32_t kGammaBatch = 512;               // segments staged per round
constexpr uint32_t kGammaRow = 4 * kGammaBatch + 4;  // a lane's row (the rows start four banks apart)
constexpr uint32_t kGammaAhead = 8;                 // segments loaded ahead of the adds
constexpr size_t kGammaSmem = 2 * 8 * size_t(kGammaRow) * sizeof(float);
// The iteration's form (start 0) also finishes the iteration (beta, or the
// SAFTY exit) and, when set_cond, sets the loop condition.
__global__ void __launch_bounds__(kGammaThreads) k_gamma_exact(Level B, Ctl* ctl, int start,
                                                               cudaGraphConditionalHandle h, uint32_t cap,
                                                               int dyn_cap, int set_cond) {
    extern __shared__ __align__(16) float stage[];  // two buffers of eight rows
    pdl_wait();
    if (ctl->pcg_done) return;
    const uint32_t t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const uint32_t nseg = ctl->seg_count[0];
    const float* __restrict__ res = pcg::cur_res(B, ctl);
    const uint32_t full = (B.cells / 8u) * 8u;
    const uint32_t nbatch = (nseg + kGammaBatch - 1) / kGammaBatch;
    // warps 1..31 stage batch b into buffer b % 2
    auto fill = [&](uint32_t b) {
        float* buf = stage + (b & 1u) * 8u * kGammaRow + (lane & 7u) * kGammaRow + (lane >> 3);
        const uint32_t k0 = b * kGammaBatch, nb = min(kGammaBatch, nseg - k0);
#pragma unroll 4
        for (uint32_t q = warp - 1; q < nb; q += kGammaThreads / 32 - 1) {
            const uint32_t w = B.seg[k0 + q];
            const uint32_t raw = w * 32u + lane;
            const bool on = ((B.fluid[w] >> lane) & 1u) && raw < full;
            buf[4u * q] = on ? res[raw + B.w] * B.err[raw + B.w] : 0.0f;
        }
    };
    float acc = 0.0f;
    if (warp != 0 && nbatch > 0) fill(0);
    __syncthreads();
    for (uint32_t b = 0; b < nbatch; ++b) {
        if (warp == 0) {
            if (t < 8) {
                const float4* row = reinterpret_cast<const float4*>(stage + (b & 1u) * 8u * kGammaRow + t * kGammaRow);
                const uint32_t nb = min(kGammaBatch, nseg - b * kGammaBatch);
                acc = add_in_order<kGammaAhead>(row, nb, acc);
            }
        } else if (b + 1 < nbatch) {
            fill(b + 1);
        }
        __syncthreads();
    }
    __shared__ float lanes[8];
    if (t < 8) lanes[t] = acc;
    __syncthreads();
    if (t != 0) return;
    float g = ((lanes[0] + lanes[2]) + (lanes[1] + lanes[3])) + ((lanes[4] + lanes[6]) + (lanes[5] + lanes[7]));
    for (uint32_t raw = full; raw < B.cells; ++raw)
        if (bit_at(B.fluid, raw)) g = g + res[raw + B.w] * B.err[raw + B.w];
    if (start) {
        ctl->gamma = g;
        ctl->dgamma = double(g);
        if (g < kSafety) ctl->pcg_done = 1;
        if (set_cond) cudaGraphSetConditional(h, pcg_entry(ctl, cap, dyn_cap) ? 1u : 0u);
    } else {
        pcg::finish_rz_reference(ctl, g);
        if (set_cond) {
            const uint32_t c = dyn_cap ? ctl->inner_cap : cap;
            const bool cont = !ctl->pcg_done && ctl->pcg_iters < c;
            if (!cont && !ctl->pcg_done) ctl->pcg_done = kStoppedAtCap;
            cudaGraphSetConditional(h, cont ? 1u : 0u);
        }
    }
}

// Fluid cells before each base segment (seg_pre[k], k <= nseg; seg_pre[nseg]
// = all fluid cells): the position of a segment's cells in the reference's
// ascending fluid list; and the segment that holds the first cell of each of
// the chunks of k_delta_exact (chunk_seg).  The reference mode's solve starts
// here: block 0 resets the PCG state and counts, four segments a thread and
// round; the others clear the pressure.
__global__ void __launch_bounds__(1024) k_reference_start(Level B, float* p, Ctl* ctl, uint32_t* seg_pre,
                                                          uint32_t* chunk_seg) {
    pdl_wait();
    const uint32_t nseg = ctl->seg_count[0];
    if (blockIdx.x != 0) {
        pcg::ph_clear_pressure(B, nseg, (blockIdx.x - 1u) * 32u + (threadIdx.x >> 5), (gridDim.x - 1u) * 32u, p);
        return;
    }
    if (threadIdx.x == 0) {
        ctl->solve_t0 = global_ns();
        pcg_reset(ctl);
    }
    __shared__ uint32_t sw[32];
    const uint32_t t = threadIdx.x, lane = t & 31, warp = t >> 5;
    uint32_t carry = 0;
    for (uint32_t k0 = 0; k0 < nseg; k0 += 4096) {
        const uint32_t k = k0 + 4u * t;
        uint32_t v[4], x = 0;
#pragma unroll
        for (uint32_t j = 0; j < 4; ++j) v[j] = k + j < nseg ? B.seg[k + j] : 0u;
#pragma unroll
        for (uint32_t j = 0; j < 4; ++j) {
            v[j] = k + j < nseg ? uint32_t(__popc(B.fluid[v[j]])) : 0u;
            x += v[j];
        }
        const uint32_t own = x;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= uint32_t(o)) x += y;
        }
        if (lane == 31) sw[warp] = x;
        __syncthreads();
        if (warp == 0) {
            uint32_t u = sw[lane];
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(0xffffffffu, u, o);
                if (lane >= uint32_t(o)) u += y;
            }
            sw[lane] = u;
        }
        __syncthreads();
        uint32_t at = carry + (warp > 0 ? sw[warp - 1] : 0u) + x - own;
#pragma unroll
        for (uint32_t j = 0; j < 4; ++j) {
            if (k + j >= nseg) break;
            seg_pre[k + j] = at;
            const uint32_t c = (at + kDeltaChunk - 1u) / kDeltaChunk;  // the first chunk that starts here or later
            if (c * kDeltaChunk < at + v[j]) chunk_seg[c] = k + j;
            at += v[j];
        }
        const uint32_t tot = sw[31];
        __syncthreads();
        carry += tot;
    }
    if (t == 0) seg_pre[nseg] = carry;
}

// Ap = A s' and delta, apply_matrix_and_dot's sum (:1823-1863): s'.Ap over the
// fluid cells in ascending order, in chunks of 8192 cells each summed serially
// from zero (rayon's par_chunks(8192)); the update then adds the chunk sums in
// chunk order.  s' is the iteration's search direction, z + beta s (the search
// update :1945-1954 is folded in).  One block per chunk: warps 1..15 form Ap and
// stage the products in fluid order in shared memory (positions from
// seg_pre), a stretch of segments at a time, while thread 0 adds those staged
// before, in order, the loads ahead of its add chain: a chunk costs its 8192
// dependent adds, and Ap is formed behind them.  An iteration of a 256^2 grid
// with 30657 fluid cells: 117 us staged as a whole first, 82 with this chain and
// the r.z sum's rows; Ap formed here instead of by a kernel before, and the
// chunk's segments from a table instead of a binary search, took 3 us more off
// it (64^2 44.2 -> 41.4, 256^2 88.1 -> 85.4, 1024^2 355 -> 349, moving scenes).
constexpr int kDeltaThreads = 512;
constexpr uint32_t kDeltaStretch = 60;  // segments staged at a time (15 warps, four each)
// first: of its loop body (counted).
__global__ void __launch_bounds__(kDeltaThreads) k_delta_exact(Level B, const float* __restrict__ s,
                                                               float* __restrict__ ap,
                                                               const uint32_t* __restrict__ seg_pre,
                                                               const uint32_t* __restrict__ chunk_seg, Ctl* ctl,
                                                               float* __restrict__ parts, int first) {
    __shared__ __align__(16) float prod[kDeltaChunk];
    pdl_wait();
    const float beta = ctl->beta;
    const bool beta_valid = ctl->beta_valid != 0;
    const uint32_t nseg = ctl->seg_count[0], nfluid = ctl->fluid_cells;
    const uint32_t c = blockIdx.x;
    const uint32_t f0 = c * kDeltaChunk;
    if (c == 0 && threadIdx.x == 0 && first) ctl->pcg_bodies++;
    if (ctl->pcg_done) return;
    // the buffer this iteration's update writes the residual to
    if (c == 0 && threadIdx.x == 0) ctl->res_sel = (ctl->pcg_iters + 1u) & 1u;
    if (f0 >= nfluid) return;
    const uint32_t f1 = min(f0 + kDeltaChunk, nfluid);
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    // segments [k0, k1) hold fluid cells f0 .. f1-1 (the last one may hold cells
    // of the next chunk too)
    const uint32_t k0 = chunk_seg[c];
    uint32_t k1 = nseg;
    if (f1 < nfluid) {
        k1 = chunk_seg[c + 1];
        if (seg_pre[k1] < f1) ++k1;
    }
    auto stage = [&](uint32_t from) {
        const uint32_t end = min(from + kDeltaStretch, k1);
#pragma unroll 4
        for (uint32_t k = from + warp - 1u; k < end; k += kDeltaThreads / 32 - 1) {
            const uint32_t w = B.seg[k], raw = w * 32u + lane;
            const uint32_t m = B.fluid[w], pre = seg_pre[k];
            if (raw >= B.cells) continue;
            float sc;
            const float v = pcg::apply_search(B, raw, s, beta, beta_valid, &sc);
            if (!((m >> lane) & 1u)) continue;
            const uint32_t pos = pre + uint32_t(__popc(m & ((1u << lane) - 1u)));
            if (pos < f0 || pos >= f1) continue;
            ap[raw + B.w] = v;
            prod[pos - f0] = v * sc;
        }
    };
    if (warp != 0) stage(k0);
    __syncthreads();
    float sum = 0.0f;
    uint32_t done = 0;  // products added (thread 0)
    for (uint32_t k = k0; k < k1; k += kDeltaStretch) {
        if (warp != 0) {
            if (k + kDeltaStretch < k1) stage(k + kDeltaStretch);
        } else if (threadIdx.x == 0) {
            // staged so far; the last stretch adds what is left, the others
            // whole vectors
            const uint32_t next = min(k + kDeltaStretch, k1);
            const uint32_t have = min(seg_pre[next], f1) - f0;
            const uint32_t n4 = (have - done) / 4u;
            sum = add_in_order<8>(reinterpret_cast<const float4*>(prod + done), n4, sum);
            done += 4u * n4;
            if (next == k1)
                for (; done < have; ++done) sum = sum + prod[done];
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) parts[c] = sum;
}

// ---- FP64 refinement helpers (APIC_SOLVER_REL_MIXED) ----------------------

// b64 = res, p64 = 0 (unless warm) and ||b||^2.
__device__ __forceinline__ void kb_mixed_init(Blk bk, const Level& B, double* b64, double* p64, Ctl* ctl,
                                              double* partials, int warm) {
    if (bk.id == 0 && threadIdx.x == 0) ctl->solve_t0 = global_ns();  // the relative-mode solve starts here
    double bb = pcg::ph_mixed_init(B, ctl->seg_count[0], blk_warp(bk), blk_nwarps(bk), b64, p64, warm);
    double tot;
    if (block_sum_last<kSegBlock>(bk, bb, partials, &ctl->red_counter, &tot) && threadIdx.x == 0) ctl->bnorm2 = tot;
}
// True relative residual of p64 (flags: see pcg::ph_true_residual).
// True in the one thread that formed it.
__device__ __forceinline__ bool kb_true_residual(Blk bk, const Level& B, const double* b64, const double* p64,
                                                 float* x, Ctl* ctl, double* partials, int flags) {
    if ((flags & 1) && bk.id == 0 && threadIdx.x == 0) ctl->res_sel = 0;
    double rr = pcg::ph_true_residual(B, ctl->seg_count[0], blk_warp(bk), blk_nwarps(bk), b64, p64, x, flags);
    double tot;
    if (!block_sum_last<kSegBlock>(bk, rr, partials, &ctl->red_counter, &tot) || threadIdx.x != 0) return false;
    ctl->true_rel = ctl->bnorm2 > 0.0 ? sqrt(tot / ctl->bnorm2) : 0.0;
    return true;
}
// p64 += x (finalize 0; the refinement also counts the inner solve's
// iterations), or pressure = float(p64) (finalize 1).
__device__ __forceinline__ void kb_mixed_accumulate(Blk bk, const Level& B, double* p64, const float* x,
                                                    float* pressure, Ctl* ctl, int finalize) {
    pcg::ph_accumulate(B, ctl->seg_count[0], blk_warp(bk), blk_nwarps(bk), p64, x, pressure, finalize);
    if (!finalize && bk.id == 0 && threadIdx.x == 0) ctl->used_iters += ctl->pcg_iters;
}
// ---- loop control (device side; each sets a graph conditional) ------------

__device__ __forceinline__ void finish_solve(Ctl* ctl, uint32_t cap) {
    ctl->solve_ns += global_ns() - ctl->solve_t0;
    ctl->pcg_iters_total += ctl->pcg_iters;
    if (ctl->pcg_iters >= cap && ctl->pcg_done != 1u) ctl->not_converged++;
}
__global__ void k_finish_solve(Ctl* ctl, uint32_t cap) { finish_solve(ctl, cap); }

// The FP32 mode's end: p64 = pressure, for its true residual.
__global__ void __launch_bounds__(kSegBlock) k_pressure_to64(Level B, const float* pressure, double* p64, Ctl* ctl,
                                                             uint32_t cap) {
    pdl_wait();
    if (blockIdx.x == 0 && threadIdx.x == 0) finish_solve(ctl, cap);
    pcg::ph_pressure_to64(B, ctl->seg_count[0], gwarp(), gnwarps(), pressure, p64);
}

__device__ __forceinline__ void rel_begin(Ctl* ctl, double tol, uint32_t cap) {
    pcg::set_target(ctl, tol);
    ctl->inner_cap = cap;
    ctl->refinements = 0;
    ctl->used_iters = 0;
}

// Refinement loop: go on while the FP64 true residual is above tol and
// iterations remain.  Each inner FP32 solve reduces its own right-hand side
// (the current true residual) by kInnerReduction, or down to tol / 2 of ||b||
// when that is reached first; FP32 cannot usefully reduce it further.
constexpr double kInnerReduction = 1e-4;
__device__ __forceinline__ bool refine_cond(Ctl* ctl, double tol, uint32_t cap) {
    bool cont = ctl->true_rel > tol && ctl->used_iters < cap && ctl->refinements < 32u;
    // an inner solve that could not take a single step (r.z underflows or is
    // zero) will not make progress on the next round either
    if (ctl->refinements > 0u && ctl->pcg_iters == 0u) cont = false;
    if (cont) {
        ctl->refinements++;
        ctl->inner_cap = cap - ctl->used_iters;
        double t = kInnerReduction * ctl->true_rel;  // target relative to ||b||
        pcg::set_target(ctl, t > 0.5 * tol ? t : 0.5 * tol);
        pcg_reset(ctl);  // the inner solve that follows starts here
    }
    ctl->cond = cont ? 1u : 0u;
    return cont;
}
// The true residual, and the refinement loop's decision on it (decide).
__global__ void __launch_bounds__(kSegBlock) k_true_residual(Level B, const double* b64, const double* p64, float* x,
                                                             Ctl* ctl, double* partials, int flags, int decide,
                                                             double tol, LoopEntry loop) {
    pdl_wait();
    if (!kb_true_residual(hw_blk(), B, b64, p64, x, ctl, partials, flags) || !decide) return;
    const bool cont = refine_cond(ctl, tol, loop.cap);
    if (loop.set) cudaGraphSetConditional(loop.h, cont ? 1u : 0u);
}

// A relative solve's start (pcg::ph_solve_start) with its targets and, mixed,
// the refinement loop's first decision.  One kernel: the five that stood here
// (||b||, zero pressure, targets, true residual, decision) took 25 us of a
// small scene's substep.
__global__ void __launch_bounds__(kSegBlock) k_solve_start(Level B, double* b64, double* p64, float* x,
                                                           float* pressure, Ctl* ctl, double* partials, int warm,
                                                           int mixed, double tol, LoopEntry loop) {
    pdl_wait();
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        ctl->solve_t0 = global_ns();
        ctl->res_sel = 0;
    }
    const double2 sums = pcg::ph_solve_start(B, ctl->seg_count[0], gwarp(), gnwarps(), b64, p64, x, pressure, warm, mixed);
    double2 tot;
    if (!block_sum_last<kSegBlock>(hw_blk(), sums, partials, partials + kMaxRedBlocks, &ctl->red_counter, &tot) ||
        threadIdx.x != 0)
        return;
    ctl->bnorm2 = tot.x;
    rel_begin(ctl, tol, loop.cap);
    if (!mixed) return;
    ctl->true_rel = tot.x > 0.0 ? sqrt(tot.y / tot.x) : 0.0;
    const bool cont = refine_cond(ctl, tol, loop.cap);
    if (loop.set) cudaGraphSetConditional(loop.h, cont ? 1u : 0u);
}

__device__ __forceinline__ void refine_end(Ctl* ctl, double tol) {
    ctl->solve_ns += global_ns() - ctl->solve_t0;
    ctl->refinements_total += ctl->refinements;
    ctl->pcg_iters = ctl->used_iters;
    ctl->pcg_iters_total += ctl->used_iters;
    if (ctl->true_rel > tol) ctl->not_converged++;
}

__global__ void __launch_bounds__(kSegBlock) k_mixed_accumulate(Level B, double* p64, const float* x, float* pressure,
                                                                Ctl* ctl, int finalize, double tol) {
    pdl_wait();
    kb_mixed_accumulate(hw_blk(), B, p64, x, pressure, ctl, finalize);
    if (finalize && blockIdx.x == 0 && threadIdx.x == 0) refine_end(ctl, tol);
}

// ---- the same phases over a batch of scenes (batch.h) ----------------------
// Segment phases: persistent CTAs walk the listed items of their gate (each a
// block of a scene's own launch, with that launch's coordinates) and run the
// single-scene body.  Control phases: one CTA, a thread per scene; they list
// the scenes for the phases that follow, and the OR of the scenes' loop
// decisions is the batch loop's condition.  The PCG runs in a relative mode
// (APIC_SOLVER_REL_FP32 arithmetic, as the inner solves of both relative
// modes do).
constexpr int kBatCtlThreads = 1024;
constexpr int kRel = APIC_SOLVER_REL_FP32;

// Start of the batch's solves: list the scenes with a substep due (their
// segment lists are those of this substep's multigrid setup).
__global__ void __launch_bounds__(kBatCtlThreads) k_bat_solve_begin(const BScene* __restrict__ tab, uint32_t n,
                                                                   const BCtl* bc, BListRef l1) {
    bat_build_list(tab, n, kGateSolve, l1, bc);
}

__global__ void __launch_bounds__(kBatCtlThreads) k_bat_rel_begin(const BScene* __restrict__ tab, uint32_t n,
                                                                 int mixed, const BCtl* bc, BListRef l2) {
    for (uint32_t i = threadIdx.x; i < n; i += blockDim.x) {
        Ctl* ctl = tab[i].ctl;
        if (!bat_gate(ctl, kGateSolve)) continue;
        rel_begin(ctl, tab[i].tol, tab[i].max_iter);
        if (!mixed) ctl->cond = 1u;  // no refinement loop: its gate stays open
    }
    if (mixed) return;
    __syncthreads();
    bat_build_list(tab, n, kGateRefine, l2, bc);
}

// gate kGateSolve: the loop's entry (every scene with a substep due decides);
// kGateRefine: the end of a refinement (the scenes still refining decide).
__global__ void __launch_bounds__(kBatCtlThreads) k_bat_refine_cond(const BScene* __restrict__ tab, uint32_t n,
                                                                   BCtl* bc, cudaGraphConditionalHandle h, int gate,
                                                                   BListRef l2) {
    bool any = false;
    for (uint32_t i = threadIdx.x; i < n; i += blockDim.x) {
        Ctl* ctl = tab[i].ctl;
        if (bat_gate(ctl, gate) && refine_cond(ctl, tab[i].tol, tab[i].max_iter)) any = true;
    }
    any = __syncthreads_or(any) != 0;
    if (threadIdx.x == 0) {
        cudaGraphSetConditional(h, any ? 1u : 0u);
        if (any) bc->refine_iters++;
    }
    if (any) bat_build_list(tab, n, kGateRefine, l2, bc);
}

__global__ void __launch_bounds__(kBatCtlThreads) k_bat_refine_end(const BScene* __restrict__ tab, uint32_t n) {
    for (uint32_t i = threadIdx.x; i < n; i += blockDim.x)
        if (bat_gate(tab[i].ctl, kGateSolve)) refine_end(tab[i].ctl, tab[i].tol);
}

__global__ void __launch_bounds__(kBatCtlThreads) k_bat_finish_solve(const BScene* __restrict__ tab, uint32_t n) {
    for (uint32_t i = threadIdx.x; i < n; i += blockDim.x)
        if (bat_gate(tab[i].ctl, kGateSolve)) finish_solve(tab[i].ctl, tab[i].max_iter);
}

__global__ void __launch_bounds__(kBatCtlThreads) k_bat_pcg_begin(const BScene* __restrict__ tab, uint32_t n,
                                                                 int gate) {
    for (uint32_t i = threadIdx.x; i < n; i += blockDim.x)
        if (bat_gate(tab[i].ctl, gate)) pcg_reset(tab[i].ctl);
}

// Entry of the PCG loops (k_pcg_cond with the refinement's dynamic cap).
__global__ void __launch_bounds__(kBatCtlThreads) k_bat_pcg_cond(const BScene* __restrict__ tab, uint32_t n,
                                                                const BCtl* bc, cudaGraphConditionalHandle h,
                                                                int gate, BListRef l3) {
    pdl_wait();
    bool any = false;
    for (uint32_t i = threadIdx.x; i < n; i += blockDim.x) {
        Ctl* ctl = tab[i].ctl;
        if (!bat_gate(ctl, gate)) continue;
        const bool cont = pcg_entry(ctl, 0u, 1);
        ctl->pcg_on = cont ? 1u : 0u;
        any = any || cont;
    }
    any = __syncthreads_or(any) != 0;
    if (threadIdx.x == 0) cudaGraphSetConditional(h, any ? 1u : 0u);
    if (any) bat_build_list(tab, n, kGatePcg, l3, bc);
}

// End of a batch PCG iteration: the exit items have taken every listed
// scene's decision.  CTA 0 lists the scenes that go on and sets the loop
// condition; CTA 1 + i sums scene i's r.z parts (stored by the V-cycle's
// last kernel) for the next iteration, once instead of in every block of
// k_spmv_dot and k_update_down (the same function of the same parts).
__global__ void __launch_bounds__(kSegBlock) k_bat_round_end(const BScene* __restrict__ tab, uint32_t n, BCtl* bc,
                                                            cudaGraphConditionalHandle h, BListRef l3) {
    pdl_wait();
    if (blockIdx.x == 0) {
        bat_build_list(tab, n, kGatePcg, l3, bc);
        if (threadIdx.x == 0) {
            cudaGraphSetConditional(h, l3.p[0] ? 1u : 0u);
            bc->pcg_iters++;
        }
        return;
    }
    const BScene& S = tab[blockIdx.x - 1];
    Ctl* ctl = S.ctl;
    if (!bat_gate(ctl, kGatePcg) || ctl->pcg_done) return;
    const float rz = sum_partials<kSegBlock>(bs_part_rz(S), busy_tile_blocks(S));
    if (threadIdx.x == 0) ctl->b_rz = rz;
}

// s.Ap of every listed scene (after k_bat_spmv_dot), once per scene.
__global__ void __launch_bounds__(kSegBlock) k_bat_sap(const BScene* __restrict__ tab, uint32_t n) {
    pdl_wait();
    const BScene& S = tab[blockIdx.x];
    Ctl* ctl = S.ctl;
    if (!bat_gate(ctl, kGatePcg) || ctl->pcg_done) return;
    const float sap = sum_partials<kSegBlock>(bs_part_sap(S), busy_blocks(S));
    if (threadIdx.x == 0) ctl->b_sap = sap;
}

__global__ void __launch_bounds__(kSegBlock) k_bat_mixed_init(const BScene* __restrict__ tab, BListRef L, int gate) {
    bat_for_items(L, kKindBase, false, [&](uint32_t sc, uint32_t lb, Shape sh) {
        const BScene& S = tab[sc];
        if (!bat_gate(S.ctl, gate)) return;
        kb_mixed_init(Blk{lb, S.grid[0]}, S.lv[0], S.b64, S.p64, S.ctl, S.partials, S.warm);
    });
}

__global__ void __launch_bounds__(kSegBlock) k_bat_clear_pressure(const BScene* __restrict__ tab, BListRef L,
                                                                  int gate) {
    bat_for_items(L, kKindChunk, false, [&](uint32_t sc, uint32_t lb, Shape sh) {
        const BScene& S = tab[sc];
        if (!bat_gate(S.ctl, gate)) return;
        const Chunk ch = chunk_of(lb, S.ctl->seg_count[0], sh);
        pcg::ph_clear_pressure(S.lv[0], ch.end, ch.warp, ch.nwarps, S.pressure);
    });
}

__global__ void __launch_bounds__(kSegBlock) k_bat_true_residual(const BScene* __restrict__ tab, BListRef L, int gate,
                                                                 int flags) {
    bat_for_items(L, kKindBase, false, [&](uint32_t sc, uint32_t lb, Shape sh) {
        const BScene& S = tab[sc];
        if (!bat_gate(S.ctl, gate)) return;
        kb_true_residual(Blk{lb, S.grid[0]}, S.lv[0], S.b64, S.p64, S.corr, S.ctl, S.partials, flags);
    });
}

__global__ void __launch_bounds__(kSegBlock) k_bat_pcg_start(const BScene* __restrict__ tab, BListRef L, int gate) {
    bat_for_items(L, kKindBase, false, [&](uint32_t sc, uint32_t lb, Shape sh) {
        const BScene& S = tab[sc];
        if (!bat_gate(S.ctl, gate)) return;
        kb_pcg_start(Blk{lb, S.grid[0]}, S.lv[0], S.search, S.ctl, S.partials, kRel);
    });
}

__global__ void __launch_bounds__(kSegBlock, 8) k_bat_spmv_dot(const BScene* __restrict__ tab, BListRef L) {
    bat_for_items(L, kKindBlocks, false, [&](uint32_t sc, uint32_t item, Shape sh) {
        const BScene& S = tab[sc];
        Ctl* ctl = S.ctl;
        if (!bat_gate(ctl, kGatePcg)) return;
        const uint32_t nseg = ctl->seg_count[0], end = group_end(S, item, sh);
        for (uint32_t b = item * sh.block_group; b < end; ++b) {
            kb_spmv_dot(Blk{b, S.sgrid}, S.lv[0], nseg, 0xFFFFFFFFu, S.search, S.ap, ctl, bs_part_sap(S),
                        bs_part_rz(S), S.tgrid, &ctl->b_rz);
            __syncthreads();  // block_store's shared slots are reused by the next block
        }
    });
}

__global__ void __launch_bounds__(kTileBlock, 4) k_bat_update_down(const BScene* __restrict__ tab, BListRef L,
                                                                     int into_corr) {
    __shared__ tile::Shared sh;
    bat_for_items(L, kKindTiles0, true, [&](uint32_t sc, uint32_t item, Shape shp) {
        const BScene& S = tab[sc];
        Ctl* ctl = S.ctl;
        if (!bat_gate(ctl, kGatePcg)) return;
        const uint32_t count = ctl->tile_count[0], end = tile_group_end(S, item, shp);
        const StepArgs a{bs_part_sap(S), S.sgrid, kRel, nullptr, nullptr, bs_part_rz(S), S.tgrid};
        for (uint32_t b = item * shp.block_group; b < end; ++b) {
            tile::DownRegs g;
            const uint32_t id = b < count ? S.lv[0].tiles[b] : 0u;
            if (b < count) tile::down_load_const<true>(S.lv[0], id, g);
            kb_update_down<true>(Blk{b, S.tgrid}, S.lv[0], S.lv[1], sh, g, count, id, into_corr ? S.corr : S.pressure,
                           into_corr, S.search, S.ap, ctl, a, bs_part_res(S), -1, &ctl->b_rz, &ctl->b_sap);
            __syncthreads();
        }
    });
}

// The exit test and loop decision of every listed scene after its update
// (k_bat_round_end then lists the scenes that go on).
__global__ void __launch_bounds__(kSegBlock) k_bat_exit(const BScene* __restrict__ tab, uint32_t n) {
    pdl_wait();
    const BScene& S = tab[blockIdx.x];
    Ctl* ctl = S.ctl;
    if (!bat_gate(ctl, kGatePcg)) return;
    if (!ctl->pcg_done) pcg::residual_exit(ctl, bs_part_res(S), busy_tile_blocks(S), APIC_SOLVER_REL_FP32, 0.0f);
    if (threadIdx.x == 0) ctl->pcg_on = pcg::loop_continue(ctl, APIC_SOLVER_REL_FP32, 0u, 1) ? 1u : 0u;
}

// (k_mixed_accumulate: chunk 0 also counts the inner solve's iterations)
__global__ void __launch_bounds__(kSegBlock) k_bat_mixed_accumulate(const BScene* __restrict__ tab, BListRef L,
                                                                    int gate, int finalize) {
    bat_for_items(L, kKindChunk, false, [&](uint32_t sc, uint32_t lb, Shape sh) {
        const BScene& S = tab[sc];
        Ctl* ctl = S.ctl;
        if (!bat_gate(ctl, gate)) return;
        const Chunk ch = chunk_of(lb, ctl->seg_count[0], sh);
        pcg::ph_accumulate(S.lv[0], ch.end, ch.warp, ch.nwarps, S.p64, S.corr, S.pressure, finalize);
        if (!finalize && lb == 0 && threadIdx.x == 0) ctl->used_iters += ctl->pcg_iters;
    });
}

__global__ void __launch_bounds__(kSegBlock) k_bat_pressure_to64(const BScene* __restrict__ tab, BListRef L,
                                                                 int gate) {
    bat_for_items(L, kKindChunk, false, [&](uint32_t sc, uint32_t lb, Shape sh) {
        const BScene& S = tab[sc];
        if (!bat_gate(S.ctl, gate)) return;
        const Chunk ch = chunk_of(lb, S.ctl->seg_count[0], sh);
        pcg::ph_pressure_to64(S.lv[0], ch.end, ch.warp, ch.nwarps, S.pressure, S.p64);
    });
}

}  // namespace

// ---- batch phase launchers (batch.h); launch kinds as in the single-scene
// graph: programmatic dependent launch where the predecessor is a kernel of
// the PCG setup or loop, plain launches elsewhere ----
#define APIC_PGRID(kern) static const uint32_t g = persistent_grid(kern, kSegBlock, 0)
void bat_solve_begin(const BatchRun& r) {
    k_bat_solve_begin<<<1, kBatCtlThreads, 0, r.st>>>(r.tab, r.nscenes, r.bc, r.list[kGateSolve]);
}
void bat_mixed_init(const BatchRun& r, int gate) {
    APIC_PGRID(k_bat_mixed_init);
    launch(false, k_bat_mixed_init, g, kSegBlock, 0, r.st, r.tab, r.list[gate], gate);
}
void bat_clear_pressure(const BatchRun& r, int gate) {
    APIC_PGRID(k_bat_clear_pressure);
    launch(false, k_bat_clear_pressure, g, kSegBlock, 0, r.st, r.tab, r.list[gate], gate);
}
void bat_rel_begin(const BatchRun& r, int mixed) {
    k_bat_rel_begin<<<1, kBatCtlThreads, 0, r.st>>>(r.tab, r.nscenes, mixed, r.bc, r.list[kGateRefine]);
}
void bat_true_residual(const BatchRun& r, int gate, int flags) {
    APIC_PGRID(k_bat_true_residual);
    launch(false, k_bat_true_residual, g, kSegBlock, 0, r.st, r.tab, r.list[gate], gate, flags);
}
void bat_refine_cond(const BatchRun& r, cudaGraphConditionalHandle h, int gate) {
    k_bat_refine_cond<<<1, kBatCtlThreads, 0, r.st>>>(r.tab, r.nscenes, r.bc, h, gate, r.list[kGateRefine]);
}
void bat_pcg_begin(const BatchRun& r, int gate) {
    k_bat_pcg_begin<<<1, kBatCtlThreads, 0, r.st>>>(r.tab, r.nscenes, gate);
}
void bat_pcg_start(const BatchRun& r, int gate) {
    APIC_PGRID(k_bat_pcg_start);
    launch(r.pdl, k_bat_pcg_start, g, kSegBlock, 0, r.st, r.tab, r.list[gate], gate);
}
void bat_pcg_cond(const BatchRun& r, cudaGraphConditionalHandle h, int gate) {
    launch(r.pdl, k_bat_pcg_cond, 1, kBatCtlThreads, 0, r.st, r.tab, r.nscenes, static_cast<const BCtl*>(r.bc), h,
           gate, r.list[kGatePcg]);
}
void bat_round_end(const BatchRun& r, cudaGraphConditionalHandle h) {
    launch(r.pdl, k_bat_round_end, r.nscenes + 1, kSegBlock, 0, r.st, r.tab, r.nscenes, r.bc, h, r.list[kGatePcg]);
}
void bat_sap(const BatchRun& r) { launch(r.pdl, k_bat_sap, r.nscenes, kSegBlock, 0, r.st, r.tab, r.nscenes); }
void bat_spmv_dot(const BatchRun& r) {
    APIC_PGRID(k_bat_spmv_dot);
    k_bat_spmv_dot<<<g, kSegBlock, 0, r.st>>>(r.tab, r.list[kGatePcg]);
}
void bat_update_down(const BatchRun& r, int into_corr) {
    APIC_PGRID(k_bat_update_down);
    launch(r.pdl, k_bat_update_down, g, kTileBlock, 0, r.st, r.tab, r.list[kGatePcg], into_corr);
}
void bat_exit(const BatchRun& r) { launch(r.pdl, k_bat_exit, r.nscenes, kSegBlock, 0, r.st, r.tab, r.nscenes); }
void bat_mixed_accumulate(const BatchRun& r, int gate, int finalize) {
    APIC_PGRID(k_bat_mixed_accumulate);
    launch(false, k_bat_mixed_accumulate, g, kSegBlock, 0, r.st, r.tab, r.list[gate], gate, finalize);
}
void bat_refine_end(const BatchRun& r) { k_bat_refine_end<<<1, kBatCtlThreads, 0, r.st>>>(r.tab, r.nscenes); }
void bat_finish_solve(const BatchRun& r) { k_bat_finish_solve<<<1, kBatCtlThreads, 0, r.st>>>(r.tab, r.nscenes); }
void bat_pressure_to64(const BatchRun& r, int gate) {
    APIC_PGRID(k_bat_pressure_to64);
    launch(false, k_bat_pressure_to64, g, kSegBlock, 0, r.st, r.tab, r.list[gate], gate);
}
#undef APIC_PGRID

ExitArgs exit_args(const Scene& s, int mode) {
    ExitArgs a;
    a.on = 1;
    a.part = part_res(s);
    a.nparts = s.nlevels >= 2 ? tile_grid(s.lv[0]) : seg_grid(s.lv[0].words);
    a.mode = mode;
    a.solve_error = s.props.solve_error;
    a.h = s.pcg_h;
    a.cap = s.pcg_cap;
    a.dyn_cap = s.pcg_dyn_cap;
    a.set_cond = s.pcg_set_cond ? 1 : 0;
    return a;
}

// (behind the prefix counts of the base level's segments)
static uint32_t* chunk_seg(const Scene& s) { return s.seg_pre + s.lv[0].words + 1; }

// One PCG iteration (src/apic.rs:1899-1955); x receives alpha * s.  The
// search update that ends the reference's iteration happens at the start of
// the next one (inside k_spmv_dot / k_update_down).
static void pcg_iteration(Scene& s, int mode, float* x, int p_padded, bool first, int sel) {
    const Level& B = s.lv[0];
    const uint32_t g = seg_grid(B.words), tg = tile_grid(B), sg = spmv_grid(B);
    cudaStream_t st = s.stream;
    const bool pdl = s.use_pdl, tiled = s.nlevels >= 2;
    const uint32_t nrz = tiled ? tg : g;
    if (mode == APIC_SOLVER_REFERENCE)
        launch(pdl && !first, k_delta_exact, div_up(B.cells, kDeltaChunk), kDeltaThreads, 0, st, B,
               static_cast<const float*>(s.search), s.ap, static_cast<const uint32_t*>(s.seg_pre),
               static_cast<const uint32_t*>(chunk_seg(s)), s.ctl, s.exact_parts, first ? 1 : 0);
    else
        launch(pdl && !first, k_spmv_dot, sg, kSegBlock, 0, st, B, static_cast<const float*>(s.search), s.ap, s.ctl,
               part_sap(s), static_cast<const float2*>(part_rz(s)), nrz, first ? 1 : 0);
    const StepArgs a{part_sap(s), sg, mode, s.exact_parts, s.seg_pre, part_rz(s), nrz};
    if (tiled) {
        launch(pdl, tile::reads_all(B) ? k_update_down<true> : k_update_down<false>, tg, kTileBlock, 0, st, B, s.lv[1], x, p_padded, s.search,
               static_cast<const float*>(s.ap), s.ctl, a, part_res(s), sel);
        // the V-cycle's next kernel runs the residual's exit test, its last
        // one stores the parts of r.z
        enqueue_vcycle(s, true, exit_args(s, mode), sel);
    } else {
        launch(pdl, k_pcg_update, g, kSegBlock, 0, st, B, x, p_padded, s.search, static_cast<const float*>(s.ap),
               s.ctl, a, part_res(s));
        launch(pdl, k_residual_exit, 1, kSegBlock, 0, st, s.ctl, exit_args(s, mode));
        enqueue_vcycle(s, true);
        launch(pdl, k_dot_rz, g, kSegBlock, 0, st, B, s.ctl, part_rz(s));
    }
    if (mode == APIC_SOLVER_REFERENCE)
        launch(pdl, k_gamma_exact, 1, kGammaThreads, kGammaSmem, st, B, s.ctl, 0, s.pcg_h, s.pcg_cap, s.pcg_dyn_cap,
               s.pcg_set_cond ? 1 : 0);
}

// Iterations in the body of the PCG loop.  Going round a graph's WHILE node
// costs 5 us; within the body the next iteration's first kernel is a
// programmatic dependent like the others.  An iteration that the body holds
// beyond the solve's last one costs its kernels' launches (they return at
// once).  Two iterations pay up to 768^2 cells, per iteration: 64^2 29.7 -> 28.3
// us, 216^2 36.6 -> 34.1, 512^2 46.6 -> 46.0, 768^2 55.6 -> 55.0; not at 1024^2
// (57.8, 58.0) and 1000 x 600 (70.5, 71.1).  Four are 2% faster where a solve
// takes 16 iterations or more and 1-2% slower where it takes 6 to 8.  The
// reference mode's solves take 3 to 9 and six kernels each: 128^2 67.1 us, with
// two 68.3.
static int loop_body(const Scene& s, int mode) {
    return mode != APIC_SOLVER_REFERENCE && s.cells <= 768u * 768u ? 2 : 1;
}

// PCG setup (src/apic.rs:1885-1892): z = M^-1 r, s = z, gamma, the loop's entry.
// begin: reset the PCG state first (the refinement loop's decision has already
// done so for its inner solves).
static void enqueue_pcg_start(Scene& s, int mode, bool begin, const LoopEntry& loop) {
    const Level& B = s.lv[0];
    const uint32_t g = seg_grid(B.words);
    cudaStream_t st = s.stream;
    const bool pdl = s.use_pdl;
    if (mode == APIC_SOLVER_REFERENCE) {
        launch(pdl, k_reference_start, 1u + std::min(div_up(B.words, 32), 304u), 1024, 0, st, B, s.pressure, s.ctl,
               s.seg_pre, chunk_seg(s));
    } else if (begin) {
        launch(pdl, k_pcg_begin, 1, 1, 0, st, s.ctl);
    }
    enqueue_vcycle(s);
    launch(pdl, k_pcg_start, g, kSegBlock, 0, st, B, s.search, s.ctl, s.partials, mode, loop);
    if (mode == APIC_SOLVER_REFERENCE)
        launch(pdl, k_gamma_exact, 1, kGammaThreads, kGammaSmem, st, B, s.ctl, 1, loop.h, loop.cap, loop.dyn_cap,
               loop.set);
}

// The setup followed by a device-controlled WHILE loop over iterations.
static cudaError_t build_pcg(Scene& s, GraphCursor& c, int mode, float* x, int p_padded, uint32_t cap, int dyn_cap,
                             bool begin = true) {
    cudaGraphConditionalHandle h;
    cudaError_t e = cudaGraphConditionalHandleCreate(&h, c.g, 0, cudaGraphCondAssignDefault);
    if (e != cudaSuccess) return e;
    const LoopEntry loop{h, cap, dyn_cap, 1};
    e = capture_into(s, c, [&]() {
        enqueue_pcg_start(s, mode, begin, loop);
        return cudaGetLastError();
    });
    if (e != cudaSuccess) return e;
    GraphCursor body;
    e = add_conditional_with(c, cudaGraphCondTypeWhile, h, &body);
    if (e != cudaSuccess) return e;
    // the loop condition is set inside the iteration (the residual's exit test,
    // or k_gamma_exact in the reference mode): no kernel of its own
    s.pcg_h = h;
    s.pcg_cap = cap;
    s.pcg_dyn_cap = dyn_cap;
    s.pcg_set_cond = true;
    e = capture_into(s, body, [&]() {
        const int n = loop_body(s, mode);
        for (int k = 0; k < n; ++k) pcg_iteration(s, mode, x, p_padded, k == 0, n % 2 == 0 ? (k + 1) & 1 : -1);
        return cudaGetLastError();
    });
    s.pcg_set_cond = false;
    s.kn_pcg = count_kernel_nodes(body.g);
    return e;
}

cudaError_t build_solve(Scene& s, GraphCursor& c) {
    s.kn_pcg = s.kn_refine = 0;
    cudaFuncSetAttribute(k_gamma_exact, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kGammaSmem));
    const Level& B = s.lv[0];
    uint32_t g = seg_grid(B.words);
    int mode = s.solver_mode;
    s.p64_valid = false;
    cudaError_t e;
    if (mode == APIC_SOLVER_REFERENCE) {
        e = build_pcg(s, c, mode, s.pressure, 0, 100, 0);
        if (e != cudaSuccess) return e;
        return capture_into(s, c, [&]() {
            k_finish_solve<<<1, 1, 0, s.stream>>>(s.ctl, 100);
            return cudaGetLastError();
        });
    }
    const double tol = double(s.rel_tol);
    const bool mixed = mode == APIC_SOLVER_REL_MIXED;
    cudaGraphConditionalHandle hr = 0;
    if (mixed) {
        e = cudaGraphConditionalHandleCreate(&hr, c.g, 0, cudaGraphCondAssignDefault);
        if (e != cudaSuccess) return e;
    }
    const LoopEntry refine{hr, s.max_iter, 0, mixed ? 1 : 0}, none{};
    e = capture_into(s, c, [&]() {
        launch(s.use_pdl, k_solve_start, g, kSegBlock, 0, s.stream, B, s.b64, s.p64, s.corr, s.pressure, s.ctl,
               s.partials, int(warm_start(s)), mixed ? 1 : 0, tol, refine);
        return cudaGetLastError();
    });
    if (e != cudaSuccess) return e;
    auto true_residual = [&](int flags, int decide, const LoopEntry& loop) {
        launch(s.use_pdl, k_true_residual, g, kSegBlock, 0, s.stream, B, static_cast<const double*>(s.b64),
               static_cast<const double*>(s.p64), s.corr, s.ctl, s.partials, flags, decide, tol, loop);
    };
    if (!mixed) {
        e = build_pcg(s, c, APIC_SOLVER_REL_FP32, s.pressure, 0, s.max_iter, 1);
        if (e != cudaSuccess) return e;
        // true residual of the FP32 pressure that the projection will use
        return capture_into(s, c, [&]() {
            k_pressure_to64<<<g, kSegBlock, 0, s.stream>>>(B, s.pressure, s.p64, s.ctl, s.max_iter);
            true_residual(1, 0, none);
            return cudaGetLastError();
        });
    }
    // APIC_SOLVER_REL_MIXED: r = b - A p in FP64, FP32 PCG on A d = r, p += d.
    GraphCursor body;
    e = add_conditional_with(c, cudaGraphCondTypeWhile, hr, &body);
    if (e != cudaSuccess) return e;
    e = build_pcg(s, body, APIC_SOLVER_REL_FP32, s.corr, 1, s.max_iter, 1, false);
    if (e != cudaSuccess) return e;
    e = capture_into(s, body, [&]() {
        k_mixed_accumulate<<<g, kSegBlock, 0, s.stream>>>(B, s.p64, s.corr, s.pressure, s.ctl, 0, tol);
        true_residual(3, 1, refine);
        return cudaGetLastError();
    });
    if (e != cudaSuccess) return e;
    s.kn_refine = count_kernel_nodes(body.g);
    // the projection uses the FP64 pressure; its true residual is the one reported
    s.p64_valid = true;
    return capture_into(s, c, [&]() {
        k_mixed_accumulate<<<g, kSegBlock, 0, s.stream>>>(B, s.p64, s.corr, s.pressure, s.ctl, 1, tol);
        return cudaGetLastError();
    });
}

// ---- eager form (profiling): same kernels, host-side loop control ----------

static cudaError_t read_ctl(Scene& s) {
    cudaError_t e = cudaMemcpyAsync(s.ctl_host, s.ctl, sizeof(Ctl), cudaMemcpyDeviceToHost, s.stream);
    if (e != cudaSuccess) return e;
    return cudaStreamSynchronize(s.stream);
}

// PCG setup and iterations until the device flags convergence or the cap.
static cudaError_t eager_pcg(Scene& s, int mode, float* x, int p_padded, uint32_t cap) {
    enqueue_pcg_start(s, mode, true, LoopEntry{});
    s.pcg_set_cond = false;
    s.pcg_cap = cap;
    s.pcg_dyn_cap = 0;
    for (;;) {
        cudaError_t e = read_ctl(s);
        if (e != cudaSuccess) return e;
        if (s.ctl_host->pcg_done || s.ctl_host->pcg_iters >= cap) break;
        pcg_iteration(s, mode, x, p_padded, true, -1);
    }
    return cudaGetLastError();
}

cudaError_t run_solve_eager(Scene& s) {
    cudaFuncSetAttribute(k_gamma_exact, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kGammaSmem));
    const Level& B = s.lv[0];
    uint32_t g = seg_grid(B.words);
    cudaStream_t st = s.stream;
    int mode = s.solver_mode;
    s.p64_valid = false;
    cudaError_t e;
    if (mode == APIC_SOLVER_REFERENCE) {
        if ((e = eager_pcg(s, mode, s.pressure, 0, 100)) != cudaSuccess) return e;
        k_finish_solve<<<1, 1, 0, st>>>(s.ctl, 100);
        return cudaGetLastError();
    }
    const double tol = double(s.rel_tol);
    const bool mixed = mode == APIC_SOLVER_REL_MIXED;
    const LoopEntry refine{0, s.max_iter, 0, 0};
    k_solve_start<<<g, kSegBlock, 0, st>>>(B, s.b64, s.p64, s.corr, s.pressure, s.ctl, s.partials, int(warm_start(s)),
                                            mixed ? 1 : 0, tol, refine);
    if (!mixed) {
        if ((e = eager_pcg(s, mode, s.pressure, 0, s.max_iter)) != cudaSuccess) return e;
        k_pressure_to64<<<g, kSegBlock, 0, st>>>(B, s.pressure, s.p64, s.ctl, s.max_iter);
        k_true_residual<<<g, kSegBlock, 0, st>>>(B, s.b64, s.p64, s.corr, s.ctl, s.partials, 1, 0, tol, refine);
        return cudaGetLastError();
    }
    for (;;) {
        if ((e = read_ctl(s)) != cudaSuccess) return e;
        if (!s.ctl_host->cond) break;
        if ((e = eager_pcg(s, APIC_SOLVER_REL_FP32, s.corr, 1, s.ctl_host->inner_cap)) != cudaSuccess) return e;
        k_mixed_accumulate<<<g, kSegBlock, 0, st>>>(B, s.p64, s.corr, s.pressure, s.ctl, 0, tol);
        k_true_residual<<<g, kSegBlock, 0, st>>>(B, s.b64, s.p64, s.corr, s.ctl, s.partials, 3, 1, tol, refine);
    }
    s.p64_valid = true;
    k_mixed_accumulate<<<g, kSegBlock, 0, st>>>(B, s.p64, s.corr, s.pressure, s.ctl, 1, tol);
    return cudaGetLastError();
}

}  // namespace apic
