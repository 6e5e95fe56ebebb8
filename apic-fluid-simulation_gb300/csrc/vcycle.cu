// vcycle.cu — the multigrid V-cycle preconditioner (z = M^-1 r).
//
// Restates Apic::apply_preconditioner (src/apic.rs:1788-1821) and the
// MultiGridLevel methods it calls: red/black SOR with omega = 1.2 and one
// sweep each way (smooth_level, :471-535), restriction of r - A e over the 2x2
// children of each coarse fluid cell (restrict, :537-594), piecewise-constant
// prolongation (prolongate, :596-616) and plain CG on the coarsest level
// (solve_coarse_exact, :618-704).
//
// Launch structure (one CUDA-graph node each), chosen to cut dependent
// launches per PCG iteration while keeping the reference's arithmetic:
//   * a level that the whole grid works on takes two kernels, on tiles with a
//     halo in shared memory (k_down, k_up; tiles.cuh): the two sweeps and the
//     restriction going down, the prolongation and the two reverse sweeps
//     going up; on the base level the PCG update runs in the down kernel and
//     r.z in the up kernel;
//   * all levels that fit in shared memory (the coarse tail, including the
//     coarsest CG) run in ONE cooperative CTA: coefficients are loaded from L2
//     once per V-cycle and every sweep is a __syncthreads()-separated phase
//     (k_vcycle_tail);
//   * the middle levels above the tail (a few thousand to some tens of
//     thousands of fluid cells: too small to fill the GPU, so each of their
//     launches costs mostly its latency) live in the distributed shared
//     memory of one thread-block cluster together with the tail
//     (k_vcycle_dsm, vcycle_dsm.cu).
// On the base level the last fluid cell receives the coarse correction once
// more per duplicate that pads the reference's fluid list to a multiple of 8
// (:1487-1494, iterated by prolongate :611-615).
#include <cuda_runtime.h>

#include "apic_device.cuh"
#include "apic_internal.h"
#include "batch.h"
#include "pcg_common.cuh"
#include "tiles.cuh"
#include "vcycle_common.cuh"

namespace apic {
using namespace vc;
namespace {

__device__ __forceinline__ uint32_t gwarp() { return (blockIdx.x * blockDim.x + threadIdx.x) >> 5; }
__device__ __forceinline__ uint32_t gnwarps() { return (gridDim.x * blockDim.x) >> 5; }

// Segment lists and their lengths are written by the multigrid setup, never
// by the kernel just before: each warp loads its first segment word before
// waiting on that kernel (programmatic dependent launch).
__device__ __forceinline__ uint32_t early_word(const uint32_t* seg, uint32_t nseg) {
    const uint32_t s = gwarp();
    return s < nseg ? seg[s] : kNoWord;
}

// One colour sweep (grids without a coarser level).
__global__ void __launch_bounds__(kSegBlock) k_smooth(Level L, int li, const Ctl* ctl, int color, int init) {
    const uint32_t nseg = ctl->seg_count[li];
    const uint32_t w0 = early_word(L.seg, nseg);
    pdl_wait();
    if (ctl->pcg_done) return;
    ph_smooth(L, nseg, gwarp(), gnwarps(), color, init, w0);
}

// Level f's red and black sweeps and the restriction into c (tiles.cuh).  In
// an iteration the first of these kernels after the update also runs the
// update's exit test and the loop's decision, in an extra block beside the
// sweeps; later kernels see its verdict.
template <bool kAll>
__device__ __forceinline__ void kb_down(Blk bk, const Level& f, const Level& c, tile::Shared& sh, tile::DownRegs& g,
                                        uint32_t id, uint32_t end, const float* res) {
    const tile::Update none{};
    for (uint32_t i = bk.id; i < end; i += bk.n) {
        if (i != bk.id) {
            id = f.tiles[i];
            __syncthreads();  // the tile before this one has been read
            tile::down_load_const<kAll>(f, id, g);
        }
        tile::down_load<false, kAll>(f, res, none, g);
        tile::down_tile<false>(sh, f, c, id, g, none, 0.0f, 0.0f, false, nullptr, nullptr);
    }
}
template <bool kAll>
__global__ void __launch_bounds__(kTileBlock, 4) k_down(Level f, Level c, int lf, Ctl* ctl, ExitArgs exit) {
    __shared__ tile::Shared sh;
    const uint32_t extra = exit.on ? 1u : 0u;
    if (exit.on && blockIdx.x == 0) {
        pdl_wait();
        if (!ctl->pcg_done) pcg::residual_exit(ctl, exit.part, exit.nparts, exit.mode, exit.solve_error);
        if (threadIdx.x == 0)
            pcg::loop_decision(ctl, exit.mode, exit.h, exit.cap, exit.dyn_cap, exit.set_cond);
        return;
    }
    const Blk bk{blockIdx.x - extra, gridDim.x - extra};
    const uint32_t count = ctl->tile_count[lf];
    const uint32_t id = bk.id < count ? f.tiles[bk.id] : 0u;
    tile::DownRegs g;
    if (bk.id < count) tile::down_load_const<kAll>(f, id, g);
    pdl_wait();
    // (block 0 may be writing the flag: the block's threads must agree on it, or
    // some would sweep a tile that others have left)
    if (exit.on ? __syncthreads_or(ctl->pcg_done != 0) != 0 : ctl->pcg_done != 0) return;
    kb_down<kAll>(bk, f, c, sh, g, id, count, lf == 0 ? pcg::cur_res(f, ctl) : f.res);
}

// The prolongation from c and level f's black and red sweeps; kRz: the base
// level in an iteration, whose part of r.z is stored too (the next iteration
// sums the parts).
template <bool kRz, bool kAll>
__device__ __forceinline__ F2 kb_up(Blk bk, const Level& c, const Level& f, tile::Shared& sh, tile::UpRegs& g,
                                    uint32_t id, uint32_t end, const float* res, uint32_t last, uint32_t extra) {
    F2 acc{0.0f, 0.0f};
    for (uint32_t i = bk.id; i < end; i += bk.n) {
        if (i != bk.id) {
            id = f.tiles[i];
            __syncthreads();  // the tile before this one has been read
            tile::up_load_const<kAll>(f, id, g);
        }
        tile::up_load<kAll>(c, f, res, last, extra, g);
        tile::up_tile<kRz>(sh, f, g, &acc);
    }
    return acc;
}
// sel: the base residual's buffer, or -1: as Ctl::res_sel says.
template <bool kRz, bool kAll>
__global__ void __launch_bounds__(kTileBlock, 4) k_up(Level c, Level f, int lf, const Ctl* ctl, int base,
                                                        float2* part, int sel) {
    __shared__ tile::Shared sh;
    const uint32_t count = ctl->tile_count[lf];
    const uint32_t id = blockIdx.x < count ? f.tiles[blockIdx.x] : 0u;
    const uint32_t last = base ? ctl->last_fluid : 0xFFFFFFFFu, extra = base ? ctl->pad_count : 0u;
    tile::UpRegs g;
    if (blockIdx.x < count) tile::up_load_const<kAll>(f, id, g);
    pdl_wait();
    if (ctl->pcg_done) return;
    const float* res = !base ? f.res : sel < 0 ? pcg::cur_res(f, ctl) : sel ? f.res2 : f.res;
    const F2 acc = kb_up<kRz, kAll>(hw_blk(), c, f, sh, g, id, count, res, last, extra);
    if (kRz) block_store<kTileBlock>(hw_blk(), acc, part);
}

// CG on a coarsest level that is too large for the shared-memory tail (a
// grid whose sides stop halving early: 1000 x 600 ends at 125 x 75).  The
// arrays that every iteration reads move into shared memory, the most used
// first, as many as fit (`nsm` of them: directions, couplings, diagonal,
// residual); the rest stay in L2.  Mask and coefficients do not change
// during a solve: their copies start while the previous kernel drains.
constexpr size_t kCoarseSmemBudget = 220 * 1024;
inline __host__ __device__ size_t coarse_smem_bytes(uint32_t words, uint32_t padded, int nsm) {
    return 4ull * (words + size_t(nsm) * padded);
}
__global__ void __launch_bounds__(kTailThreads) k_coarse_solve(Level L, float* __restrict__ cs, float* __restrict__ cap,
                                                               float* __restrict__ cr, Ctl* __restrict__ ctl,
                                                               int exact, int nsm, ExitArgs exit) {
    extern __shared__ uint32_t sm[];
    CgArrays A{L.fluid, L.w, L.cells, L.diag, L.px, L.py, L.res, L.err, cs, cap, cr};
    float* f = reinterpret_cast<float*>(sm + L.words);
    auto copy = [&](float* dst, const float* src) {
        for (uint32_t i = threadIdx.x; i < L.padded; i += kTailThreads) cp_async4(dst + i, src + i);
        return dst;
    };
    if (nsm > 0) {
        for (uint32_t i = threadIdx.x; i < L.words; i += kTailThreads) cp_async4(sm + i, L.fluid + i);
        A.bits = sm;
        A.cs = f;
        if (nsm > 1) A.px = copy(f + L.padded, L.px);
        if (nsm > 2) A.py = copy(f + 2 * L.padded, L.py);
        if (nsm > 3) A.diag = copy(f + 3 * L.padded, L.diag);
        if (nsm > 4) A.cr = f + 4 * L.padded;
        if (nsm > 5) A.cap = f + 5 * L.padded;
    }
    pdl_wait();
    cp_async_wait_all();
    if (pcg::solve_over(ctl, exit, true)) return;
    __syncthreads();
    cta_coarse_cg(A, exact != 0);
}

__global__ void __launch_bounds__(kTailThreads) k_vcycle_tail(const __grid_constant__ TailParams tp, Ctl* ctl,
                                                              ExitArgs exit) {
    extern __shared__ uint32_t sm[];
    cta_tail_issue_coeffs(tp, sm);  // while the previous kernel drains
    pdl_wait();
    if (pcg::solve_over(ctl, exit, true)) {
        cp_async_wait_all();
        return;
    }
    cta_tail(tp, sm);
}

size_t tail_level_bytes(const Level& L) { return 4ull * (L.words + 6ull * L.padded); }

// ---- the V-cycle's phases over a batch of scenes (batch.h) ------------------
// Persistent CTAs walk the listed items of their gate; each runs the
// single-scene kernel's work for a few tiles of its scene, or (the base
// level in an iteration, whose blocks store partial sums) for the tiles of a
// group of the blocks of its scene's own launch.

__global__ void __launch_bounds__(kTileBlock, 4) k_bat_down(const BScene* __restrict__ tab, BListRef L, int lf,
                                                              int gate) {
    __shared__ tile::Shared sh;
    bat_for_items(L, kind_tiles(lf), gate == kGatePcg, [&](uint32_t sc, uint32_t item, Shape shp) {
        const BScene& S = tab[sc];
        const Ctl* ctl = S.ctl;
        if (!bat_gate(ctl, gate) || ctl->pcg_done) return;
        const uint32_t i0 = item * tile_chunk(shp), end = min(ctl->tile_count[lf], i0 + tile_chunk(shp));
        if (i0 >= end) return;
        const uint32_t id = S.lv[lf].tiles[i0];
        tile::DownRegs g;
        tile::down_load_const<true>(S.lv[lf], id, g);
        kb_down<true>(Blk{i0, 1u}, S.lv[lf], S.lv[lf + 1], sh, g, id, end,
                lf == 0 ? pcg::cur_res(S.lv[0], ctl) : S.lv[lf].res);
    });
}

__global__ void __launch_bounds__(kTileBlock, 4) k_bat_up(const BScene* __restrict__ tab, BListRef L, int lf,
                                                            int gate, int base) {
    __shared__ tile::Shared sh;
    bat_for_items(L, kind_tiles(lf), gate == kGatePcg, [&](uint32_t sc, uint32_t item, Shape shp) {
        const BScene& S = tab[sc];
        const Ctl* ctl = S.ctl;
        if (!bat_gate(ctl, gate) || ctl->pcg_done) return;
        const uint32_t i0 = item * tile_chunk(shp), end = min(ctl->tile_count[lf], i0 + tile_chunk(shp));
        if (i0 >= end) return;
        const uint32_t id = S.lv[lf].tiles[i0];
        const uint32_t last = base ? ctl->last_fluid : 0xFFFFFFFFu, extra = base ? ctl->pad_count : 0u;
        tile::UpRegs g;
        tile::up_load_const<true>(S.lv[lf], id, g);
        kb_up<false, true>(Blk{i0, 1u}, S.lv[lf + 1], S.lv[lf], sh, g, id, end,
                     base ? pcg::cur_res(S.lv[0], ctl) : S.lv[lf].res, last, extra);
    });
}

// The iteration's last V-cycle kernel (k_up<true>).
__global__ void __launch_bounds__(kTileBlock, 4) k_bat_up_rz(const BScene* __restrict__ tab, BListRef L) {
    __shared__ tile::Shared sh;
    bat_for_items(L, kKindTiles0, true, [&](uint32_t sc, uint32_t item, Shape shp) {
        const BScene& S = tab[sc];
        const Ctl* ctl = S.ctl;
        if (!bat_gate(ctl, kGatePcg) || ctl->pcg_done) return;
        const uint32_t count = ctl->tile_count[0], end = tile_group_end(S, item, shp);
        for (uint32_t b = item * shp.block_group; b < end; ++b) {
            const Blk bk{b, S.tgrid};
            tile::UpRegs g;
            const uint32_t id = b < count ? S.lv[0].tiles[b] : 0u;
            if (b < count) tile::up_load_const<true>(S.lv[0], id, g);
            const F2 acc = kb_up<true, true>(bk, S.lv[1], S.lv[0], sh, g, id, count, pcg::cur_res(S.lv[0], ctl),
                                       ctl->last_fluid, ctl->pad_count);
            block_store<kTileBlock>(bk, acc, bs_part_rz(S));
            __syncthreads();  // shared slots and the tile are reused by the next block
        }
    });
}

// The coarse tail (k_vcycle_tail): persistent CTAs take the listed scenes one
// at a time; the scene's tail parameters are copied into shared memory beside
// the levels.
__global__ void __launch_bounds__(kTailThreads) k_bat_tail(const BScene* __restrict__ tab, BListRef L, int gate) {
    __shared__ TailParams s_tp;
    extern __shared__ uint32_t sm[];
    pdl_wait();
    const uint32_t nact = L.p[0];
    for (uint32_t j = blockIdx.x; j < nact; j += gridDim.x) {
        const BScene& S = tab[L.scenes()[j]];
        if (!bat_gate(S.ctl, gate) || S.ctl->pcg_done) continue;
        const uint32_t* src = reinterpret_cast<const uint32_t*>(&S.tp);
        uint32_t* dst = reinterpret_cast<uint32_t*>(&s_tp);
        for (uint32_t i = threadIdx.x; i < sizeof(TailParams) / 4; i += blockDim.x) dst[i] = src[i];
        __syncthreads();
        cta_tail_issue_coeffs(s_tp, sm);
        cta_tail(s_tp, sm);
        __syncthreads();
    }
}

}  // namespace

void bat_down(const BatchRun& r, int l, int gate) {
    static const uint32_t g = persistent_grid(k_bat_down, kTileBlock, 0);
    launch(r.pdl, k_bat_down, g, kTileBlock, 0, r.st, r.tab, r.list[gate], l, gate);
}
void bat_up(const BatchRun& r, int l, int gate, int base) {
    static const uint32_t g = persistent_grid(k_bat_up, kTileBlock, 0);
    launch(r.pdl, k_bat_up, g, kTileBlock, 0, r.st, r.tab, r.list[gate], l, gate, base);
}
void bat_up_rz(const BatchRun& r) {
    static const uint32_t g = persistent_grid(k_bat_up_rz, kTileBlock, 0);
    launch(r.pdl, k_bat_up_rz, g, kTileBlock, 0, r.st, r.tab, r.list[kGatePcg]);
}
void bat_tail(const BatchRun& r, int gate) {
    const uint32_t g = r.nscenes < 152u ? r.nscenes : 152u;  // one CTA per SM holds the largest tail
    launch(r.pdl, k_bat_tail, g, kTailThreads, r.tail_smem, r.st, r.tab, r.list[gate], gate);
}
void bat_prepare_tail() {
    cudaFuncSetAttribute(k_bat_tail, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kTailSmemBudget));
}

// Choose the coarse levels that run in one CTA (all of them fit in shared memory).
void plan_vcycle(Scene& s) {
    s.tail_first = s.nlevels;  // none
    s.tail_smem = 0;
    if (s.nlevels < 2) return;
    const Level& C = s.lv[s.nlevels - 1];
    size_t bytes = 3ull * 4 * C.padded;  // coarse CG vectors
    for (int l = s.nlevels - 1; l >= 1; --l) {
        size_t b = bytes + tail_level_bytes(s.lv[l]);
        if (b > kTailSmemBudget) break;
        bytes = b;
        s.tail_first = l;
    }
    if (s.tail_first < s.nlevels) {
        s.tail_smem = bytes;
        cudaFuncSetAttribute(k_vcycle_tail, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kTailSmemBudget));
    }
    // (also where the tail holds every level: levels that a caller wrote take this kernel)
    cudaFuncSetAttribute(k_coarse_solve, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kCoarseSmemBudget));
    plan_vcycle_dsm(s);
}

// One V-cycle on s.stream: z = M^-1 r in lv[0].err.  Two kernels per level
// (k_down, k_up) above the levels that the distributed-shared-memory cluster
// or the shared-memory tail holds, or above the coarsest level's CG.
void enqueue_vcycle(Scene& s, bool base_done, const ExitArgs& exit_in, int sel) {
    cudaStream_t st = s.stream;
    Level* L = s.lv;
    const int last = s.nlevels - 1;
    const bool pdl = s.use_pdl;
    if (last < 1) {
        const uint32_t g = seg_grid(L[0].words);
        if (!base_done) launch(pdl, k_smooth, g, kSegBlock, 0, st, L[0], 0, s.ctl, 0, 1);
        launch(pdl, k_smooth, g, kSegBlock, 0, st, L[0], 0, s.ctl, 1, 1);
        launch(pdl, k_smooth, g, kSegBlock, 0, st, L[0], 0, s.ctl, 1, 0);
        launch(pdl, k_smooth, g, kSegBlock, 0, st, L[0], 0, s.ctl, 0, 0);
        return;
    }
    const bool dsm = s.use_dsm && s.dsm_first < s.dsm_tail && s.dsm_tail < s.nlevels;
    ExitArgs exit = exit_in;
    auto down = [&](int l) {
        launch(pdl, tile::reads_all(L[l]) ? k_down<true> : k_down<false>, tile_grid(L[l]) + (exit.on ? 1u : 0u), kTileBlock, 0, st, L[l], L[l + 1], l, s.ctl, exit);
        exit.on = 0;
    };
    if (!base_done) down(0);
    int l = 1;  // the deepest levels, from l on, run in one launch
    for (;; ++l) {
        if (dsm && l == s.dsm_first) {
            launch_vcycle_dsm(s, st, exit);
            break;
        }
        if (l == s.tail_first) {
            uint32_t off = 0;
            TailParams tp = make_tail_params(s, l, &off);
            launch(pdl, k_vcycle_tail, 1, kTailThreads, size_t(off) * 4, st, tp, s.ctl, exit);
            break;
        }
        if (l == last) {
            int nsm = 6;
            while (nsm > 0 && coarse_smem_bytes(L[l].words, L[l].padded, nsm) > kCoarseSmemBudget) --nsm;
            launch(pdl, k_coarse_solve, 1, kTailThreads, nsm ? coarse_smem_bytes(L[l].words, L[l].padded, nsm) : 0, st,
                   L[l], s.cg_s, s.cg_ap, s.cg_r, s.ctl, coarse_cg_exact(s) ? 1 : 0, nsm, exit);
            break;
        }
        down(l);
    }
    for (int k = l - 1; k >= 1; --k)
        launch(pdl, tile::reads_all(L[k]) ? k_up<false, true> : k_up<false, false>, tile_grid(L[k]), kTileBlock, 0, st, L[k + 1], L[k], k,
               static_cast<const Ctl*>(s.ctl), 0, static_cast<float2*>(nullptr), -1);
    const bool all = tile::reads_all(L[0]);
    auto up = base_done ? (all ? k_up<true, true> : k_up<true, false>) : all ? k_up<false, true> : k_up<false, false>;
    launch(pdl, up, tile_grid(L[0]), kTileBlock, 0, st, L[1], L[0], 0,
           static_cast<const Ctl*>(s.ctl), 1, part_rz(s), sel);
}

}  // namespace apic
