// tiles.cuh — the V-cycle's grid-wide sweeps and transfers, a 32 x 16 tile of
// cells per step, shared by the single-scene kernels (vcycle.cu, solver.cu)
// and the batch's (batch.h).
//
// Restates MultiGridLevel::smooth_level (src/apic.rs:471-535), restrict
// (:537-594) and prolongate (:596-616), and on the base level the update of
// an iteration of solve_pcg (:1907-1932).
//
// On a level that a whole grid works on, a phase of the V-cycle is a few
// hundred nanoseconds of work behind 4-5 us of launch and drain, and moves
// every array it reads through L2 once more.  So a level takes two kernels:
//   down: [PCG update;] red sweep, black sweep and restriction,
//   up:   prolongation, black sweep and red sweep [; r.z],
// each on a tile with a halo of two cells in shared memory.  A sweep of one
// colour needs the other colour one cell further out, so the halo's values
// are computed again by every tile that needs them (720 cells for 512, from
// the same inputs with the same operations: the same bits).  What a kernel
// writes is therefore never what another tile of it reads: the down kernel
// writes the smoothed error to `pre`, the up kernel reads that and writes
// `err`, and the update's residual alternates between two buffers.
//
// Cells outside the fluid mask hold zero error and zero couplings in the
// tile: where the reference skips a neighbour, a term of zero is added.
//
// 32 x 16 cells, 256 threads and four CTAs per SM: the 1024^2 scene's 550
// fluid tiles fill the chip once.  Bound by launch and drain (six kernels an
// iteration, eleven before) up to 2 M cells, by L2 and DRAM above.  A PCG
// iteration, separate sweeps -> tiles: 1024^2 87.1 -> 69.6 us, 4096^2
// 913 -> 699 us, 1000 x 600 (three levels) 119 -> 73 us.
#pragma once

#include <cuda_runtime.h>

#include "apic_device.cuh"
#include "apic_internal.h"
#include "vcycle_common.cuh"

namespace apic {
namespace tile {

static_assert(kTileBlock == kSegBlock, "block partials are formed by blocks of one size");
constexpr int kHalo = 2;
constexpr int kSX = int(kTileX) + 2 * kHalo, kSY = int(kTileY) + 2 * kHalo;
constexpr int kCells = kSX * kSY;                                 // 720
constexpr int kPer = (kCells + kTileBlock - 1) / kTileBlock;  // cells a thread stages: 3

struct Shared {
    float r[kCells], px[kCells], py[kCells], e[kCells];
};

// What a thread knows of one staged cell before the solve's vectors are read
// (mask and coefficients do not change during a solve).
struct Cell {
    uint32_t c;       // padded index
    float inv, px, py;
    bool fluid, red;
    bool own;         // one of the tile's 512 (not a halo cell), inside the grid
};

// kAll: a tile's reads go ahead of its mask bits (one latency instead of two);
// else only fluid cells are read.  On a level of more than kManyTiles tiles the
// bytes count: all / fluid cells only, an iteration: 216^2 32.7 / 33.5 us, 488^2
// 47.5 / 48.8, 1000 x 600 68.8 / 70.3; 2048^2 (noise) 241 / 230, 4096^2 675 / 633.
inline bool reads_all(const Level& L) { return L.ntiles <= kManyTiles; }

// (a raw index lies below 2^31, so y * w + x fits the 64-bit product)
// Raw indices run on past a row's end: the cell right of a row's last one is
// the first of the next row, as in the reference's flat index (raw +- 1).
template <bool kAll>
__device__ __forceinline__ void load_cell(const Level& L, int x0, int y0, int i, Cell& q) {
    const int idx = int(threadIdx.x) + i * kTileBlock;
    q.fluid = false;
    q.inv = q.px = q.py = 0.0f;
    q.c = L.w;
    q.red = q.own = false;
    if (idx >= kCells) return;
    const int sy = idx / kSX, sx = idx - sy * kSX;
    const int x = x0 + sx - kHalo, y = y0 + sy - kHalo;
    const long long raw = (long long)y * L.w + x;
    if (raw < 0 || raw >= (long long)L.cells) return;
    // colour by the cell's true coordinates (a wrapped cell lies one row on)
    const uint32_t wrapped = (x < 0 || x >= int(L.w)) ? L.w + 1u : 0u;
    q.red = ((uint32_t(x) + uint32_t(y) + wrapped) & 1u) == 0u;
    q.own = sx >= kHalo && sx < kSX - kHalo && sy >= kHalo && sy < kSY - kHalo && wrapped == 0u;
    q.c = uint32_t(raw) + L.w;
    if (kAll) {
        const float inv = L.inv_diag[q.c], px = L.px[q.c], py = L.py[q.c];
        q.fluid = bit_at(L.fluid, uint32_t(raw)) != 0;
        q.inv = q.fluid ? inv : 0.0f;
        q.px = q.fluid ? px : 0.0f;
        q.py = q.fluid ? py : 0.0f;
    } else {
        q.fluid = bit_at(L.fluid, uint32_t(raw)) != 0;
        if (!q.fluid) return;
        q.inv = L.inv_diag[q.c];
        q.px = L.px[q.c];
        q.py = L.py[q.c];
    }
}
// The staged cells but for the outermost ring: those the black sweep computes.
__device__ __forceinline__ bool inner(int i) {
    const int idx = int(threadIdx.x) + i * kTileBlock;
    const int sy = idx / kSX, sx = idx - sy * kSX;
    return sx >= 1 && sx < kSX - 1 && sy >= 1 && sy < kSY - 1;
}

// One SOR update (smooth_level :487-507) of a staged cell from the tile.
__device__ __forceinline__ float sor(const Shared& t, int idx, const Cell& q, float r, float old) {
    float sum = r;
    sum = __fmaf_rn(-q.px, t.e[idx + 1], sum);
    sum = __fmaf_rn(-q.py, t.e[idx + kSX], sum);
    sum = __fmaf_rn(-t.px[idx - 1], t.e[idx - 1], sum);
    sum = __fmaf_rn(-t.py[idx - kSX], t.e[idx - kSX], sum);
    const float gs = sum * q.inv;
    const float nv = old + (vc::kOmega * (gs - old));
    return q.inv == 0.0f ? old : nv;
}

__device__ __forceinline__ void tile_origin(const Level& L, uint32_t id, int& x0, int& y0) {
    x0 = int(id % L.tiles_x) * int(kTileX);
    y0 = int(id / L.tiles_x) * int(kTileY);
}

// The update of a PCG iteration that the base level's down kernel carries.
struct Update {
    const float* res;  // residual before
    const float* ap;
    const float* z;    // the preconditioned residual the search direction takes
    float* s;
    float* x;
    int x_padded;
    float* res_out;
};

// The vectors of a tile as the down kernel reads them: the staged cells'
// residual (and A s), this thread's own two cells (a pair in x: rows of 16
// pairs, two rows per warp, so a warp holds whole coarse cells).
struct DownRegs {
    Cell q[kPer];
    float r[kPer], ap[kPer];
    uint32_t c;      // padded index of the own pair's first cell
    bool own;        // the pair lies inside the grid
    float2 d, x, s, z;
};

template <bool kAll>
__device__ __forceinline__ void down_load_const(const Level& f, uint32_t id, DownRegs& g) {
    int x0, y0;
    tile_origin(f, id, x0, y0);
#pragma unroll
    for (int i = 0; i < kPer; ++i) load_cell<kAll>(f, x0, y0, i, g.q[i]);
    const int x = x0 + 2 * int(threadIdx.x & 15u), y = y0 + int(threadIdx.x >> 4);
    g.own = x < int(f.w) && y < int(f.h);
    g.c = g.own ? uint32_t(y) * f.w + uint32_t(x) + f.w : f.w;
    g.d = *reinterpret_cast<const float2*>(f.diag + g.c);  // (f.w is even: aligned)
}
template <bool kUpdate, bool kAll>
__device__ __forceinline__ void down_load(const Level& f, const float* res, const Update& u, DownRegs& g) {
#pragma unroll
    for (int i = 0; i < kPer; ++i) {  // (masked where they are used)
        const bool read = kAll || g.q[i].fluid;
        g.r[i] = read ? res[g.q[i].c] : 0.0f;
        if (kUpdate) g.ap[i] = read ? u.ap[g.q[i].c] : 0.0f;
    }
    if (kUpdate) {
        g.s = *reinterpret_cast<const float2*>(u.s + g.c);
        g.z = *reinterpret_cast<const float2*>(u.z + g.c);
        g.x = *reinterpret_cast<const float2*>(u.x + (u.x_padded ? g.c : g.c - f.w));
    }
}

// Red sweep from zero error, black sweep, restriction into c (whose first red
// sweep is formed where its residual is read).  kUpdate: first r = fma(-alpha, Ap, r), x += alpha s',
// s = s', and this thread's part of sum r^2 and max |r|.
template <bool kUpdate>
__device__ __forceinline__ void down_tile(Shared& t, const Level& f, const Level& c, uint32_t id, const DownRegs& g,
                                          const Update& u, float alpha, float beta, bool beta_valid, F2* acc,
                                          float* mx) {
    int x0, y0;
    tile_origin(f, id, x0, y0);
    float r[kPer];
#pragma unroll
    for (int i = 0; i < kPer; ++i) {
        const int idx = int(threadIdx.x) + i * kTileBlock;
        r[i] = !g.q[i].fluid ? 0.0f : kUpdate ? __fmaf_rn(-alpha, g.ap[i], g.r[i]) : g.r[i];
        if (idx >= kCells) continue;
        t.r[idx] = r[i];
        t.px[idx] = g.q[i].px;
        t.py[idx] = g.q[i].py;
        t.e[idx] = g.q[i].red ? vc::red_first(r[i], g.q[i].inv) : 0.0f;
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < kPer; ++i) {
        const int idx = int(threadIdx.x) + i * kTileBlock;
        if (idx >= kCells || !g.q[i].fluid || g.q[i].red || !inner(i)) continue;
        t.e[idx] = sor(t, idx, g.q[i], r[i], 0.0f);
    }
    __syncthreads();
    // own pair: residual of the smoothed error, and the coarse sum of the
    // 2 x 2 children (two here, two half a warp further on) in their order
    const int idx = (int(threadIdx.x >> 4) + kHalo) * kSX + 2 * int(threadIdx.x & 15u) + kHalo;
    const uint32_t raw = g.c - f.w;
    const uint32_t two = g.own ? (f.fluid[raw >> 5] >> (raw & 31u)) & 3u : 0u;  // (raw is even)
    const bool f0 = two & 1u, f1 = (two >> 1) & 1u;
    auto left_over = [&](int k, float d) {
        float ax = d * t.e[k];
        ax = ax + t.px[k] * t.e[k + 1];
        ax = ax + t.py[k] * t.e[k + kSX];
        ax = ax + t.px[k - 1] * t.e[k - 1];
        ax = ax + t.py[k - kSX] * t.e[k - kSX];
        return t.r[k] - ax;
    };
    const float d0 = left_over(idx, g.d.x), d1 = left_over(idx + 1, g.d.y);
    const float d2 = __shfl_down_sync(0xffffffffu, d0, 16), d3 = __shfl_down_sync(0xffffffffu, d1, 16);
    const uint32_t two_up = __shfl_down_sync(0xffffffffu, two, 16);
    if (two) {
        *reinterpret_cast<float2*>(f.pre + g.c) = make_float2(t.e[idx], t.e[idx + 1]);
        if (kUpdate) {
            const float r0 = t.r[idx], r1 = t.r[idx + 1];
            *reinterpret_cast<float2*>(u.res_out + g.c) = make_float2(r0, r1);
            const float s0 = beta_valid ? g.z.x + (beta * g.s.x) : g.s.x;
            const float s1 = beta_valid ? g.z.y + (beta * g.s.y) : g.s.y;
            *reinterpret_cast<float2*>(u.s + g.c) = make_float2(f0 ? s0 : g.s.x, f1 ? s1 : g.s.y);
            const float n0 = g.x.x + alpha * s0, n1 = g.x.y + alpha * s1;
            *reinterpret_cast<float2*>(u.x + (u.x_padded ? g.c : raw)) = make_float2(f0 ? n0 : g.x.x, f1 ? n1 : g.x.y);
            if (f0) {
                *mx = fmaxf(*mx, fabsf(r0));
                *acc = f2_add(*acc, f2_square(r0));
            }
            if (f1) {
                *mx = fmaxf(*mx, fabsf(r1));
                *acc = f2_add(*acc, f2_square(r1));
            }
        }
    }
    if ((threadIdx.x & 16u) == 0 && (two | two_up)) {
        float sum = 0.0f;
        sum = f0 ? sum + d0 : sum;
        sum = f1 ? sum + d1 : sum;
        sum = (two_up & 1u) ? sum + d2 : sum;
        sum = (two_up & 2u) ? sum + d3 : sum;
        const uint32_t cx = uint32_t(x0 >> 1) + (threadIdx.x & 15u), cy = uint32_t(y0 >> 1) + (threadIdx.x >> 5);
        const uint32_t cp = cy * c.w + cx + c.w;
        c.res[cp] = sum;
    }
}

// The staged cells' vectors as the up kernel reads them.
struct UpRegs {
    Cell q[kPer];
    float r[kPer], e[kPer];
};
template <bool kAll>
__device__ __forceinline__ void up_load_const(const Level& f, uint32_t id, UpRegs& g) {
    int x0, y0;
    tile_origin(f, id, x0, y0);
#pragma unroll
    for (int i = 0; i < kPer; ++i) load_cell<kAll>(f, x0, y0, i, g.q[i]);
}
// last / extra: the base level's last fluid cell receives the correction
// again per duplicate of the reference's padded list (:611-615).
template <bool kAll>
__device__ __forceinline__ void up_load(const Level& c, const Level& f, const float* res, uint32_t last,
                                        uint32_t extra, UpRegs& g) {
    float ec[kPer];
#pragma unroll
    for (int i = 0; i < kPer; ++i) {
        g.r[i] = g.e[i] = ec[i] = 0.0f;
        if (!kAll && !g.q[i].fluid) continue;
        uint32_t x, y;
        raw_xy(g.q[i].c - f.w, f.w, f.wshift, x, y);
        g.r[i] = res[g.q[i].c];
        g.e[i] = f.pre[g.q[i].c];
        ec[i] = c.err[(y >> 1) * c.w + (x >> 1) + c.w];
    }
#pragma unroll
    for (int i = 0; i < kPer; ++i) {
        if (!g.q[i].fluid) g.r[i] = g.e[i] = 0.0f;
        else g.e[i] = vc::prolonged(g.e[i], ec[i], g.q[i].c == last ? extra : 0u);
    }
}

// Prolongation (done by up_load), black sweep, red sweep; the final error of
// the tile's cells goes to f.err.  kRz: this thread's part of r.z.
template <bool kRz>
__device__ __forceinline__ void up_tile(Shared& t, const Level& f, const UpRegs& g, F2* acc) {
#pragma unroll
    for (int i = 0; i < kPer; ++i) {
        const int idx = int(threadIdx.x) + i * kTileBlock;
        if (idx >= kCells) continue;
        t.px[idx] = g.q[i].px;
        t.py[idx] = g.q[i].py;
        t.e[idx] = g.e[i];
    }
    __syncthreads();
    float z[kPer];
#pragma unroll
    for (int i = 0; i < kPer; ++i) {
        const int idx = int(threadIdx.x) + i * kTileBlock;
        z[i] = g.e[i];
        if (idx >= kCells || !g.q[i].fluid || g.q[i].red || !inner(i)) continue;
        z[i] = sor(t, idx, g.q[i], g.r[i], g.e[i]);
        t.e[idx] = z[i];
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < kPer; ++i) {
        const int idx = int(threadIdx.x) + i * kTileBlock;
        if (!g.q[i].fluid || !g.q[i].own) continue;
        if (g.q[i].red) z[i] = sor(t, idx, g.q[i], g.r[i], g.e[i]);
        f.err[g.q[i].c] = z[i];
        if (kRz) *acc = f2_add(*acc, g.r[i] * z[i]);
    }
}

}  // namespace tile
}  // namespace apic
