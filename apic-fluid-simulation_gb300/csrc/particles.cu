// particles.cu — particle <-> grid transfers on the GPU.
//
//   k_p2g_*     transfer_particles_to_grid's scatter (src/apic.rs:1237-1426):
//               APIC momentum and weight to the 4 u and 4 v faces, temporal
//               weight w_t (:1246-1248), cell-centred density (:1260-1284) and
//               the fluid bit of the particle's cell (:1358-1360).
//   k_g2p       transfer_grid_to_particles_and_advect (src/apic.rs:2057-2264)
//               over all padded lanes, fused with the max-speed reduction that
//               the next substep's CFL limit needs (get_max_particle_velocity,
//               :2412-2427) and a count of non-finite lanes.
//   k_vmax      stand-alone max speed (after the particle set is written).
//   k_permute   gather of the nine fields by the sorted `val` (:1068-1110).
//
// The reference sums P2G contributions with float CAS loops, so its sums come
// in thread-schedule order.  Here every face is summed by one thread in a fixed
// order (below).  Every other result of these kernels is computed lane by lane
// with the reference's operation order.
#include <cuda_runtime.h>

#include <algorithm>
#include <climits>

#include "apic_device.cuh"
#include "apic_internal.h"

namespace apic {
namespace {

// ---- P2G as an ordered gather ------------------------------------------------
//
// The reference adds every chunk's contributions to a face with a CAS loop
// (add_to_mac :296-344, add_to_vec_f32 :347-369): per chunk of 8 slots and per
// stencil corner k (bl, br, tl, tr), the lanes that hit the same face are
// summed in lane order and that group sum is added to the face.  Run on one
// thread, chunk after chunk, a face's sum is therefore the fold of its
// (chunk, corner) group sums in that order, which is the order the oracle
// defines.  Here every face is summed by one thread in exactly that order, so
// the result is bit-identical to the oracle and the same on every run:
//
//   k_p2g_bin_keys  key = the cell of the density stencil's base (cx0, cy0)
//                   for every particle; fluid bits (an OR: order-free)
//   radix sort      stable, so each cell's particles stay in slot order
//   k_p2g_bounds    each cell's run [lo, hi) in the sorted pairs
//   k_p2g_gather    per grid and 16 x 8 tile of faces: stage the
//                   contributions of the particles that reach the tile, in
//                   one run per stencil base and in slot order, then let each
//                   face merge the runs of its four bases and fold them in
//                   (chunk, corner, lane) order.
//
// Which cells can reach a face follows from the clamped index arithmetic
// (u_index / v_index, :1029-1041): the u stencil's rows equal the density
// stencil's rows and its columns start at cx0 or cx0 + 1; the v stencil's
// columns equal the density stencil's and its rows start at cy0 or cy0 + 1.
// So u face (i, j) gathers from cells x in [i-2, i], y in [j-1, j], v face
// (i, j) from x in [i-1, i], y in [j-2, j], and density cell (i, j) from
// x in [i-1, i], y in [j-1, j].  A particle whose corners fall outside those
// offsets (impossible by the arithmetic above, checked anyway) raises
// kStatusP2gLayout.
constexpr int kGatherTW = 32, kGatherTH = 8;           // tile of cells (cell order), one thread per cell
constexpr int kGatherThreads = kGatherTW * kGatherTH;
constexpr int kRegionW = kGatherTW + 2, kRegionH = kGatherTH + 2;

enum { kGridU = 0, kGridV = 1, kGridD = 2 };

// Exclusive scan over the threads of a block (blockDim.x a multiple of 32).
__device__ __forceinline__ uint32_t block_exclusive_scan_u32(uint32_t v, uint32_t* total) {
    __shared__ uint32_t sw[32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) sw[warp] = x;
    __syncthreads();
    if (warp == 0) {
        uint32_t t = lane < int(blockDim.x / 32) ? sw[lane] : 0u;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, t, o);
            if (lane >= o) t += y;
        }
        sw[lane] = t;
    }
    __syncthreads();
    const uint32_t pre = warp > 0 ? sw[warp - 1] : 0u;
    *total = sw[blockDim.x / 32 - 1];
    __syncthreads();
    return pre + x - v;
}

// Four particles per thread with 16-byte loads and stores (the arrays hold
// npad, a multiple of 8, lanes; keys of lanes n .. npad-1 are never read).
__global__ void __launch_bounds__(256) k_p2g_bin_keys(const PartPtrs* __restrict__ pp, uint32_t n, int W, int H,
                                                      CellSize cs, uint32_t* __restrict__ keys,
                                                      uint32_t* __restrict__ fluid, uint32_t* __restrict__ head,
                                                      uint32_t* __restrict__ lo, uint32_t* __restrict__ hi) {
    pdl_wait();
    clear_sort_head(head);
    // the cells' runs, empty until k_p2g_bounds (a grid with particles has even
    // sides, so whole vectors)
    for (uint32_t c = blockIdx.x * blockDim.x + threadIdx.x; c < uint32_t(W) * uint32_t(H) / 4u; c += gridDim.x * blockDim.x) {
        reinterpret_cast<uint4*>(lo)[c] = make_uint4(0u, 0u, 0u, 0u);
        reinterpret_cast<uint4*>(hi)[c] = make_uint4(0u, 0u, 0u, 0u);
    }
    const uint32_t i0 = 4u * (blockIdx.x * blockDim.x + threadIdx.x);
    const bool any = i0 < n;
    float4 px = make_float4(0.0f, 0.0f, 0.0f, 0.0f), py = px;
    if (any) {
        px = *reinterpret_cast<const float4*>(pp->f[PX] + i0);
        py = *reinterpret_cast<const float4*>(pp->f[PY] + i0);
    }
    const float xs[4] = {px.x, px.y, px.z, px.w}, ys[4] = {py.x, py.y, py.z, py.w};
    uint32_t k[4];
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const bool live = i0 + uint32_t(q) < n;
        const float gx = over_dx(xs[q], cs), gy = over_dx(ys[q], cs);
        const int cx0 = max(min(trunc_x86(floorf(gx - 0.5f)), W - 1), 0);
        const int cy0 = max(min(trunc_x86(floorf(gy - 0.5f)), H - 1), 0);
        k[q] = uint32_t(cy0) * uint32_t(W) + uint32_t(cx0);
        // the particle's own cell (:1358-1360); one OR per mask word the warp touches
        const int fx = trunc_x86(fmax_x86(fmin_x86(gx, float(W) - 1.0f), 0.0f));
        const int fy = trunc_x86(fmax_x86(fmin_x86(gy, float(H) - 1.0f), 0.0f));
        const uint32_t fi = uint32_t(fy * W + fx);
        const uint32_t word = live ? fi >> 5 : 0xFFFFFFFFu, bit = live ? 1u << (fi & 31u) : 0u;
        const uint32_t peers = __match_any_sync(0xffffffffu, word);
        const uint32_t m = __reduce_or_sync(peers, bit);
        if (live && (peers & ((1u << lane) - 1u)) == 0) atomicOr(fluid + word, m);
    }
    if (any) *reinterpret_cast<uint4*>(keys + i0) = make_uint4(k[0], k[1], k[2], k[3]);
}

__global__ void __launch_bounds__(256) k_p2g_bounds(const uint32_t* __restrict__ keys, uint32_t n,
                                                    uint32_t* __restrict__ lo, uint32_t* __restrict__ hi,
                                                    uint32_t cells, uint32_t* __restrict__ status) {
    pdl_wait();
    const uint32_t j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= n) return;
    const uint32_t k = keys[j];
    if (!APIC_IN_BOUNDS(k, cells, status)) return;
    if (j == 0 || keys[j - 1] != k) lo[k] = j;
    if (j == n - 1 || keys[j + 1] != k) hi[k] = j + 1;
}

// One particle's contributions to one grid: per corner k the value and weight
// (value unused for the density) and, per relative face position q of the
// face that gathers it (q = ry * nx + rx, offsets from the particle's density
// base cell), a 4-bit mask of the corners that land there.
struct P2gRec {
    uint32_t code;
    float val[4], w[4];
};

// The quantities of one particle that every grid's contributions share:
// grid position and temporal weight (:1246-1256).
struct P2gBase {
    float gx, gy, wt;
};
__device__ __forceinline__ P2gBase p2g_base(const PartPtrs* __restrict__ pp, uint32_t slot, CellSize cs,
                                            float prev_dt) {
    const float tr = pp->f[TR][slot];
    const float tau = (-tr) / prev_dt;
    P2gBase b;
    b.wt = temporal_w(tau);
    b.gx = over_dx(pp->f[PX][slot], cs);
    b.gy = over_dx(pp->f[PY][slot], cs);
    return b;
}

__device__ __forceinline__ bool p2g_record(const PartPtrs* __restrict__ pp, uint32_t slot, const P2gBase& b, int grid,
                                           int W, int H, float dx, P2gRec& r) {
    const float gx = b.gx, gy = b.gy, wt = b.wt;
    const int cx0 = max(min(trunc_x86(floorf(gx - 0.5f)), W - 1), 0);
    const int cy0 = max(min(trunc_x86(floorf(gy - 0.5f)), H - 1), 0);
    int xs[2], ys[2], nx, ny;
    if (grid == kGridD) {
        // cell-centred density stencil (:1260-1284)
        const float cgx = gx - 0.5f, cgy = gy - 0.5f;
        const float cbx = floorf(cgx), cby = floorf(cgy);
        const float ctx = cgx - cbx, cty = cgy - cby;
        r.w[0] = ((1.0f - ctx) * (1.0f - cty)) * wt;
        r.w[1] = (ctx * (1.0f - cty)) * wt;
        r.w[2] = ((1.0f - ctx) * cty) * wt;
        r.w[3] = (ctx * cty) * wt;
        const int tbx = trunc_x86(cbx), tby = trunc_x86(cby);
        xs[0] = max(min(tbx, W - 1), 0); xs[1] = max(min(tbx + 1, W - 1), 0);
        ys[0] = max(min(tby, H - 1), 0); ys[1] = max(min(tby + 1, H - 1), 0);
        nx = 2; ny = 2;
    } else if (grid == kGridU) {
        Stencil su;
        u_stencil(gx, gy, W, H, dx, su);
        const float vx = pp->f[VX][slot], cux = pp->f[CUX][slot], cuy = pp->f[CUY][slot];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            r.w[k] = su.w[k] * wt;
            r.val[k] = (vx + cux * su.ox[k] + cuy * su.oy[k]) * r.w[k];
        }
        const int ix = trunc_x86(floorf(gx)), iy = trunc_x86(floorf(gy - 0.5f));
        xs[0] = max(min(ix, W), 0); xs[1] = max(min(ix + 1, W), 0);
        ys[0] = max(min(iy, H - 1), 0); ys[1] = max(min(iy + 1, H - 1), 0);
        nx = 3; ny = 2;
    } else {
        Stencil sv;
        v_stencil(gx, gy, W, H, dx, sv);
        const float vy = pp->f[VY][slot], cvx = pp->f[CVX][slot], cvy = pp->f[CVY][slot];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            r.w[k] = sv.w[k] * wt;
            r.val[k] = (vy + cvx * sv.ox[k] + cvy * sv.oy[k]) * r.w[k];
        }
        const int jx = trunc_x86(floorf(gx - 0.5f)), jy = trunc_x86(floorf(gy));
        xs[0] = max(min(jx, W - 1), 0); xs[1] = max(min(jx + 1, W - 1), 0);
        ys[0] = max(min(jy, H), 0); ys[1] = max(min(jy + 1, H), 0);
        nx = 2; ny = 3;
    }
    uint32_t code = 0;
    bool ok = true;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const int rx = xs[k & 1] - cx0, ry = ys[k >> 1] - cy0;
        if (rx < 0 || rx >= nx || ry < 0 || ry >= ny) {
            ok = false;
            continue;
        }
        code |= (1u << k) << (4 * (ry * nx + rx));
    }
    r.code = code;
    return ok;
}

// A particle whose three stencils lie inside their grids, so that no index is
// clamped: it reaches four different nodes of each grid, and its u base is
// its density base or the column after it, its v base that or the row above.
__device__ __forceinline__ bool p2g_inside(const P2gBase& b, int W, int H) {
    const float cx = floorf(b.gx - 0.5f), cy = floorf(b.gy - 0.5f);
    return cx >= 0.0f && cx <= float(W - 2) && cy >= 0.0f && cy <= float(H - 2);
}

struct GatherOut {
    float *acc_u, *acc_uw, *acc_v, *acc_vw, *dens;
};

// ---- one face from global memory (any particles) ----
// The face's cells' runs are merged by slot and each particle's record is
// computed when its turn comes.  For tiles whose particles do not fit the
// stage even for one row of faces, and for particles outside the inner cells
// (the first substep after such a set was written: advection keeps particles
// 1.001 cells from the walls).
__device__ __noinline__ void fold_face_global(const PartPtrs* __restrict__ pp, const uint32_t* __restrict__ vals,
                                              const uint32_t* __restrict__ lo, const uint32_t* __restrict__ hi,
                                              int grid, int x, int y, int W, int H, CellSize cs, float prev_dt,
                                              uint32_t* status, uint32_t n, uint32_t npad, float& out_v,
                                              float& out_w) {
    // the cell of run r lies at offset (r % nx, r / nx) below and to the left,
    // the index by which p2g_record codes the corners
    const int nx = grid == kGridU ? 3 : 2, nr = grid == kGridD ? 4 : 6;
    uint32_t b[6], e[6], head[6];
    auto slot_at = [&](uint32_t p) {
        const uint32_t sl = APIC_IN_BOUNDS(p, n, status) ? vals[p] : 0u;
        return APIC_IN_BOUNDS(sl, npad, status) ? sl : 0u;
    };
#pragma unroll
    for (int r = 0; r < 6; ++r) {
        const int cx = x - r % nx, cy = y - r / nx;
        b[r] = e[r] = 0;
        if (r < nr && cx >= 0 && cx < W && cy >= 0 && cy < H) {
            const uint32_t c = uint32_t(cy) * uint32_t(W) + uint32_t(cx);
            b[r] = lo[c];
            e[r] = hi[c];
        }
        head[r] = b[r] < e[r] ? slot_at(b[r]) : 0xFFFFFFFFu;
    }
    // per chunk and corner the lanes' contributions in lane order; at the end
    // of the chunk the corners' sums are added to the face in corner order
    float av = 0.0f, aw = 0.0f, gv[4] = {0.0f, 0.0f, 0.0f, 0.0f}, gw[4] = {0.0f, 0.0f, 0.0f, 0.0f};
    uint32_t chunk = 0xFFFFFFFFu;
    bool bad = false;
    auto flush = [&] {
#pragma unroll
        for (int k = 0; k < 4; ++k) {  // (no sum here is ever -0: a corner without terms adds nothing)
            av = av + gv[k];
            aw = aw + gw[k];
            gv[k] = gw[k] = 0.0f;
        }
    };
    for (;;) {
        uint32_t slot = head[0];
        int m = 0;
#pragma unroll
        for (int r = 1; r < 6; ++r)
            if (head[r] < slot) { slot = head[r]; m = r; }
        if (slot == 0xFFFFFFFFu) break;
#pragma unroll
        for (int r = 0; r < 6; ++r)
            if (r == m) {
                ++b[r];
                head[r] = b[r] < e[r] ? slot_at(b[r]) : 0xFFFFFFFFu;
            }
        P2gRec rec;
        if (!p2g_record(pp, slot, p2g_base(pp, slot, cs, prev_dt), grid, W, H, cs.dx, rec)) bad = true;
        const uint32_t hit = (rec.code >> (4 * m)) & 0xFu;
        if (!hit) continue;
        if ((slot >> 3) != chunk) {
            flush();
            chunk = slot >> 3;
        }
#pragma unroll
        for (int k = 0; k < 4; ++k)
            if (hit & (1u << k)) {
                if (grid != kGridD) gv[k] = gv[k] + rec.val[k];
                gw[k] = gw[k] + rec.w[k];
            }
    }
    flush();
    if (bad) atomicOr(status, kStatusP2gLayout);
    out_v = av;
    out_w = aw;
}

// ---- the gather in the reference's order ----
// One CTA per grid (u, v, density) and 16 x 8 tile of its faces.  A particle
// inside the grids reaches a face through one corner, given by the offset of
// its stencil base from the face, so a face's terms are those of four runs of
// particles, one per base, corner k of the run at base (-(k & 1), -(k >> 1)).
// The sorted pairs give the runs of the density bases; the u base is that or
// the next column (s = 1), the v base that or the next row, so a u or v run is
// the s = 0 particles of one cell and the s = 1 particles of the cell before it
// on the line (a row of cells for u, a column for v).  A particle's place in
// its run is a count of s bits in its own cell and a binary search by slot in
// the other.  Within a run the chunk never falls, so merging the four heads by
// (chunk, corner) yields the terms group by group in the reference's order:
// some 40 instructions a term.  The stage holds two words and four (value,
// weight) pairs a particle; a tile whose particles exceed it is done in bands
// of rows.
//
// What bounds it is issue slots and the latency of the field loads together: a
// particle's place and record (about 250 instructions a grid, on 1.2-1.3 times
// the particles for the halo) and the merge (12 terms a particle).  Three CTAs
// an SM are 24 warps; half of a CTA's threads have no face, they help to stage.
// 4.6 million particles, nine a cell: 655 -> 392 us against one CTA per 32 x 8
// tile and all grids whose faces merged six runs of unsplit cells; the stage
// of a 64 x 64 grid, where 96 CTAs run instead of 16, 143 -> 42 us.
constexpr int kFaceTW = 16, kFaceTH = 8, kFaceThreads = 256;
constexpr int kFaceCap = 1760;  // staged particles (three CTAs per SM)
constexpr size_t kFaceSmem = size_t(kFaceCap) * (4 + 4 + 4 * 8 + 1);
constexpr int kFaceRegion = (kFaceTW + 1) * (kFaceTH + 2);  // cells, of v the most (u: 18 x 9)
static_assert(kFaceRegion >= (kFaceTW + 2) * (kFaceTH + 1) && kFaceRegion <= kFaceThreads, "one thread per cell");

struct FaceShared {
    uint32_t sums[kFaceThreads / 32];
    uint32_t cnt[kFaceRegion], glo[kFaceRegion];  // particles of each cell, first sorted pair (row by row)
    uint32_t off[kFaceRegion + 1];                // the band's cells along its lines: first place,
    uint32_t from[kFaceRegion];                   // sorted pair of place 0 of a row that starts with the cell,
    uint32_t one[kFaceRegion + 1];                // and how many places before it hold s = 1
    uint32_t bits[kFaceCap / 32 + 1], before[kFaceCap / 32 + 1];  // s of 32 places, s = 1 before them
    uint32_t row_n[kFaceTH + 2];                  // particles of each row
};

// The sum over the block, to every thread.
__device__ __forceinline__ uint32_t block_sum(uint32_t v, uint32_t* sums) {
    const uint32_t lane = threadIdx.x & 31u;
    v = __reduce_add_sync(0xffffffffu, v);
    if (lane == 0) sums[threadIdx.x / 32u] = v;
    __syncthreads();
    return __reduce_add_sync(0xffffffffu, lane < kFaceThreads / 32 ? sums[lane] : 0u);
}

template <int G>
__device__ __forceinline__ void gather_tile(const PartPtrs* __restrict__ pp, const uint32_t* __restrict__ vals,
                                            const uint32_t* __restrict__ lo, const uint32_t* __restrict__ hi, int W,
                                            int H, CellSize cs, Ctl* __restrict__ ctl, float* __restrict__ out_v,
                                            float* __restrict__ out_w, uint32_t n, uint32_t npad, FaceShared& sh,
                                            unsigned char* smem) {
    constexpr int HX = G == kGridU ? 2 : 1, HY = G == kGridV ? 2 : 1;
    constexpr int RW = kFaceTW + HX, RH = kFaceTH + HY;
    const int FW = G == kGridU ? W + 1 : W, FH = G == kGridV ? H + 1 : H;
    float2* rec = reinterpret_cast<float2*>(smem);                         // [4][kFaceCap]
    uint32_t* cells = reinterpret_cast<uint32_t*>(rec + 4 * kFaceCap);     // by cell: slot | s << 31
    uint32_t* runs = cells + kFaceCap;                                     // by run: slot & ~7 | last of its run
    uint8_t* cell_of = reinterpret_cast<uint8_t*>(runs + kFaceCap);
    const float *fpx = pp->f[PX], *fpy = pp->f[PY], *ftr = pp->f[TR];
    const float* fvel = pp->f[G == kGridU ? VX : VY];
    const float *fgx = pp->f[G == kGridU ? CUX : CVX], *fgy = pp->f[G == kGridU ? CUY : CVY];
    const int x0 = blockIdx.x * kFaceTW, y0 = blockIdx.y * kFaceTH;
    if (x0 >= FW || y0 >= FH) return;
    const int rx0 = x0 - HX, ry0 = y0 - HY;
    const uint32_t t = threadIdx.x, lane = t & 31u, warp = t >> 5;
    const int tx = int(t) % kFaceTW, ty = int(t) / kFaceTW;
    const int fx = x0 + tx, fy = y0 + ty;
    const bool face = ty < kFaceTH && fx < FW && fy < FH;
    const uint32_t f = uint32_t(fy) * uint32_t(FW) + uint32_t(fx);
    const float prev_dt = ctl->prev_dt;

    // the region's cells
    uint32_t cnt = 0;
    if (t < RW * RH) {
        const int x = rx0 + int(t) % RW, y = ry0 + int(t) / RW;
        uint32_t gl = 0, gh = 0;
        if (x >= 0 && x < W && y >= 0 && y < H) {
            const uint32_t c = uint32_t(y) * uint32_t(W) + uint32_t(x);
            gl = lo[c];
            gh = hi[c];
            if (!APIC_IN_BOUNDS(gh, uint64_t(n) + 1u, &ctl->status)) gh = gl;
        }
        cnt = gh - gl;
        sh.cnt[t] = cnt;
        sh.glo[t] = gl;
    }
    const uint32_t total = block_sum(cnt, sh.sums);
    if (total == 0) {
        if (face) {
            if (G != kGridD) out_v[f] = 0.0f;
            out_w[f] = 0.0f;
        }
        return;
    }
    // the tallest band whose every region fits the stage (0: none)
    uint32_t band = kFaceTH;
    if (total > uint32_t(kFaceCap)) {
        for (uint32_t r = warp; r < RH; r += kFaceThreads / 32) {
            const uint32_t sum = __reduce_add_sync(0xffffffffu, lane < RW ? sh.cnt[r * RW + lane] : 0u);
            if (lane == 0) sh.row_n[r] = sum;
        }
        __syncthreads();
        for (band = kFaceTH / 2; band >= 1; band >>= 1) {
            bool fits = true;
            for (uint32_t r0 = 0; r0 < uint32_t(kFaceTH); r0 += band) {
                uint32_t sum = 0;
                for (uint32_t r = r0; r < r0 + band + HY; ++r) sum += sh.row_n[r];
                fits = fits && sum <= uint32_t(kFaceCap);
            }
            if (fits) break;
        }
    }

    for (uint32_t r0 = 0; r0 < uint32_t(kFaceTH); r0 += band ? band : uint32_t(kFaceTH)) {
        const uint32_t nrow = (band ? band : uint32_t(kFaceTH)) + HY;  // region rows [r0, r0 + nrow)
        const bool mine = face && uint32_t(ty) >= r0 && uint32_t(ty) < r0 + nrow - HY;
        // cell (x, y) of the band's region along the lines
        auto at = [&](uint32_t x, uint32_t y) { return G == kGridV ? x * nrow + y : y * RW + x; };
        bool odd = band == 0;
        uint32_t P = 0;
        if (band) {
            const uint32_t x = G == kGridV ? t / nrow : t % RW, y = G == kGridV ? t % nrow : t / RW;
            const bool in = t < RW * nrow;
            const uint32_t mine_n = in ? sh.cnt[(r0 + y) * RW + x] : 0u;
            const uint32_t ex = block_exclusive_scan_u32(mine_n, &P);
            if (in) {
                sh.off[t] = ex;
                sh.from[t] = sh.glo[(r0 + y) * RW + x] - ex;
                for (uint32_t k = 0; k < mine_n; ++k) cell_of[ex + k] = uint8_t(t);
            }
            if (t == 0) sh.off[RW * nrow] = P;
            if (P == 0) {  // (the same for every thread)
                if (mine) {
                    if (G != kGridD) out_v[f] = 0.0f;
                    out_w[f] = 0.0f;
                }
                __syncthreads();
                continue;
            }
            __syncthreads();
            // each cell's particles in slot order, with s; three a thread in flight
            for (uint32_t p0 = t; p0 - lane < P; p0 += 3 * kFaceThreads) {
                uint32_t slot[3];
                float px[3], py[3];
#pragma unroll
                for (int i = 0; i < 3; ++i) {
                    const uint32_t p = p0 + uint32_t(i) * kFaceThreads;
                    slot[i] = 0;
                    if (p < P) {
                        const uint32_t g = sh.from[cell_of[p]] + p;
                        if (APIC_IN_BOUNDS(g, n, &ctl->status)) slot[i] = vals[g];
                        if (!APIC_IN_BOUNDS(slot[i], npad, &ctl->status)) slot[i] = 0;
                    }
                }
#pragma unroll
                for (int i = 0; i < 3; ++i) {
                    px[i] = fpx[slot[i]];
                    py[i] = fpy[slot[i]];
                }
#pragma unroll
                for (int i = 0; i < 3; ++i) {
                    const uint32_t p = p0 + uint32_t(i) * kFaceThreads;
                    if (p - lane >= P) break;  // (warps as a whole)
                    const float gx = over_dx(px[i], cs), gy = over_dx(py[i], cs);
                    odd = odd || (p < P && !p2g_inside(P2gBase{gx, gy, 0.0f}, W, H));
                    const bool s = p < P && (G == kGridU   ? floorf(gx) != floorf(gx - 0.5f)
                                             : G == kGridV ? floorf(gy) != floorf(gy - 0.5f)
                                                           : false);
                    if (p < P) cells[p] = slot[i] | (s ? 0x80000000u : 0u);
                    if (G != kGridD) {
                        const uint32_t b = __ballot_sync(0xffffffffu, s);
                        if (lane == 0) sh.bits[p / 32u] = b;
                    }
                }
            }
            odd = __syncthreads_or(odd) != 0;
        }
        if (odd) {
            float v, w;
            if (mine) {
                fold_face_global(pp, vals, lo, hi, G, fx, fy, W, H, cs, prev_dt, &ctl->status, n, npad, v, w);
                if (G != kGridD) out_v[f] = v;
                out_w[f] = w;
            }
            __syncthreads();
            continue;
        }
        auto ones = [&](uint32_t p) {  // places before p with s = 1
            return sh.before[p / 32u] + uint32_t(__popc(sh.bits[p / 32u] & ((1u << (p % 32u)) - 1u)));
        };
        if (G != kGridD) {
            // the count of s = 1 before every word of places (each warp for
            // itself), then before every cell
            {
                const uint32_t words = (P + 31u) / 32u;
                const uint32_t a = 2u * lane < words ? __popc(sh.bits[2u * lane]) : 0u;
                const uint32_t b = 2u * lane + 1u < words ? __popc(sh.bits[2u * lane + 1u]) : 0u;
                uint32_t sum = a + b;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const uint32_t up = __shfl_up_sync(0xffffffffu, sum, o);
                    if (lane >= uint32_t(o)) sum += up;
                }
                if (2u * lane <= words) sh.before[2u * lane] = sum - a - b;
                if (2u * lane + 1u <= words) sh.before[2u * lane + 1u] = sum - b;
                __syncwarp();
            }
            if (t <= RW * nrow) sh.one[t] = ones(sh.off[t]);
            __syncthreads();
        }
        // the run of base c: the s = 1 particles of the cell before it on the
        // line and the s = 0 particles of cell c, in slot order (the runs that
        // a line starts or ends with reach no face of the tile)
        auto run_begin = [&](uint32_t c) { return G == kGridD ? sh.off[c] : sh.off[c] - (sh.one[c] - sh.one[c - 1]); };
        auto run_end = [&](uint32_t c) { return G == kGridD ? sh.off[c + 1] : sh.off[c + 1] - (sh.one[c + 1] - sh.one[c]); };
        // (the next particle's fields are on their way while this one is placed)
        struct Fields {
            uint32_t own;
            float px, py, tr, vel, gx, gy;
        };
        auto load = [&](uint32_t p) {
            Fields r;
            r.own = p < P ? cells[p] : 0u;
            const uint32_t slot = r.own & 0x7FFFFFFFu;
            r.px = fpx[slot];
            r.py = fpy[slot];
            r.tr = ftr[slot];
            if (G != kGridD) {
                r.vel = fvel[slot];
                r.gx = fgx[slot];
                r.gy = fgy[slot];
            }
            return r;
        };
        Fields ahead = load(t);
        for (uint32_t p = t; p < P; p += kFaceThreads) {
            const Fields cur = ahead;
            ahead = load(p + kFaceThreads);
            const uint32_t slot = cur.own & 0x7FFFFFFFu, s = cur.own >> 31;
            P2gBase b;
            b.gx = over_dx(cur.px, cs);
            b.gy = over_dx(cur.py, cs);
            uint32_t c = cell_of[p], place = p;
            if (G != kGridD) {
                const uint32_t pos = G == kGridU ? uint32_t(int(floorf(b.gx - 0.5f)) - rx0)
                                                 : uint32_t(int(floorf(b.gy - 0.5f)) - ry0) - r0;
                const uint32_t len = G == kGridU ? uint32_t(RW) : nrow;
                if (pos + s == 0u || pos + s == len) continue;  // (a run that no face reads)
                // its place: the cell's earlier particles with the same s, and the
                // lower slots of the run's other cell with the other s
                const uint32_t o = s ? c + 1u : c - 1u, ob = sh.off[o];
                uint32_t at2 = ob, len2 = sh.off[o + 1] - ob;
                while (len2 > 0) {
                    const uint32_t half = len2 >> 1;
                    const bool below = (cells[at2 + half] & 0x7FFFFFFFu) < slot;
                    at2 = below ? at2 + half + 1u : at2;
                    len2 = below ? len2 - half - 1u : half;
                }
                const uint32_t k1 = ones(p) - sh.one[c], o1 = ones(at2) - sh.one[o];
                place = s ? k1 + (at2 - ob) - o1 : p - sh.off[c] - k1 + o1;
                c += s;
                place += run_begin(c);
            }
            runs[place] = (slot & ~7u) | (place + 1u == run_end(c) ? 1u : 0u);
            b.wt = temporal_w((-cur.tr) / prev_dt);
            if (G == kGridD) {
                const float cgx = b.gx - 0.5f, cgy = b.gy - 0.5f;
                const float ctx = cgx - floorf(cgx), cty = cgy - floorf(cgy);
                float* rw = reinterpret_cast<float*>(rec);
                rw[0 * kFaceCap + place] = ((1.0f - ctx) * (1.0f - cty)) * b.wt;
                rw[1 * kFaceCap + place] = (ctx * (1.0f - cty)) * b.wt;
                rw[2 * kFaceCap + place] = ((1.0f - ctx) * cty) * b.wt;
                rw[3 * kFaceCap + place] = (ctx * cty) * b.wt;
            } else {
                Stencil st;
                if (G == kGridU) u_stencil(b.gx, b.gy, W, H, cs.dx, st);
                else v_stencil(b.gx, b.gy, W, H, cs.dx, st);
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const float w = st.w[k] * b.wt;
                    rec[k * kFaceCap + place] = make_float2((cur.vel + cur.gx * st.ox[k] + cur.gy * st.oy[k]) * w, w);
                }
            }
        }
        __syncthreads();
        if (mine) {
            uint32_t head[4], pos[4];
#pragma unroll
            for (uint32_t k = 0; k < 4; ++k) {
                const uint32_t c = at(uint32_t(tx) + HX - (k & 1u), uint32_t(ty) - r0 + HY - (k >> 1));
                const uint32_t b = run_begin(c);
                pos[k] = b;
                head[k] = b < run_end(c) ? runs[b] | (k << 1) : 0xFFFFFFFFu;
            }
            float av = 0.0f, aw = 0.0f, gv = 0.0f, gw = 0.0f;
            uint32_t group = 0xFFFFFFFFu;
            for (;;) {
                const uint32_t best = min(min(head[0], head[1]), min(head[2], head[3]));
                if (best == 0xFFFFFFFFu) break;
                const uint32_t m = (best >> 1) & 3u;
                const uint32_t p = m & 2u ? (m & 1u ? pos[3] : pos[2]) : (m & 1u ? pos[1] : pos[0]);
                const uint32_t next = best & 1u ? 0xFFFFFFFFu : runs[p + 1u] | (best & 6u);
                float2 r;
                if (G == kGridD) r = make_float2(0.0f, reinterpret_cast<const float*>(rec)[m * kFaceCap + p]);
                else r = rec[m * kFaceCap + p];
                // a new (chunk, corner) group: the one before goes to the face
                // (no sum here is ever -0, so adding an empty one changes nothing)
                const bool fresh = (best >> 1) != group;
                group = best >> 1;
                if (G != kGridD) {
                    av = fresh ? av + gv : av;
                    gv = fresh ? r.x : gv + r.x;
                }
                aw = fresh ? aw + gw : aw;
                gw = fresh ? r.y : gw + r.y;
#pragma unroll
                for (uint32_t k = 0; k < 4; ++k) {
                    head[k] = k == m ? next : head[k];
                    pos[k] = k == m ? p + 1u : pos[k];
                }
            }
            if (G != kGridD) out_v[f] = av + gv;
            out_w[f] = aw + gw;
        }
        __syncthreads();
    }
}

__global__ void __launch_bounds__(kFaceThreads, 3) k_p2g_gather(const PartPtrs* __restrict__ pp,
                                                                const uint32_t* __restrict__ vals,
                                                                const uint32_t* __restrict__ lo,
                                                                const uint32_t* __restrict__ hi, int W, int H,
                                                                CellSize cs, Ctl* __restrict__ ctl, GatherOut o,
                                                                uint32_t n, uint32_t npad) {
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ FaceShared sh;
    pdl_wait();
    if (blockIdx.z == kGridU)
        gather_tile<kGridU>(pp, vals, lo, hi, W, H, cs, ctl, o.acc_u, o.acc_uw, n, npad, sh, smem);
    else if (blockIdx.z == kGridV)
        gather_tile<kGridV>(pp, vals, lo, hi, W, H, cs, ctl, o.acc_v, o.acc_vw, n, npad, sh, smem);
    else
        gather_tile<kGridD>(pp, vals, lo, hi, W, H, cs, ctl, nullptr, o.dens, n, npad, sh, smem);
}

// Cell order (APIC_OPT_P2G_ORDER 2), one CTA per 32 x 8 tile.  Each cell of
// the tile's region (the tile plus two halo columns on the left and two halo
// rows below) is summed by one thread: its particles in slot order, each
// particle's corners in corner order, into one partial sum per relative face
// position (6 u, 6 v, 4 density positions; the code bits of p2g_record).
// Each face then adds the partial sums of the cells that reach it in run
// order (the reference-order gather's cell offsets); empty cells are
// skipped.  The terms are those of the reference's order; only the
// association differs.  No particle is staged, so dense cells need no
// fallback.
constexpr int kCellRegion = kRegionW * kRegionH;  // 340
struct CellPartials {
    float uv[6][kCellRegion], uw[6][kCellRegion];
    float vv[6][kCellRegion], vw[6][kCellRegion];
    float dw[4][kCellRegion];
    uint8_t has[kCellRegion];
};

template <int NQ, bool kVal>
__device__ __forceinline__ void add_partials(const P2gRec& rec, float (&pv)[NQ], float (&pw)[NQ]) {
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
        const uint32_t hit = (rec.code >> (4 * q)) & 0xFu;
#pragma unroll
        for (int k = 0; k < 4; ++k)
            if (hit & (1u << k)) {
                if (kVal) pv[q] = pv[q] + rec.val[k];
                pw[q] = pw[q] + rec.w[k];
            }
    }
}

// For a particle inside (p2g_inside) the u corners start at column 0 or 1 of
// the six positions, the v corners at row 0 or 1, the density corners are the
// four positions.  Every position then takes at most one corner, by a select,
// where the general form tests each corner against each position (24 tests a
// grid).
struct P2gRaw {
    float px, py, tr, vx, cux, cuy, vy, cvx, cvy;
};
__device__ __forceinline__ P2gRaw p2g_raw(const PartPtrs* __restrict__ pp, uint32_t slot) {
    return P2gRaw{pp->f[PX][slot],  pp->f[PY][slot],  pp->f[TR][slot],  pp->f[VX][slot], pp->f[CUX][slot],
                  pp->f[CUY][slot], pp->f[VY][slot], pp->f[CVX][slot], pp->f[CVY][slot]};
}
__device__ __forceinline__ P2gBase p2g_base(const P2gRaw& r, CellSize cs, float prev_dt) {
    const float tau = (-r.tr) / prev_dt;
    return P2gBase{over_dx(r.px, cs), over_dx(r.py, cs), temporal_w(tau)};
}
__device__ __forceinline__ void p2g_add_inside(const P2gRaw& p, const P2gBase& b, int W, int H, float dx,
                                               float (&uv)[6], float (&uw)[6], float (&vv)[6], float (&vw)[6],
                                               float (&dw)[4]) {
    Stencil su, sv;
    u_stencil(b.gx, b.gy, W, H, dx, su);
    v_stencil(b.gx, b.gy, W, H, dx, sv);
    const float cgx = b.gx - 0.5f, cgy = b.gy - 0.5f;
    const float cbx = floorf(cgx), cby = floorf(cgy);
    const bool sx = floorf(b.gx) != cbx, sy = floorf(b.gy) != cby;
    float w[4], v[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        w[k] = su.w[k] * b.wt;
        v[k] = (p.vx + p.cux * su.ox[k] + p.cuy * su.oy[k]) * w[k];
    }
#pragma unroll
    for (int r = 0; r < 2; ++r) {
        uv[3 * r + 0] = uv[3 * r + 0] + (sx ? 0.0f : v[2 * r]);
        uv[3 * r + 1] = uv[3 * r + 1] + (sx ? v[2 * r] : v[2 * r + 1]);
        uv[3 * r + 2] = uv[3 * r + 2] + (sx ? v[2 * r + 1] : 0.0f);
        uw[3 * r + 0] = uw[3 * r + 0] + (sx ? 0.0f : w[2 * r]);
        uw[3 * r + 1] = uw[3 * r + 1] + (sx ? w[2 * r] : w[2 * r + 1]);
        uw[3 * r + 2] = uw[3 * r + 2] + (sx ? w[2 * r + 1] : 0.0f);
    }
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        w[k] = sv.w[k] * b.wt;
        v[k] = (p.vy + p.cvx * sv.ox[k] + p.cvy * sv.oy[k]) * w[k];
    }
#pragma unroll
    for (int c = 0; c < 2; ++c) {
        vv[c] = vv[c] + (sy ? 0.0f : v[c]);
        vv[2 + c] = vv[2 + c] + (sy ? v[c] : v[2 + c]);
        vv[4 + c] = vv[4 + c] + (sy ? v[2 + c] : 0.0f);
        vw[c] = vw[c] + (sy ? 0.0f : w[c]);
        vw[2 + c] = vw[2 + c] + (sy ? w[c] : w[2 + c]);
        vw[4 + c] = vw[4 + c] + (sy ? w[2 + c] : 0.0f);
    }
    const float ctx = cgx - cbx, cty = cgy - cby;
    dw[0] = dw[0] + ((1.0f - ctx) * (1.0f - cty)) * b.wt;
    dw[1] = dw[1] + (ctx * (1.0f - cty)) * b.wt;
    dw[2] = dw[2] + ((1.0f - ctx) * cty) * b.wt;
    dw[3] = dw[3] + (ctx * cty) * b.wt;
}

// One thread per region cell (352 threads for 340 cells, then the tile's 256
// cells' faces), two CTAs per SM.  The per-cell loops wait on loads: slot,
// then nine fields, then some 230 instructions.  The slot two particles ahead
// and the fields one ahead are in flight meanwhile (80 registers; three CTAs
// with 56 and spills were faster without the fields ahead, are slower with
// them: 460 against 352 us).  1024^2 dam break (1.0 M particles) 73 -> 53 us,
// 2048^2 noise (8.3 M) 589 -> 352 us, of which the selects of
// p2g_add_inside and the exact reciprocal took 17 and 182.
constexpr int kCellThreads = 352;
__global__ void __launch_bounds__(kCellThreads, 2) k_p2g_cells(const PartPtrs* __restrict__ pp,
                                                             const uint32_t* __restrict__ vals,
                                                             const uint32_t* __restrict__ lo,
                                                             const uint32_t* __restrict__ hi, int W, int H,
                                                             CellSize cs, Ctl* __restrict__ ctl, GatherOut o,
                                                             uint32_t n, uint32_t npad) {
    __shared__ CellPartials sp;
    const float dx = cs.dx;
    const int x0 = blockIdx.x * kGatherTW, y0 = blockIdx.y * kGatherTH;
    const int rx0 = x0 - 2, ry0 = y0 - 2;
    pdl_wait();
    const float prev_dt = ctl->prev_dt;
    bool bad = false, some = false;
    for (int rc = threadIdx.x; rc < kCellRegion; rc += kCellThreads) {
        const int x = rx0 + rc % kRegionW, y = ry0 + rc / kRegionW;
        uint32_t b = 0, e = 0;
        if (x >= 0 && x < W && y >= 0 && y < H) {
            const uint32_t c = uint32_t(y) * uint32_t(W) + uint32_t(x);
            b = lo[c];
            e = hi[c];
        }
        float uv[6] = {}, uw[6] = {}, vv[6] = {}, vw[6] = {}, dv[4] = {}, dw[4] = {};
        // two particles ahead the slot is loaded, one ahead the fields
        if (!APIC_IN_BOUNDS(e, uint64_t(n) + 1u, &ctl->status)) e = b;
        auto slot_at = [&](uint32_t p) {
            const uint32_t sl = p < e ? vals[p] : 0u;
            return APIC_IN_BOUNDS(sl, npad, &ctl->status) ? sl : 0u;
        };
        uint32_t slot = slot_at(b), next = slot_at(b + 1);
        P2gRaw raw = b < e ? p2g_raw(pp, slot) : P2gRaw{};
        for (uint32_t p = b; p < e; ++p) {
            const P2gRaw cur = raw;
            const uint32_t here = slot;
            slot = next;
            if (p + 1 < e) raw = p2g_raw(pp, slot);
            next = slot_at(p + 2);
            const P2gBase bs = p2g_base(cur, cs, prev_dt);
            if (p2g_inside(bs, W, H)) {
                p2g_add_inside(cur, bs, W, H, dx, uv, uw, vv, vw, dw);
                continue;
            }
            P2gRec rec;
            if (!p2g_record(pp, here, bs, kGridU, W, H, dx, rec)) bad = true;
            add_partials<6, true>(rec, uv, uw);
            if (!p2g_record(pp, here, bs, kGridV, W, H, dx, rec)) bad = true;
            add_partials<6, true>(rec, vv, vw);
            if (!p2g_record(pp, here, bs, kGridD, W, H, dx, rec)) bad = true;
            add_partials<4, false>(rec, dv, dw);
        }
#pragma unroll
        for (int q = 0; q < 6; ++q) {
            sp.uv[q][rc] = uv[q];
            sp.uw[q][rc] = uw[q];
            sp.vv[q][rc] = vv[q];
            sp.vw[q][rc] = vw[q];
        }
#pragma unroll
        for (int q = 0; q < 4; ++q) sp.dw[q][rc] = dw[q];
        sp.has[rc] = e > b;
        some = e > b;
    }
    if (bad) atomicOr(&ctl->status, kStatusP2gLayout);
    some = __syncthreads_or(some) != 0;  // (a region without particles: zeros, no sums)
    if (threadIdx.x >= kGatherThreads) return;
    const int tx = threadIdx.x % kGatherTW, ty = threadIdx.x / kGatherTW;
    const int i = x0 + tx, j = y0 + ty;
    if (i >= W || j >= H) return;
    // region index of cell (x, y), or -1 when it holds no particle (or lies
    // outside the grid)
    auto cell = [&](int x, int y) -> int {
        if (!some || x < 0 || y < 0 || x >= W || y >= H) return -1;
        const int rc = (y - ry0) * kRegionW + (x - rx0);
        return sp.has[rc] ? rc : -1;
    };
    for (int fi = i; fi <= (i == W - 1 ? W : i); ++fi) {
        float av = 0.0f, aw = 0.0f;
#pragma unroll
        for (int r = 0; r < 6; ++r) {
            const int rc = cell(fi - r % 3, j - r / 3);
            if (rc >= 0) {
                av = av + sp.uv[r][rc];
                aw = aw + sp.uw[r][rc];
            }
        }
        const uint32_t f = uint32_t(j) * uint32_t(W + 1) + uint32_t(fi);
        o.acc_u[f] = av;
        o.acc_uw[f] = aw;
    }
    for (int fj = j; fj <= (j == H - 1 ? H : j); ++fj) {
        float av = 0.0f, aw = 0.0f;
#pragma unroll
        for (int r = 0; r < 6; ++r) {
            const int rc = cell(i - r % 2, fj - r / 2);
            if (rc >= 0) {
                av = av + sp.vv[r][rc];
                aw = aw + sp.vw[r][rc];
            }
        }
        const uint32_t f = uint32_t(fj) * uint32_t(W) + uint32_t(i);
        o.acc_v[f] = av;
        o.acc_vw[f] = aw;
    }
    float aw = 0.0f;
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        const int rc = cell(i - r % 2, j - r / 2);
        if (rc >= 0) aw = aw + sp.dw[r][rc];
    }
    o.dens[uint32_t(j) * uint32_t(W) + uint32_t(i)] = aw;
}

// bilinear_interpolate, src/apic.rs:138-172.
__device__ __forceinline__ float bilinear(const float w[4], const float v[4]) {
    float ws = w[0] + w[1] + w[2] + w[3];
    float inv = 1.0f / fmax_x86(ws, 1e-6f);
    float vel = 0.0f;
#pragma unroll
    for (int k = 0; k < 4; ++k) vel += v[k] * w[k] * inv;
    return vel;
}

__device__ __forceinline__ void block_max_count(float m, uint32_t bad, Ctl* ctl) {
    __shared__ float sm[8];
    __shared__ uint32_t sb[8];
    m = warp_maxf(m);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) bad += __shfl_xor_sync(0xffffffffu, bad, o);
    int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (lane == 0) { sm[warp] = m; sb[warp] = bad; }
    __syncthreads();
    if (threadIdx.x == 0) {
        float bm = 0.0f;
        uint32_t bb = 0;
        for (int w = 0; w < int(blockDim.x / 32); ++w) { bm = fmaxf(bm, sm[w]); bb += sb[w]; }
        if (bm > 0.0f) atomicMax(&ctl->vmax_bits, __float_as_uint(bm));
        if (bb) atomicAdd(&ctl->nonfinite, bb);
    }
}

// four CTAs per SM (64 registers): G2P is bound by the latency of its
// dependent loads (particle, then the faces it gathers); at 4096^2 four CTAs
// per SM take the stage from 0.88 to 0.73 ms
__global__ void __launch_bounds__(256, 4) k_g2p(const PartPtrs* __restrict__ pp, uint32_t npad, int W, int H, float dx,
                                             float border_damping, Ctl* __restrict__ ctl,
                                             const float* __restrict__ gu, const float* __restrict__ gv,
                                             const uint32_t* __restrict__ u_open,
                                             const uint32_t* __restrict__ v_open) {
    pdl_wait();
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    float speed_out = 0.0f;
    uint32_t bad = 0;
    if (i < npad) {
        const float dt = ctl->dt;
        const uint32_t ts = ctl->timestamp;
        const float min_x = 1.001f * dx, max_x = (float(W) - 1.001f) * dx;
        const float min_y = 1.001f * dx, max_y = (float(H) - 1.001f) * dx;
        const float h2 = dx * dx, eps = 1e-6f, bd = -border_damping;
        float px = pp->f[PX][i], py = pp->f[PY][i];
        float gx = px / dx, gy = py / dx;
        Stencil su, sv;
        u_stencil(gx, gy, W, H, dx, su);
        v_stencil(gx, gy, W, H, dx, sv);
        float un[4], vn[4], uwm[4], vwm[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const bool uin = APIC_IN_BOUNDS(su.idx[k], uint32_t(W + 1) * uint32_t(H), &ctl->status);
            const bool vin = APIC_IN_BOUNDS(sv.idx[k], uint32_t(W) * uint32_t(H + 1), &ctl->status);
            un[k] = uin ? gu[su.idx[k]] : 0.0f;
            vn[k] = vin ? gv[sv.idx[k]] : 0.0f;
            uwm[k] = uin && bit_at(u_open, su.idx[k]) ? su.w[k] : 0.0f;
            vwm[k] = vin && bit_at(v_open, sv.idx[k]) ? sv.w[k] : 0.0f;
        }
        float nvx = bilinear(uwm, un), nvy = bilinear(vwm, vn);
        float res = pp->f[TR][i];
        float speed = sqrtf(nvx * nvx + nvy * nvy);
        float cfl_local = speed * dt / dx;
        float scale = fmin_x86(fmax_x86(cfl_local, 0.0f), 1.0f);
        float gam = scale * scale * (3.0f - (2.0f * scale));
        float jitter = gam * random_lane(i, ts) * dt;
        float dt_raw = dt + res + jitter;
        float dt_act = fmin_x86(fmax_x86(dt_raw, 0.0f), dt * 2.0f);
        float nres = dt + res - dt_act;
        float nx = px + dt_act * nvx, ny = py + dt_act * nvy;
        bool oxmin = nx < min_x, oxmax = nx > max_x, oymin = ny < min_y, oymax = ny > max_y;
        bool ovxmin = oxmin && nvx < 0.0f, ovxmax = oxmax && nvx > 0.0f;
        bool ovymin = oymin && nvy < 0.0f, ovymax = oymax && nvy > 0.0f;
        if (oxmin) nx = min_x;
        if (oxmax) nx = max_x;
        if (ovxmin) nvx = nvx * bd;
        if (ovxmax) nvx = nvx * bd;
        if (oymin) ny = min_y;
        if (oymax) ny = max_y;
        if (ovymin) nvy = nvy * bd;
        if (ovymax) nvy = nvy * bd;
        float udx = h2 * su.tx * (1.0f - su.tx), udy = h2 * su.ty * (1.0f - su.ty);
        float vdx = h2 * sv.tx * (1.0f - sv.tx), vdy = h2 * sv.ty * (1.0f - sv.ty);
        float uix = udx > eps ? 1.0f / udx : 0.0f, uiy = udy > eps ? 1.0f / udy : 0.0f;
        float vix = vdx > eps ? 1.0f / vdx : 0.0f, viy = vdy > eps ? 1.0f / vdy : 0.0f;
        float cux = 0.0f, cuy = 0.0f, cvx = 0.0f, cvy = 0.0f;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            cux += su.w[k] * un[k] * su.ox[k];
            cuy += su.w[k] * un[k] * su.oy[k];
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            cvx += sv.w[k] * vn[k] * sv.ox[k];
            cvy += sv.w[k] * vn[k] * sv.oy[k];
        }
        float cu_x = cux * uix, cu_y = cuy * uiy, cv_x = cvx * vix, cv_y = cvy * viy;
        bool rx = ovxmin || ovxmax, ry = ovymin || ovymax;
        if (rx) { cu_y = cu_y * -1.0f; cv_x = cv_x * -1.0f; }
        if (ry) { cu_y = cu_y * -1.0f; cv_x = cv_x * -1.0f; }
        pp->f[PX][i] = nx;
        pp->f[PY][i] = ny;
        pp->f[VX][i] = nvx;
        pp->f[VY][i] = nvy;
        pp->f[CUX][i] = cu_x;
        pp->f[CUY][i] = cu_y;
        pp->f[CVX][i] = cv_x;
        pp->f[CVY][i] = cv_y;
        pp->f[TR][i] = nres;
        float m = sqrtf(nvx * nvx + nvy * nvy);  // Vec2x8::mag of the stored velocity
        speed_out = (m == m) ? m : 0.0f;
        bad = (isfinite(nx) && isfinite(ny)) ? 0u : 1u;
    }
    block_max_count(speed_out, bad, ctl);
}

// Max |v| over all npad lanes (a multiple of 8): a grid of one wave, four
// lanes per step with 16-byte loads, one atomic per block.
__global__ void __launch_bounds__(256) k_vmax(const PartPtrs* __restrict__ pp, uint32_t npad, Ctl* __restrict__ ctl) {
    pdl_wait();
    float m = 0.0f;
    const float* vx = pp->f[VX];
    const float* vy = pp->f[VY];
    for (uint32_t i0 = 4u * (blockIdx.x * blockDim.x + threadIdx.x); i0 < npad; i0 += 4u * gridDim.x * blockDim.x) {
        const float4 x = *reinterpret_cast<const float4*>(vx + i0), y = *reinterpret_cast<const float4*>(vy + i0);
        const float xs[4] = {x.x, x.y, x.z, x.w}, ys[4] = {y.x, y.y, y.z, y.w};
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const float mg = sqrtf(xs[q] * xs[q] + ys[q] * ys[q]);
            m = fmaxf(m, (mg == mg) ? mg : 0.0f);
        }
    }
    block_max_count(m, 0u, ctl);
}

__global__ void k_zero_vmax(Ctl* ctl) {
    pdl_wait(); ctl->vmax_bits = 0; ctl->nonfinite = 0; }

// Four consecutive slots per thread: 128-bit loads of the sorted slots and
// 128-bit stores of each field (the gathered reads are one float each).
__global__ void __launch_bounds__(256) k_permute(PartPtrs* __restrict__ pp, const uint32_t* __restrict__ vals,
                                                 uint32_t n, uint32_t npad, uint32_t* __restrict__ status) {
    pdl_wait();
    const uint32_t i0 = 4u * (blockIdx.x * blockDim.x + threadIdx.x);
    if (i0 >= npad) return;  // npad is a multiple of 8
    uint32_t src[4];
    bool ok[4];
    if (i0 + 4u <= n) {
        const uint4 v = *reinterpret_cast<const uint4*>(vals + i0);
        src[0] = v.x; src[1] = v.y; src[2] = v.z; src[3] = v.w;
#pragma unroll
        for (int k = 0; k < 4; ++k) ok[k] = true;
    } else {
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            ok[k] = i0 + uint32_t(k) < n;
            src[k] = ok[k] ? vals[i0 + k] : 0u;
        }
    }
#pragma unroll
    for (int k = 0; k < 4; ++k) ok[k] = ok[k] && APIC_IN_BOUNDS(src[k], npad, status);
#pragma unroll
    for (int f = 0; f < NPF; ++f) {
        const float* a = pp->f[f];
        float4 o;
        o.x = ok[0] ? a[src[0]] : 0.0f;
        o.y = ok[1] ? a[src[1]] : 0.0f;
        o.z = ok[2] ? a[src[2]] : 0.0f;
        o.w = ok[3] ? a[src[3]] : 0.0f;
        *reinterpret_cast<float4*>(pp->alt[f] + i0) = o;
    }
}

__global__ void k_swap_tables(PartPtrs* pp) {
    pdl_wait();
    int f = threadIdx.x;
    if (f < NPF) {
        float* t = pp->f[f];
        pp->f[f] = pp->alt[f];
        pp->alt[f] = t;
    }
}

}  // namespace

static CellSize cell_size(const Scene& s) { return CellSize{s.dx, exact_reciprocal(s.dx)}; }

// P2G stage; the base fluid mask, and without particles bin_lo / bin_hi, must be
// zero (the caller clears them), every accumulator entry is written.
cudaError_t launch_p2g(Scene& s) {
    const bool ref = p2g_reference_order(s);
    cudaError_t e = cudaFuncSetAttribute(k_p2g_gather, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         int(kFaceSmem));
    if (e != cudaSuccess) return e;
    const uint32_t* svals = s.bin_vals;
    if (s.n > 0) {
        // blocks for the particles, or for the cells' runs where a large grid holds
        // few (one wave at most: the clearing walks the grid).  By the particles
        // alone, a thousand on 4096^2 cells left 134 MB to one CTA: the stage
        // took 2572 us, 554 now (1024^2 190 -> 67)
        const uint32_t blocks = std::max(div_up(s.n, 1024), std::min(div_up(s.cells, 4096), 152u * 8u));
        launch(s.use_pdl, k_p2g_bin_keys, blocks, 256, 0, s.stream, static_cast<const PartPtrs*>(s.pp), s.n,
               int(s.W), int(s.H), cell_size(s), s.bin_keys, s.lv[0].fluid, s.sort_scratch, s.bin_lo, s.bin_hi);
        uint32_t *kres, *vres;
        e = radix_sort_pairs(s.bin_keys, s.bin_vals, s.bin_keys_alt, s.bin_vals_alt, s.sort_scratch, s.n,
                             bin_key_bits(s), 0, s.stream, s.use_pdl, &kres, &vres, &s.ctl->status);
        if (e != cudaSuccess) return e;
        launch(s.use_pdl, k_p2g_bounds, div_up(s.n, 256), 256, 0, s.stream, static_cast<const uint32_t*>(kres), s.n,
               s.bin_lo, s.bin_hi, s.cells, &s.ctl->status);
        svals = vres;
    }
    GatherOut o{s.acc_u, s.acc_uw, s.acc_v, s.acc_vw, s.density};
    const dim3 grid(div_up(s.W, kGatherTW), div_up(s.H, kGatherTH));
    // a grid has up to (W + 1) x H or W x (H + 1) faces
    const dim3 faces(div_up(s.W + 1, kFaceTW), div_up(s.H + 1, kFaceTH), 3);
    if (ref)
        launch(s.use_pdl && s.n > 0, k_p2g_gather, faces, kFaceThreads, kFaceSmem, s.stream,
               static_cast<const PartPtrs*>(s.pp), svals, static_cast<const uint32_t*>(s.bin_lo),
               static_cast<const uint32_t*>(s.bin_hi), int(s.W), int(s.H), cell_size(s), s.ctl, o, s.n, s.npad);
    else
        launch(s.use_pdl && s.n > 0, k_p2g_cells, grid, kCellThreads, 0, s.stream,
               static_cast<const PartPtrs*>(s.pp), svals, static_cast<const uint32_t*>(s.bin_lo),
               static_cast<const uint32_t*>(s.bin_hi), int(s.W), int(s.H), cell_size(s), s.ctl, o, s.n, s.npad);
    return cudaGetLastError();
}

cudaError_t launch_g2p(Scene& s) {
    if (s.npad == 0) return cudaSuccess;
    launch(s.use_pdl, k_g2p, div_up(s.npad, 256), 256, 0, s.stream, s.pp, s.npad, int(s.W), int(s.H), s.dx, s.props.border_damping,
                                                      s.ctl, s.u, s.v, s.u_open, s.v_open);
    return cudaGetLastError();
}

// Zero the running maximum, then reduce over the current velocities.
cudaError_t launch_vmax(Scene& s) {
    launch(s.use_pdl, k_zero_vmax, 1, 1, 0, s.stream, s.ctl);
    if (s.npad) {
        const uint32_t g = std::min(div_up(s.npad, 1024), uint32_t(kMaxRedBlocks));
        launch(s.use_pdl, k_vmax, g, 256, 0, s.stream, s.pp, s.npad, s.ctl);
    }
    return cudaGetLastError();
}

// Interleave two SoA particle fields into the reference's Vec2x8 layout
// (per chunk: 8 x lanes then 8 y lanes), for one contiguous copy to the host.
// Thread t writes 16 bytes of the packed output: chunk t / 4, quarter t % 4
// (quarters 0-1: x lanes 0-3, 4-7; quarters 2-3: y lanes).
__global__ void __launch_bounds__(256) k_pack_vec2x8(const PartPtrs* __restrict__ pp, int fx, int fy, uint32_t nchunks,
                                                     float* __restrict__ out) {
    const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= nchunks * 4u) return;
    const uint32_t c = t >> 2, q = t & 3u;
    const float* src = (q < 2u ? pp->f[fx] : pp->f[fy]) + c * 8u + (q & 1u) * 4u;
    *reinterpret_cast<float4*>(out + size_t(t) * 4u) = *reinterpret_cast<const float4*>(src);
}

cudaError_t launch_pack_vec2x8(Scene& s, int which, float* out) {
    if (s.nchunks == 0) return cudaSuccess;
    k_pack_vec2x8<<<div_up(uint64_t(s.nchunks) * 4, 256), 256, 0, s.stream>>>(s.pp, 2 * which, 2 * which + 1,
                                                                            s.nchunks, out);
    return cudaGetLastError();
}

cudaError_t launch_permute(Scene& s, const uint32_t* sorted_vals) {
    if (s.npad == 0) return cudaSuccess;
    launch(s.use_pdl, k_permute, div_up(s.npad / 4, 256), 256, 0, s.stream, s.pp, sorted_vals, s.n, s.npad,
           &s.ctl->status);
    launch(s.use_pdl, k_swap_tables, 1, 32, 0, s.stream, s.pp);
    return cudaGetLastError();
}

}  // namespace apic
