// vcycle_dsm.cu — the middle multigrid levels in distributed shared memory.
//
// The same V-cycle arithmetic as vcycle.cu (smooth_level src/apic.rs:471-535,
// restrict :537-594, prolongate :596-616, solve_coarse_exact :618-704), with
// the levels between the grid-wide kernels and the coarse tail held in the
// shared memory of one 16-CTA thread-block cluster.  CTA r owns rows
// [r R, (r+1) R) of every such level (R = height / 16) and holds two more rows
// on each side: with them it smooths its band and the row next to it by
// itself, computing the neighbour's values again from the same inputs with
// the same operations.  What it cannot compute, the neighbours push into its
// halo rows as they form it (distributed shared memory, stores only): the
// coarse residual of the restriction, the boundary rows' final errors.  So a
// level costs one cluster barrier going down and one going up, and no phase
// waits for another CTA's shared memory.  CTA 0 runs the coarse tail (levels
// of fewer than kDsmTailRows rows) between the two halves; the restriction
// into it writes there directly and it pushes every band its rows.
//
// Bound by the latency of its phases and barriers (some 190 KB per CTA never
// leave the SMs).  The form before this one read neighbours' rows in place,
// tested fluid bits per neighbour, took a cluster barrier per sweep and read
// every level's layout from the kernel's parameters; a PCG iteration with it
// took 43.2 us at 128^2 (64^2 in the cluster), 51.2 at 256^2, 69.6 at 1024^2
// (256^2 to 64^2 in the cluster), now 32.6, 37.4 and 58.1.
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include "apic_device.cuh"
#include "apic_internal.h"
#include "pcg_common.cuh"
#include "vcycle_common.cuh"

namespace apic {
using namespace vc;
namespace {
namespace cg = cooperative_groups;

constexpr uint32_t kDsmCtas = 16;
constexpr uint32_t kDsmTailRows = 64;
constexpr int kDsmMaxLevels = 6;
constexpr size_t kDsmSmemBudget = 220 * 1024;
constexpr int kDsmHalo = 2;
constexpr int kDsmPad = 4;  // floats before and after a level's rows (reads one past a row's ends)

// One distributed level; widths are multiples of 32.
struct DsmLevel {
    const uint32_t* fluid;
    const float *diag, *inv, *px, *py;  // global, padded layout
};
struct DsmParams {
    int n;       // distributed levels, finest first
    int w, R;    // of the finest
    int hshift;  // log2(w / 2), or -1 when it is not a power of two
    int cells;
    const float* res;  // of the finest, global, padded layout
    float* err;
    const float* tinv;        // the first tail level's inverse diagonal, global
    DsmLevel lv[kDsmMaxLevels];
};

// A distributed level in this CTA's shared memory: five arrays of rows -2 ..
// R + 1 (row 0 is the band's first) with kDsmPad floats before and after,
// indexed by row * w + x, then the diagonal's rows 0 .. R - 1.  As in the flat
// index of the reference, the cell after a row's last one is the next row's
// first.  The levels lie one after another, each half the width and rows of
// the one before; behind the last, the tail's error around the band (rows -1
// .. R / 2 of its width) and its inverse diagonal under it.
struct Band {
    int w, R, hshift;
    float* at;  // the level's first float
    float *e, *r, *inv, *px, *py, *d;
};
__device__ __forceinline__ int band_floats(int w, int R) { return (R + 2 * kDsmHalo) * w + 2 * kDsmPad; }
__device__ __forceinline__ Band band_at(float* at, int w, int R, int hshift) {
    const int n = band_floats(w, R);
    float* e = at + kDsmPad + kDsmHalo * w;
    return Band{w, R, hshift, at, e, e + n, e + 2 * n, e + 3 * n, e + 4 * n, at + 5 * n};
}
__device__ __forceinline__ Band band_coarser(const Band& f) {
    return band_at(f.d + f.R * f.w, f.w >> 1, f.R >> 1, f.hshift > 0 ? f.hshift - 1 : -1);
}
__device__ __forceinline__ Band band_finer(const Band& c) {
    const int w = c.w << 1, R = c.R << 1;
    return band_at(c.at - 5 * band_floats(w, R) - R * w, w, R, c.hshift >= 0 ? c.hshift + 1 : -1);
}

// The neighbours' views of an array in this CTA's shared memory.
struct Peers {
    float *below, *above;  // rank - 1, rank + 1 (this CTA's own where there is none)
    bool has_below, has_above;
};
__device__ __forceinline__ Peers peers_of(const cg::cluster_group& cl, float* p, uint32_t rank) {
    const bool b = rank > 0, a = rank + 1 < kDsmCtas;
    return Peers{cl.map_shared_rank(p, b ? rank - 1 : rank), cl.map_shared_rank(p, a ? rank + 1 : rank), b, a};
}

// Cell k of one colour in rows first, first + 1, ...
__device__ __forceinline__ void band_cell(const Band& b, int k, int first, int color, int& row, int& x) {
    const int half = b.w >> 1;
    int q;
    if (b.hshift >= 0) {
        q = k >> b.hshift;
        k &= half - 1;
    } else {
        q = k / half;
        k -= q * half;
    }
    row = first + q;
    x = 2 * k + ((row + color) & 1);  // (a band starts on an even row)
}

// Black sweep after the red one, on the band and a row on each side.
__device__ __forceinline__ void dsm_black(const Band& b) {
    const int n = (b.R + 2) * (b.w >> 1), w = b.w;
    for (int k = threadIdx.x; k < n; k += kTailThreads) {
        int row, x;
        band_cell(b, k, -1, 1, row, x);
        const int i = row * w + x;
        b.e[i] = sor_masked(b.inv[i], b.r[i], b.px[i], b.py[i], b.px[i - 1], b.py[i - w], b.e[i + 1], b.e[i + w],
                            b.e[i - 1], b.e[i - w], 0.0f);
    }
}

// Restriction of the band into its coarse rows, two threads per coarse cell
// (one per row of children); put(coarse row, x, sum) stores the residual.
template <class Put>
__device__ __forceinline__ void dsm_restrict(const Band& f, Put put) {
    const int cw = f.w >> 1, n = f.R * cw, w = f.w;  // a multiple of 32: whole warps
    for (int k = threadIdx.x; k < n; k += kTailThreads) {
        const int q = k >> 1, dy = k & 1;
        int row, x;
        if (f.hshift >= 0) {
            row = q >> f.hshift;
            x = q & (cw - 1);
        } else {
            row = q / cw;
            x = q - row * cw;
        }
        const int i = (2 * row + dy) * w + 2 * x;
        const float2 two = left_over(f.r, f.d, f.px, f.py, f.e, i, w);
        const float d0 = two.x, d1 = two.y;
        const float d2 = __shfl_down_sync(0xffffffffu, d0, 1), d3 = __shfl_down_sync(0xffffffffu, d1, 1);
        if (dy == 0) put(row, x, (((0.0f + d0) + d1) + d2) + d3);
    }
}

// Reverse sweep of one colour with the prolongation from ce (rows of w / 2,
// rows -1 .. R / 2): black on the band and a row on each side, red on the
// band.  done(row, x, value) for every cell.
template <int kColor, class Done>
__device__ __forceinline__ void dsm_up(const Band& f, const float* ce, Done done) {
    const int first = kColor == 1 ? -1 : 0, rows = kColor == 1 ? f.R + 2 : f.R;
    const int n = rows * (f.w >> 1), w = f.w, cw = f.w >> 1;
    for (int k = threadIdx.x; k < n; k += kTailThreads) {
        int row, x;
        band_cell(f, k, first, kColor, row, x);
        const int i = row * w + x, cc = (row >> 1) * cw + (x >> 1);
        float er = f.e[i + 1], eu = f.e[i + w], el = f.e[i - 1], ed = f.e[i - w], old = f.e[i];
        if (kColor == 1) {
            const bool xo = x & 1, yo = row & 1;
            const CoarseAround a = coarse_around(ce, cc, cw, xo, yo);
            old = old + a.c0;
            er = er + (xo ? a.h : a.c0);
            el = el + (xo ? a.c0 : a.h);
            eu = eu + (yo ? a.v : a.c0);
            ed = ed + (yo ? a.c0 : a.v);
        } else {
            old = old + ce[cc];
        }
        const float z = sor_masked(f.inv[i], f.r[i], f.px[i], f.py[i], f.px[i - 1], f.py[i - w], er, eu, el, ed, old);
        f.e[i] = z;
        done(row, x, z);
    }
}

// Start copying the coefficients of a band and its halo (zero outside the
// fluid; rows outside the grid are zeroed here) and zero its vectors.
__device__ __forceinline__ void dsm_issue_coeffs(const DsmLevel& L, const Band& b, uint32_t rank) {
    const int rows = b.R + 2 * kDsmHalo, n4 = rows * b.w / 4, n = band_floats(b.w, b.R);
    const int base = (int(rank) * b.R - kDsmHalo) * b.w;  // raw index of the first halo row
    const int cells = int(kDsmCtas) * b.R * b.w;
    const float4 zero = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    if (threadIdx.x < 2 * kDsmPad) {  // before and after the rows
        const int i = int(threadIdx.x) < kDsmPad ? int(threadIdx.x) : int(threadIdx.x) + rows * b.w;
        for (int k = 0; k < 5; ++k) b.at[k * n + i] = 0.0f;
    }
    for (int j = threadIdx.x; j < n4; j += kTailThreads) {
        const int raw = base + 4 * j;
        float* to = b.at + kDsmPad + 4 * j;  // e; r, inv, px, py follow every n floats
        *reinterpret_cast<float4*>(to) = zero;
        *reinterpret_cast<float4*>(to + n) = zero;
        if (raw >= 0 && raw < cells) {
            const size_t g = size_t(raw) + b.w;
            cp_async16(to + 2 * n, L.inv + g);
            cp_async16(to + 3 * n, L.px + g);
            cp_async16(to + 4 * n, L.py + g);
            const int own = 4 * j - kDsmHalo * b.w;
            if (own >= 0 && own < b.R * b.w) cp_async16(b.d + own, L.diag + g);
        } else {
            *reinterpret_cast<float4*>(to + 2 * n) = zero;
            *reinterpret_cast<float4*>(to + 3 * n) = zero;
            *reinterpret_cast<float4*>(to + 4 * n) = zero;
        }
    }
}

__global__ void __launch_bounds__(kTailThreads, 1) k_vcycle_dsm(const __grid_constant__ DsmParams p,
                                                               const __grid_constant__ TailParams tp, uint32_t dsm_off,
                                                               Ctl* ctl, ExitArgs exit) {
    extern __shared__ __align__(16) uint8_t smem[];
    cg::cluster_group cl = cg::this_cluster();
    const uint32_t rank = cl.block_rank();
    float* dsm = reinterpret_cast<float*>(smem + dsm_off);
    uint32_t* tail_sm = reinterpret_cast<uint32_t*>(smem);
    const int n = p.n;
    const Band first = band_at(dsm, p.w, p.R, p.hshift);
    // masks and coefficients were written by the multigrid setup, before the
    // solve: their copies start before the wait for the previous kernel
    Band b = first;
    for (int k = 0; k < n; ++k) {
        if (k > 0) b = band_coarser(b);
        dsm_issue_coeffs(p.lv[k], b, rank);
    }
    const Band last = b;
    const int tw = last.w >> 1, tail_rows = last.R >> 1;
    float* te = last.d + last.R * last.w;                 // the tail's error around the band
    float* ti = te + (tail_rows + 2) * tw + 2 * kDsmPad;  // its inverse diagonal under it
    for (int i = threadIdx.x; i < (tail_rows + 2) * tw + 2 * kDsmPad; i += kTailThreads) te[i] = 0.0f;
    for (int i = threadIdx.x; i < tail_rows * tw; i += kTailThreads)
        cp_async4(ti + i, p.tinv + (int(rank) * tail_rows + 1) * tw + i);
    if (rank == 0) cta_tail_issue_coeffs(tp, tail_sm);
    const int rows = first.R + 2 * kDsmHalo, n2 = rows * first.w / 2;
    const int base = (int(rank) * first.R - kDsmHalo) * first.w;
    uint32_t mask = 0;  // fluid bits of this thread's pairs of the finest level (at most 16 pairs: 220 KB)
    for (int j = threadIdx.x, k = 0; j < n2; j += kTailThreads, k += 2) {
        const int raw = base + 2 * j;
        if (raw >= 0 && raw < p.cells) mask |= ((p.lv[0].fluid[raw >> 5] >> (raw & 31)) & 3u) << k;
    }
    __syncthreads();
    // no CTA writes into another's shared memory before that one has zeroed
    // it; waited for only before the first such write
    cl.barrier_arrive();
    pdl_wait();
    // the finest level's residual (written by the kernel before), halo included
    for (int j = threadIdx.x; j < n2 / 2; j += kTailThreads) {
        const int raw = base + 4 * j;
        if (raw >= 0 && raw < p.cells)
            cp_async16(first.r - kDsmHalo * first.w + 4 * j, p.res + size_t(raw) + first.w);
    }
    // (the same verdict in every CTA)
    const bool done = pcg::solve_over(ctl, exit, rank == 0);
    cp_async_wait_all();
    __syncthreads();
    if (!done) {  // mask it (only the fluid cells' was written); its first red sweep
        for (int j = threadIdx.x, k = 0; j < n2; j += kTailThreads, k += 2) {
            const int i = 2 * j - kDsmHalo * first.w;
            float2 r = *reinterpret_cast<const float2*>(first.r + i);
            if (!((mask >> k) & 1u)) r.x = 0.0f;
            if (!((mask >> k) & 2u)) r.y = 0.0f;
            *reinterpret_cast<float2*>(first.r + i) = r;
            // the red one of the pair: the first on even rows
            const bool odd = ((2 * j) / first.w) & 1;
            const float2 inv = *reinterpret_cast<const float2*>(first.inv + i);
            *reinterpret_cast<float2*>(first.e + i) =
                odd ? make_float2(0.0f, red_first(r.y, inv.y)) : make_float2(red_first(r.x, inv.x), 0.0f);
        }
    }
    __syncthreads();
    cl.barrier_wait();
    if (done) return;

    Band f = first;
    for (int k = 0; k < n; ++k) {
        dsm_black(f);
        __syncthreads();
        if (k + 1 < n) {
            // the coarse band's residual and red sweep, and what the
            // neighbours' halos need of them: red errors two rows out, the
            // black cells' residual one row out
            const Band c = band_coarser(f);
            const Peers pe = peers_of(cl, c.e, rank), pr = peers_of(cl, c.r, rank);
            dsm_restrict(f, [&](int row, int x, float sum) {
                const int i = row * c.w + x;
                const bool red = ((row + x) & 1) == 0;
                const float e = red ? red_first(sum, c.inv[i]) : 0.0f;
                c.r[i] = sum;
                c.e[i] = e;
                if (row < kDsmHalo && pe.has_below) {
                    const int q = (c.R + row) * c.w + x;
                    if (red) pe.below[q] = e;
                    else if (row == 0) pr.below[q] = sum;
                }
                if (row >= c.R - kDsmHalo && pe.has_above) {
                    const int q = (row - c.R) * c.w + x;
                    if (red) pe.above[q] = e;
                    else if (row == c.R - 1) pr.above[q] = sum;
                }
            });
            f = c;
        } else {
            const SmemLevel t = smem_first(tp, tail_sm);
            float* tr = cl.map_shared_rank(t.res, 0);
            float* tz = cl.map_shared_rank(t.err, 0);
            const int row0 = int(rank) * tail_rows;
            dsm_restrict(f, [&](int row, int x, float sum) {
                const int y = row0 + row, q = (y + 1) * tw + x;
                tr[q] = sum;
                tz[q] = ((x + y) & 1) == 0 ? red_first(sum, ti[row * tw + x]) : 0.0f;
            });
        }
        cl.sync();
    }
    if (rank == 0) {
        cta_tail_levels(tp, tail_sm);
        // every band's rows of the tail's error, and one on each side
        const float* err = smem_first(tp, tail_sm).err;
        const int per = (tail_rows + 2) * tw;
        for (int i = threadIdx.x; i < per * int(kDsmCtas); i += kTailThreads) {
            const int to = i / per, j = i - to * per;
            // row -1 of the band of CTA `to` is row to * tail_rows of the padded layout
            cl.map_shared_rank(te, to)[kDsmPad + j] = err[to * tail_rows * tw + j];
        }
    }
    cl.sync();
    const float* ce = te + kDsmPad + tw;
    for (int k = n - 1; k >= 1; --k) {
        dsm_up<1>(f, ce, [](int, int, float) {});
        __syncthreads();
        // The finer level reads the coarse rows beside its own: the
        // neighbours have those rows' black cells and are sent the red
        // ones, into the residual's halo (whose red cells nothing reads),
        // since they may still be sweeping with the errors they hold.
        const Peers pr = peers_of(cl, f.r, rank);
        dsm_up<0>(f, ce, [&](int row, int x, float z) {
            if (row == 0 && pr.has_below) pr.below[f.R * f.w + x] = z;
            if (row == f.R - 1 && pr.has_above) pr.above[-f.w + x] = z;
        });
        cl.sync();
        for (int i = threadIdx.x; i < f.w; i += kTailThreads) {  // half a row's red cells on each side
            const int half = f.w >> 1, row = i < half ? -1 : f.R;
            const int q = row * f.w + 2 * (i < half ? i : i - half) + (row & 1);
            f.e[q] = f.r[q];
        }
        __syncthreads();
        ce = f.e;
        f = band_finer(f);
    }
    // the finest level's final error goes to global memory
    float* out = p.err + (int(rank) * f.R + 1) * f.w;
    dsm_up<1>(f, ce, [&](int row, int x, float z) {
        if (row >= 0 && row < f.R) out[row * f.w + x] = z;
    });
    __syncthreads();
    dsm_up<0>(f, ce, [&](int row, int x, float z) { out[row * f.w + x] = z; });
}

// Floats of one distributed level.
size_t dsm_level_floats(const Level& L, uint32_t R) {
    const size_t band = size_t(R + 2 * kDsmHalo) * L.w + 2 * kDsmPad;
    return 5 * band + size_t(R) * L.w;
}

int log2_exact(uint32_t v) {
    if (v == 0 || (v & (v - 1))) return -1;
    int k = 0;
    while ((1u << k) < v) ++k;
    return k;
}

cudaLaunchConfig_t dsm_config(size_t smem, cudaStream_t st, cudaLaunchAttribute* attr, bool pdl) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(kDsmCtas, 1, 1);
    cfg.blockDim = dim3(kTailThreads, 1, 1);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = kDsmCtas;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = pdl ? 2 : 1;
    return cfg;
}

}  // namespace

// Pick the distributed levels: the tail starts at the first level with fewer
// than kDsmTailRows rows (one CTA runs a level of 32 x 32 cells with
// __syncthreads between phases faster than the cluster does with cluster
// barriers); going up from there, levels join while their height divides by
// 16 into an even band height, their width is a multiple of 32 and everything
// fits in 220 KB per CTA.
void plan_vcycle_dsm(Scene& s) {
    s.dsm_first = s.dsm_tail = s.nlevels;
    s.dsm_smem = 0;
    s.dsm_off = 0;
    if (s.nlevels < 3) return;
    int d = 1;
    while (d < s.nlevels && s.lv[d].h >= kDsmTailRows) ++d;
    if (d >= s.nlevels || d < 2) return;
    uint32_t tail_size = 0;
    make_tail_params(s, d, &tail_size);
    const size_t off = (size_t(tail_size) * 4 + 15) & ~size_t(15);
    size_t bytes = off;
    int m = d;
    for (int l = d - 1; l >= 1 && d - l <= kDsmMaxLevels; --l) {
        const Level& L = s.lv[l];
        const uint32_t R = L.h / kDsmCtas;
        if (L.h % kDsmCtas != 0 || (L.w % 32u) || (R & 1u)) break;
        size_t b = bytes + 4 * dsm_level_floats(L, R);
        // the tail's error around a band, its inverse diagonal under it
        if (l == d - 1) b += 4 * (size_t(R + 2) * (L.w / 2) + 2 * kDsmPad);
        if (b > kDsmSmemBudget) break;
        bytes = b;
        m = l;
    }
    if (m == d) return;
    cudaFuncSetAttribute(k_vcycle_dsm, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kDsmSmemBudget));
    cudaFuncSetAttribute(k_vcycle_dsm, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    cudaLaunchAttribute attr[2];
    cudaLaunchConfig_t cfg = dsm_config(bytes, nullptr, attr, false);
    int clusters = 0;
    const bool ok = cudaOccupancyMaxActiveClusters(&clusters, k_vcycle_dsm, &cfg) == cudaSuccess && clusters > 0;
    cudaGetLastError();
    if (!ok) return;
    s.dsm_first = m;
    s.dsm_tail = d;
    s.dsm_smem = bytes;
    s.dsm_off = uint32_t(off);
}

// Levels dsm_first .. dsm_tail-1 and the tail in one cluster launch.  On
// entry dsm_first's residual is in global memory (the down kernel above it);
// on exit its final error is.
void launch_vcycle_dsm(Scene& s, cudaStream_t st, const ExitArgs& exit) {
    DsmParams p = {};
    p.n = s.dsm_tail - s.dsm_first;
    uint32_t tail_size = 0;
    TailParams tp = make_tail_params(s, s.dsm_tail, &tail_size);
    const Level& F = s.lv[s.dsm_first];
    p.w = int(F.w);
    p.R = int(F.h / kDsmCtas);
    p.hshift = log2_exact(F.w / 2);
    p.cells = int(F.cells);
    p.res = F.res;
    p.err = F.err;
    p.tinv = s.lv[s.dsm_tail].inv_diag;
    for (int k = 0; k < p.n; ++k) {
        const Level& L = s.lv[s.dsm_first + k];
        p.lv[k] = DsmLevel{L.fluid, L.diag, L.inv_diag, L.px, L.py};
    }
    cudaLaunchAttribute attr[2];
    cudaLaunchConfig_t cfg = dsm_config(s.dsm_smem, st, attr, s.use_pdl);
    cudaLaunchKernelEx(&cfg, k_vcycle_dsm, p, tp, s.dsm_off, s.ctl, exit);
}

}  // namespace apic
