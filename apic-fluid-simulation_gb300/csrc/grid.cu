// grid.cu — MAC-grid and cell stages of the substep.
//
//   k_faces          normalise the P2G sums (src/apic.rs:1428-1459), add the
//                    external force (:1607-1612) and gravity on faces next to
//                    fluid (:1614-1625); one thread per face, fused.
//   k_compact_*      fluid mask clean-up (:1463-1464) and the ascending list of
//                    non-zero mask words of a level (the GPU form of the
//                    reference's fluid/red/black index lists, :1461-1494 and
//                    :1526-1553), with the fluid-cell count and the last fluid
//                    cell that the padded list duplicates (:1487-1494).
//   k_smooth_density three Jacobi passes over fluid cells (:1653-1685).
//   k_laplacian      divergence, ghost-fluid diagonal, +x/+y couplings and
//                    the density-correction right-hand side (:1698-1784).
//   k_coarsen        one multigrid level from its finer level (:1499-1602).
//   k_gradient       pressure projection per face (:1958-2055), fused with the
//                    post-force add (:2453-2458).
//   k_extrapolate    two Jacobi sweeps of velocity extrapolation for u and v
//                    in shared-memory tiles (:2266-2350).
//
// Cell stages run one warp per non-zero 32-bit mask word ("segment"): lane k
// owns raw cell 32*word + k, so every field access of a warp is one 128-byte
// line.  Neighbour reads are gated by the neighbour's fluid bit, which equals
// the reference's reads of zero-filled or zero-coefficient entries.
#include <cuda_runtime.h>

#include "apic_device.cuh"
#include "apic_internal.h"

namespace apic {
namespace {

constexpr int kCompactWords = 1024;  // mask words per compaction block

__global__ void __launch_bounds__(256) k_faces(uint32_t uf, uint32_t vf, int W, int H, const float* __restrict__ acc_u,
                                               const float* __restrict__ acc_uw, const float* __restrict__ acc_v,
                                               const float* __restrict__ acc_vw, float* __restrict__ u,
                                               float* __restrict__ v, uint8_t* __restrict__ valid_u,
                                               uint8_t* __restrict__ valid_v, const float* __restrict__ ext_u,
                                               const float* __restrict__ ext_v, const uint32_t* __restrict__ fluid,
                                               const uint32_t* __restrict__ obstacle, const Ctl* __restrict__ ctl,
                                               float gravity, int normalize, int forces, int apply_gravity) {
    pdl_wait();
    uint32_t f = blockIdx.x * blockDim.x + threadIdx.x;
    if (f >= uf + vf) return;
    const float dt = ctl->dt;
    const bool ext = forces && ctl->has_ext;
    if (f < uf) {
        float val;
        if (normalize) {
            float w = acc_uw[f];
            val = 0.0f;
            uint8_t ok = 0;
            if (w > 0.0f) { val = acc_u[f] / w; ok = 1; }
            valid_u[f] = ok;
        } else {
            val = u[f];
        }
        if (ext) val += ext_u[f] * dt;
        u[f] = val;
    } else {
        uint32_t g = f - uf;
        float val;
        if (normalize) {
            float w = acc_vw[g];
            val = 0.0f;
            uint8_t ok = 0;
            if (w > 0.0f) { val = acc_v[g] / w; ok = 1; }
            valid_v[g] = ok;
        } else {
            val = v[g];
        }
        if (ext) val += ext_v[g] * dt;
        if (apply_gravity) {
            int x = int(g % uint32_t(W)), y = int(g / uint32_t(W));
            // fluid bits net of obstacles, whether or not the mask has been cleaned yet
            uint32_t fb = fluid_xy(fluid, x, y - 1, W, H) & (1u - obstacle_xy(obstacle, x, y - 1, W, H));
            uint32_t ft = fluid_xy(fluid, x, y, W, H) & (1u - obstacle_xy(obstacle, x, y, W, H));
            if (fb || ft) val += gravity * dt;
        }
        v[g] = val;
    }
}

// Block b of the compaction owns mask words [b*1024, b*1024 + 1024).
__device__ __forceinline__ uint32_t load_clean_word(uint32_t* fluid, const uint32_t* obstacle, uint32_t w, uint32_t words,
                                                    bool write_back) {
    if (w >= words) return 0u;
    uint32_t m = fluid[w];
    if (obstacle) {
        uint32_t c = m & ~obstacle[w];
        if (write_back && c != m) fluid[w] = c;
        m = c;
    }
    return m;
}

__global__ void __launch_bounds__(256) k_compact_count(uint32_t* __restrict__ fluid, const uint32_t* __restrict__ obstacle,
                                                       uint32_t words, uint32_t* __restrict__ cnt) {
    pdl_wait();
    uint32_t nz = 0, cells = 0, last = 0;
    for (int k = 0; k < 4; ++k) {
        uint32_t w = blockIdx.x * kCompactWords + threadIdx.x * 4 + k;
        uint32_t m = load_clean_word(fluid, obstacle, w, words, true);
        if (m) { nz++; cells += __popc(m); last = max(last, w + 1); }
    }
    __shared__ uint32_t s[3][256];
    s[0][threadIdx.x] = nz; s[1][threadIdx.x] = cells; s[2][threadIdx.x] = last;
    __syncthreads();
    for (int o = 128; o > 0; o >>= 1) {
        if (threadIdx.x < o) {
            s[0][threadIdx.x] += s[0][threadIdx.x + o];
            s[1][threadIdx.x] += s[1][threadIdx.x + o];
            s[2][threadIdx.x] = max(s[2][threadIdx.x], s[2][threadIdx.x + o]);
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        cnt[3 * blockIdx.x + 0] = s[0][0];
        cnt[3 * blockIdx.x + 1] = s[1][0];
        cnt[3 * blockIdx.x + 2] = s[2][0];
    }
}

__device__ __forceinline__ uint32_t scan_1024(uint32_t v, uint32_t* total) {
    __shared__ uint32_t sw[32];
    int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) sw[warp] = x;
    __syncthreads();
    if (warp == 0) {
        uint32_t s = lane < int(blockDim.x / 32) ? sw[lane] : 0u;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            uint32_t y = __shfl_up_sync(0xffffffffu, s, o);
            if (lane >= o) s += y;
        }
        sw[lane] = s;
    }
    __syncthreads();
    uint32_t pre = warp > 0 ? sw[warp - 1] : 0u;
    *total = sw[blockDim.x / 32 - 1];
    __syncthreads();
    return pre + x - v;
}

// Segment list of one level (ascending non-zero mask words): block b writes
// its words after those of blocks [0, b), whose counts (k_compact_count) it
// sums itself; the last block also records the level's totals in Ctl (and,
// on the base level, the fluid-cell count, the last fluid cell and the
// padding of the reference's fluid list to a multiple of 8).
__global__ void __launch_bounds__(256) k_compact_write(const uint32_t* __restrict__ fluid, uint32_t words,
                                                       const uint32_t* __restrict__ cnt, uint32_t* __restrict__ seg,
                                                       uint32_t W, int level, Ctl* __restrict__ ctl) {
    pdl_wait();
    const uint32_t nb = gridDim.x, b0 = blockIdx.x;
    const bool last_block = b0 + 1 == nb;
    uint32_t before = 0, total = 0, cells = 0, lastw = 0;
    for (uint32_t b = threadIdx.x; b < (last_block ? nb : b0); b += 256) {
        const uint32_t c = cnt[3 * b];
        before += b < b0 ? c : 0u;
        total += c;
        cells += cnt[3 * b + 1];
        lastw = max(lastw, cnt[3 * b + 2]);
    }
    __shared__ uint32_t red[4][256];
    red[0][threadIdx.x] = before;
    red[1][threadIdx.x] = total;
    red[2][threadIdx.x] = cells;
    red[3][threadIdx.x] = lastw;
    __syncthreads();
    for (int o = 128; o > 0; o >>= 1) {
        if (threadIdx.x < o) {
            red[0][threadIdx.x] += red[0][threadIdx.x + o];
            red[1][threadIdx.x] += red[1][threadIdx.x + o];
            red[2][threadIdx.x] += red[2][threadIdx.x + o];
            red[3][threadIdx.x] = max(red[3][threadIdx.x], red[3][threadIdx.x + o]);
        }
        __syncthreads();
    }
    uint32_t m[4], nz = 0;
    for (int k = 0; k < 4; ++k) {
        uint32_t w = b0 * kCompactWords + threadIdx.x * 4 + k;
        m[k] = w < words ? fluid[w] : 0u;
        nz += m[k] ? 1u : 0u;
    }
    uint32_t tot;
    uint32_t off = red[0][0] + scan_1024(nz, &tot);
    for (int k = 0; k < 4; ++k)
        if (m[k]) seg[off++] = b0 * kCompactWords + threadIdx.x * 4 + k;
    if (!last_block || threadIdx.x != 0) return;
    ctl->seg_count[level] = red[1][0];
    if (level == 0) {
        const uint32_t f = red[2][0], lw = red[3][0];
        ctl->fluid_cells = f;
        if (f > 0 && lw > 0) {
            const uint32_t mw = fluid[lw - 1];
            ctl->last_fluid = (lw - 1) * 32u + (31u - uint32_t(__clz(mw))) + W;
        } else {
            ctl->last_fluid = 0;
        }
        ctl->pad_count = (8u - f % 8u) % 8u;
    }
}

// Smoothed density as the consumers see it: the three-pass result at fluid
// cells, the P2G density elsewhere (src/apic.rs:1649-1685 smooths fluid cells only).
__device__ __forceinline__ float smoothed_at(const float* sm, const float* dens, const uint32_t* fluid, uint32_t c) {
    return bit_at(fluid, c) ? sm[c] : dens[c];
}
// Same, for a cell index that can fall one row past the grid when a caller
// opens the solid border (the reference reads past its array there).
__device__ __forceinline__ float smoothed_guarded(const float* sm, const float* dens, const uint32_t* fluid,
                                                  uint32_t c, uint32_t cells) {
    return c < cells ? smoothed_at(sm, dens, fluid, c) : 0.0f;
}

// A tile of a grid with a halo as wide as the sweeps that one launch runs on it.
template <int kTX, int kTY, int kSweeps>
struct SweepTile {
    static constexpr int TX = kTX, TY = kTY, N = kSweeps;
    static constexpr int RX = kTX + 2 * kSweeps, RY = kTY + 2 * kSweeps;
};

// The three smoothing passes of the density over the fluid cells (src/apic.rs:
// 1649-1685) in one launch, on tiles with a halo of three in shared memory.
// A cell's neighbours are those of its flat index (the cell after a row's last
// one is the next row's first), which a staged position's are too.  Three
// launches before, each reading what the one before wrote: 128^2 11.4 -> 4.6 us,
// the build stage 308 -> 259 us at 4096^2.
template <class T>
__global__ void __launch_bounds__(256) k_smooth_density(const uint32_t* __restrict__ fluid, uint32_t W, uint32_t H,
                                                        const float* __restrict__ src, float* __restrict__ dst,
                                                        uint32_t tiles_x) {
    __shared__ float s_val[2][T::RX * T::RY];
    __shared__ uint8_t s_on[T::RX * T::RY];
    const int x0 = int(blockIdx.x % tiles_x) * T::TX - T::N, y0 = int(blockIdx.x / tiles_x) * T::TY - T::N;
    const long long cells = (long long)W * H;
    pdl_wait();
    bool some = false;
#pragma unroll 4
    for (int i = threadIdx.x; i < T::RX * T::RY; i += 256) {
        const int x = x0 + i % T::RX, y = y0 + i / T::RX;
        const long long raw = (long long)y * W + x;
        const bool in = raw >= 0 && raw < cells;
        const bool on = in && bit_at(fluid, uint32_t(raw));
        s_val[0][i] = in ? src[raw] : 0.0f;
        s_on[i] = on;
        some = some || on;
    }
    if (!__syncthreads_or(some)) return;
    int cur = 0;
#pragma unroll
    for (int n = 1; n <= T::N; ++n) {
        const int rx_n = T::RX - 2 * n, count = rx_n * (T::RY - 2 * n);
        for (int j = threadIdx.x; j < count; j += 256) {
            const int rx = n + j % rx_n, ry = n + j / rx_n, i = ry * T::RX + rx;
            if (!s_on[i]) continue;
            const float* v = s_val[cur];
            const float fl = float(s_on[i - 1]), fr = float(s_on[i + 1]);
            const float fb = float(s_on[i - T::RX]), ft = float(s_on[i + T::RX]);
            float sum = v[i] * 4.0f;
            float weight = 4.0f;
            if (fl != 0.0f) sum += v[i - 1];
            if (fr != 0.0f) sum += v[i + 1];
            if (fb != 0.0f) sum += v[i - T::RX];
            if (ft != 0.0f) sum += v[i + T::RX];
            weight += fl + fr + fb + ft;
            const float out = sum / weight;
            if (n < T::N) {
                s_val[cur ^ 1][i] = out;
            } else {
                const int x = x0 + rx, y = y0 + ry;
                if (x < int(W) && y < int(H)) dst[size_t(y) * W + x] = out;
            }
        }
        if (n < T::N) __syncthreads();
        cur ^= 1;
    }
}

__global__ void __launch_bounds__(kSegBlock) k_laplacian(const uint32_t* __restrict__ fluid,
                                                          const uint32_t* __restrict__ obstacle,
                                                          const uint32_t* __restrict__ seg, Ctl* __restrict__ ctl,
                                                          uint32_t W, uint32_t cells, float dx,
                                                          const float* __restrict__ u, const float* __restrict__ v,
                                                          const float* __restrict__ sm, const float* __restrict__ dens,
                                                          float* __restrict__ res, float* __restrict__ diag_o,
                                                          float* __restrict__ inv_o, float* __restrict__ px_o,
                                                          float* __restrict__ py_o) {
    pdl_wait();
    const uint32_t nseg = ctl->seg_count[0];
    const int lane = threadIdx.x & 31;
    const uint32_t nw = (gridDim.x * blockDim.x) >> 5;
    if (blockIdx.x == 0 && threadIdx.x == 0) ctl->res_sel = 0;  // res is written here
    const float target = 9.0f;
    const float noise = target * 1.15f;
    const float corr = 0.1f;
    for (uint32_t s = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; s < nseg; s += nw) {
        uint32_t word = seg[s];
        uint32_t bits = fluid[word];
        if (!((bits >> lane) & 1u)) continue;
        long long raw = (long long)word * 32 + lane;
        uint32_t fi = uint32_t(raw) + W;
        uint32_t gx = uint32_t(raw) % W, gy = uint32_t(raw) / W;
        uint32_t ui = gy * (W + 1) + gx;
        float ul = u[ui], ur = u[ui + 1], vb = v[raw], vt = v[raw + W];
        uint32_t nol = 1u - obstacle_raw(obstacle, raw - 1, cells), nor = 1u - obstacle_raw(obstacle, raw + 1, cells);
        uint32_t nob = 1u - obstacle_raw(obstacle, raw - (long long)W, cells);
        uint32_t not_ = 1u - obstacle_raw(obstacle, raw + (long long)W, cells);
        ul *= float(nol);
        ur *= float(nor);
        vb *= float(nob);
        vt *= float(not_);
        float div = (ur - ul) + (vt - vb);
        float rc = sm[raw];
        float excess = fminf(fmaxf(rc - noise, 0.0f), target);
        uint32_t fl = fluid_raw(fluid, raw - 1, cells), fr = fluid_raw(fluid, raw + 1, cells);
        uint32_t fb = fluid_raw(fluid, raw - (long long)W, cells), ft = fluid_raw(fluid, raw + (long long)W, cells);
        float diag = 0.0f, px = 0.0f, py = 0.0f;
        if (nol) {
            if (fl) diag += 1.0f;
            else diag += 1.0f / theta(smoothed_at(sm, dens, fluid, uint32_t(raw - 1)), rc, target);
        }
        if (nor) {
            if (fr) { diag += 1.0f; px = -1.0f; }
            else diag += 1.0f / theta(smoothed_at(sm, dens, fluid, uint32_t(raw + 1)), rc, target);
        }
        if (nob) {
            if (fb) diag += 1.0f;
            else diag += 1.0f / theta(smoothed_at(sm, dens, fluid, uint32_t(raw - W)), rc, target);
        }
        if (not_) {
            if (ft) { diag += 1.0f; py = -1.0f; }
            else diag += 1.0f / theta(smoothed_at(sm, dens, fluid, uint32_t(raw + W)), rc, target);
        }
        res[fi] = -div * dx + excess * corr * dx * dx;
        px_o[fi] = px;
        py_o[fi] = py;
        diag_o[fi] = diag;
        inv_o[fi] = diag > 1e-6f ? 1.0f / diag : 0.0f;
    }
}

// One coarse mask word of level c from its finer level f (src/apic.rs:
// 1499-1602), by one warp: lane = the word's cell; the word itself (an OR of
// each cell's 2 x 2 children) and, for the fluid cells, the coarse
// coefficients.
__device__ __forceinline__ void coarsen_word(const Level& f, const Level& c, uint32_t word, uint32_t lane) {
    const uint32_t raw = word * 32u + lane;
    bool on = false;
    // every load at once (a level with a coarser one has even sides, so a row of
    // children is a pair, inside the padded arrays and 8-byte aligned), then
    // the mask decides
    uint32_t bits[2] = {0u, 0u};
    float2 d[2], x[2], y[2];
    if (raw < c.cells) {
        uint32_t cx, cy;
        raw_xy(raw, c.w, c.wshift, cx, cy);
#pragma unroll
        for (uint32_t dy = 0; dy < 2; ++dy) {
            const uint32_t fr = (2u * cy + dy) * f.w + 2u * cx, fp = fr + f.w;
            bits[dy] = (f.fluid[fr >> 5] >> (fr & 31u)) & 3u;
            d[dy] = *reinterpret_cast<const float2*>(f.diag + fp);
            x[dy] = *reinterpret_cast<const float2*>(f.px + fp);
            y[dy] = *reinterpret_cast<const float2*>(f.py + fp);
        }
        on = (bits[0] | bits[1]) != 0u;
    }
    const uint32_t ballot = __ballot_sync(0xffffffffu, on);
    if (lane == 0) c.fluid[word] = ballot;
    if (!on) {
        // zero coefficients outside the fluid: the V-cycle's shared-memory
        // levels run over all their cells (vcycle_common.cuh)
        if (raw < c.cells) {
            c.diag[raw + c.w] = 0.0f;
            c.inv_diag[raw + c.w] = 0.0f;
            c.px[raw + c.w] = 0.0f;
            c.py[raw + c.w] = 0.0f;
        }
        return;
    }
    float diag = 0.0f, px = 0.0f, py = 0.0f;
#pragma unroll
    for (uint32_t dy = 0; dy < 2; ++dy) {
        if (bits[dy] & 1u) {
            diag += d[dy].x;
            diag += 2.0f * x[dy].x;
            if (dy == 0) diag += 2.0f * y[dy].x;
            if (dy == 1) py += y[dy].x;
        }
        if (bits[dy] & 2u) {
            diag += d[dy].y;
            if (dy == 0) diag += 2.0f * y[dy].y;
            px += x[dy].y;
            if (dy == 1) py += y[dy].y;
        }
    }
    uint32_t cp = raw + c.w;
    float fd = diag * 0.5f;
    c.diag[cp] = fd;
    c.inv_diag[cp] = fd > 1e-6f ? 1.0f / fd : 0.0f;
    c.px[cp] = px * 0.5f;
    c.py[cp] = py * 0.5f;
}

// The same zeros on a coarsest level whose mask or coefficients a caller wrote
// (padding included), and no coupling from a fluid cell to one that is not: its
// CG runs over all cells too.
__global__ void __launch_bounds__(256) k_mask_level(Level c) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= c.padded) return;
    const long long raw = (long long)i - c.w;
    const bool on = fluid_raw(c.fluid, raw, c.cells) != 0;
    if (!on) {
        c.diag[i] = 0.0f;
        c.inv_diag[i] = 0.0f;
    }
    if (!on || !fluid_raw(c.fluid, raw + 1, c.cells)) c.px[i] = 0.0f;
    if (!on || !fluid_raw(c.fluid, raw + c.w, c.cells)) c.py[i] = 0.0f;
}

// One coarse level from its finer level: one warp per coarse mask word.
__global__ void __launch_bounds__(256) k_coarsen(Level f, Level c) {
    pdl_wait();
    const uint32_t word = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (word >= c.words) return;  // whole warps exit together
    coarsen_word(f, c, word, threadIdx.x & 31u);
}

// Segment list of one coarse level by one CTA of kOneThreads threads (levels
// of at most kOneWords mask words): thread t takes the consecutive words
// [t k, t k + k), so a block scan of the per-thread counts gives every
// non-zero word its place in ascending order.
constexpr uint32_t kOneThreads = 1024;
constexpr uint32_t kOneWords = 8192;
__device__ __forceinline__ void compact_one(const uint32_t* __restrict__ fluid, uint32_t words, uint32_t* __restrict__ seg,
                                            int level, Ctl* __restrict__ ctl) {
    const uint32_t per = (words + kOneThreads - 1) / kOneThreads;
    const uint32_t w0 = threadIdx.x * per;
    uint32_t nz = 0;
    for (uint32_t k = 0; k < per; ++k)
        if (w0 + k < words && fluid[w0 + k]) ++nz;
    uint32_t tot;
    uint32_t off = scan_1024(nz, &tot);
    for (uint32_t k = 0; k < per; ++k)
        if (w0 + k < words && fluid[w0 + k]) seg[off++] = w0 + k;
    if (threadIdx.x == 0) ctl->seg_count[level] = tot;
}

__global__ void __launch_bounds__(kOneThreads) k_compact_one(const uint32_t* __restrict__ fluid, uint32_t words,
                                                              uint32_t* __restrict__ seg, int level, Ctl* __restrict__ ctl) {
    pdl_wait();
    compact_one(fluid, words, seg, level, ctl);
}

// The base level's list by one CTA (up to kOneWords mask words: 512^2 cells),
// with what k_compact_count and k_compact_write do besides: the mask cleaned of
// obstacles, the totals, the last fluid cell.
__global__ void __launch_bounds__(kOneThreads) k_compact_base(uint32_t* __restrict__ fluid,
                                                               const uint32_t* __restrict__ obstacle, uint32_t words,
                                                               uint32_t* __restrict__ seg, uint32_t W,
                                                               Ctl* __restrict__ ctl) {
    constexpr uint32_t kPer = kOneWords / kOneThreads;
    __shared__ uint32_t s_cells[kOneThreads / 32], s_last[kOneThreads / 32];
    pdl_wait();
    const uint32_t per = (words + kOneThreads - 1) / kOneThreads, w0 = threadIdx.x * per;
    uint32_t m[kPer], nz = 0, cells = 0, last = 0;  // last: the last fluid cell, one up
#pragma unroll
    for (uint32_t k = 0; k < kPer; ++k)
        m[k] = k < per ? load_clean_word(fluid, obstacle, w0 + k, words, true) : 0u;
#pragma unroll
    for (uint32_t k = 0; k < kPer; ++k) {
        if (!m[k]) continue;
        ++nz;
        cells += uint32_t(__popc(m[k]));
        last = (w0 + k) * 32u + 32u - uint32_t(__clz(m[k]));
    }
    uint32_t tot;
    uint32_t off = scan_1024(nz, &tot);
#pragma unroll
    for (uint32_t k = 0; k < kPer; ++k)
        if (m[k]) seg[off++] = w0 + k;
    cells = __reduce_add_sync(0xffffffffu, cells);
    last = __reduce_max_sync(0xffffffffu, last);
    if ((threadIdx.x & 31u) == 0) {
        s_cells[threadIdx.x >> 5] = cells;
        s_last[threadIdx.x >> 5] = last;
    }
    __syncthreads();
    if (threadIdx.x >= 32) return;
    cells = __reduce_add_sync(0xffffffffu, s_cells[threadIdx.x]);
    last = __reduce_max_sync(0xffffffffu, s_last[threadIdx.x]);
    if (threadIdx.x != 0) return;
    ctl->seg_count[0] = tot;
    ctl->fluid_cells = cells;
    ctl->last_fluid = last > 0 ? last - 1u + W : 0u;
    ctl->pad_count = (8u - cells % 8u) % 8u;
}

// The smallest levels, [first, n), by one CTA: a level's coarsening by a warp
// per mask word, with a CTA barrier between levels, then every level's
// segment list by a warp of its own.  What it takes is the latency of each
// level's loads and stores, one after another (128^2 scene, four levels: 18.0
// -> 9.3 us against lists between the levels and loads behind their masks).
constexpr uint32_t kTailWords = 128;  // mask words of a level here at most
constexpr uint32_t kTailTileGroups = 64;
struct TailLevels {
    int first, n;
    int tiles;  // the tile lists too
    Level lv[kMaxLevels];
};
// Whether one of the tile's cells is fluid.
__device__ __forceinline__ bool tile_holds_fluid(const Level& L, uint32_t i) {
    const uint32_t x0 = (i % L.tiles_x) * kTileX, y0 = (i / L.tiles_x) * kTileY;
    const uint32_t rows = min(kTileY, L.h - y0), n = min(kTileX, L.w - x0);
    const uint32_t mask = n >= 32u ? 0xffffffffu : (1u << n) - 1u;
    uint32_t any = 0;
#pragma unroll 8
    for (uint32_t y = 0; y < rows; ++y) {
        const uint32_t raw = (y0 + y) * L.w + x0, sh = raw & 31u;
        uint32_t bits = L.fluid[raw >> 5] >> sh;
        if (sh && (raw >> 5) + 1u < L.words) bits |= L.fluid[(raw >> 5) + 1u] << (32u - sh);
        any |= bits & mask;
    }
    return any != 0;
}
__global__ void __launch_bounds__(kOneThreads) k_coarsen_tail(TailLevels t, Ctl* __restrict__ ctl) {
    pdl_wait();
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
    for (int l = t.first; l < t.n; ++l) {
        const Level& f = t.lv[l - 1];
        const Level& c = t.lv[l];
        for (uint32_t w = warp; w < c.words; w += kOneThreads / 32u) coarsen_word(f, c, w, lane);
        __syncthreads();
    }
    if (t.tiles) {
        // groups of 32 tiles over the levels with a coarser one, a warp each:
        // which hold fluid, then each group's place behind those before it
        __shared__ uint32_t s_votes[kTailTileGroups];
        uint32_t g0 = 0;
        for (int l = 0; l + 1 < t.n; ++l) {
            const uint32_t ntiles = t.lv[l].ntiles, groups = (ntiles + 31u) / 32u;
            for (uint32_t g = (warp - g0) & 31u; g < groups; g += 32u) {
                const uint32_t i = 32u * g + lane;
                const uint32_t votes = __ballot_sync(0xffffffffu, i < ntiles && tile_holds_fluid(t.lv[l], i));
                if (lane == 0) s_votes[g0 + g] = votes;
            }
            g0 += groups;
        }
        __syncthreads();
        g0 = 0;
        for (int l = 0; l + 1 < t.n; ++l) {
            const uint32_t groups = (t.lv[l].ntiles + 31u) / 32u;
            for (uint32_t g = (warp - g0) & 31u; g < groups; g += 32u) {
                const uint32_t votes = s_votes[g0 + g];
                uint32_t before = 0;
                for (uint32_t k = lane; k < g; k += 32u) before += uint32_t(__popc(s_votes[g0 + k]));
                before = __reduce_add_sync(0xffffffffu, before);
                if ((votes >> lane) & 1u)
                    t.lv[l].tiles[before + uint32_t(__popc(votes & ((1u << lane) - 1u)))] = 32u * g + lane;
                if (g + 1u == groups && lane == 0) ctl->tile_count[l] = before + uint32_t(__popc(votes));
            }
            g0 += groups;
        }
    }
    const int l = t.first + int(warp);
    if (l >= t.n) return;
    const Level& c = t.lv[l];
    uint32_t m[kTailWords / 32u];
#pragma unroll
    for (uint32_t k = 0; k < kTailWords / 32u; ++k) m[k] = 32u * k + lane < c.words ? c.fluid[32u * k + lane] : 0u;
    uint32_t count = 0;
#pragma unroll
    for (uint32_t k = 0; k < kTailWords / 32u; ++k) {
        const uint32_t some = __ballot_sync(0xffffffffu, m[k] != 0u);
        if (m[k]) c.seg[count + uint32_t(__popc(some & ((1u << lane) - 1u)))] = 32u * k + lane;
        count += uint32_t(__popc(some));
    }
    if (lane == 0) ctl->seg_count[l] = count;
}

// The ascending list of a level's tiles that hold fluid, one CTA per level
// (blockIdx.x): thread t of a round takes tile 1024 * round + t and ORs the
// 32 bits of its rows, or, on a large level, reads the flag that a grid-wide
// kernel formed (4096^2, 32768 tiles: 200 us by one CTA alone).
struct TileLists {
    int n;
    Level lv[kMaxLevels];
};
__global__ void __launch_bounds__(256) k_tile_flags(Level L) {
    pdl_wait();
    const uint32_t i = blockIdx.x * 256u + threadIdx.x;
    const uint32_t votes = __ballot_sync(0xffffffffu, i < L.ntiles && tile_holds_fluid(L, i));
    if ((threadIdx.x & 31u) == 0 && i < L.ntiles) L.tile_flags[i >> 5] = votes;
}
__global__ void __launch_bounds__(kOneThreads) k_tile_lists(TileLists t, Ctl* __restrict__ ctl) {
    pdl_wait();
    const Level& L = t.lv[blockIdx.x];
    uint32_t count = 0;
    for (uint32_t i0 = 0; i0 < L.ntiles; i0 += kOneThreads) {
        const uint32_t i = i0 + threadIdx.x;
        const bool any = i < L.ntiles && (L.tile_flags ? (L.tile_flags[i >> 5] >> (i & 31u)) & 1u : tile_holds_fluid(L, i));
        uint32_t tot;
        const uint32_t off = scan_1024(any ? 1u : 0u, &tot);
        if (any) L.tiles[count + off] = i;
        count += tot;
    }
    if (threadIdx.x == 0) ctl->tile_count[blockIdx.x] = count;
}

__global__ void __launch_bounds__(256) k_gradient(uint32_t uf, uint32_t vf, int W, int H, float inv_dx,
                                                  float* __restrict__ u, float* __restrict__ v,
                                                  uint8_t* __restrict__ valid_u, uint8_t* __restrict__ valid_v,
                                                  const uint32_t* __restrict__ fluid,
                                                  const uint32_t* __restrict__ obstacle,
                                                  const float* __restrict__ p, const float* __restrict__ sm,
                                                  const float* __restrict__ dens, const float* __restrict__ post_u,
                                                  const float* __restrict__ post_v, const Ctl* __restrict__ ctl,
                                                  const double* __restrict__ p64, int do_gradient, int do_post) {
    pdl_wait();
    uint32_t f = blockIdx.x * blockDim.x + threadIdx.x;
    if (f >= uf + vf) return;
    const float target = 9.0f;
    const uint32_t cells = uint32_t(W) * uint32_t(H);
    const bool post = do_post && ctl->has_post;
    if (f < uf) {
        int x = int(f % uint32_t(W + 1)), y = int(f / uint32_t(W + 1));
        float val = u[f];
        if (do_gradient) {
            uint32_t lo = obstacle_xy(obstacle, x - 1, y, W, H), ro = obstacle_xy(obstacle, x, y, W, H);
            if (lo != ro) {
                val = 0.0f;
                valid_u[f] = 1;
            } else {
                uint32_t lf = fluid_xy(fluid, x - 1, y, W, H), rf = fluid_xy(fluid, x, y, W, H);
                float dp = 0.0f;
                uint32_t li = uint32_t(y * W + x - 1), ri = uint32_t(y * W + x);
                if (p64) {
                    // mixed precision: differences of the FP64 refined pressure
                    double d = 0.0;
                    if (lf && rf) d = p64[ri + W] - p64[li + W];
                    else if (lf) d = -p64[li + W] / double(theta(smoothed_guarded(sm, dens, fluid, ri, cells), sm[li], target));
                    else if (rf) d = p64[ri + W] / double(theta(smoothed_guarded(sm, dens, fluid, li, cells), sm[ri], target));
                    val -= float(d * double(inv_dx));
                } else {
                    if (lf && rf) dp = p[ri] - p[li];
                    else if (lf) dp = -p[li] / theta(smoothed_guarded(sm, dens, fluid, ri, cells), sm[li], target);
                    else if (rf) dp = p[ri] / theta(smoothed_guarded(sm, dens, fluid, li, cells), sm[ri], target);
                    val -= dp * inv_dx;
                }
            }
        }
        if (post) val += post_u[f] * ctl->dt;
        u[f] = val;
    } else {
        uint32_t g = f - uf;
        int x = int(g % uint32_t(W)), y = int(g / uint32_t(W));
        float val = v[g];
        if (do_gradient) {
            uint32_t bo = obstacle_xy(obstacle, x, y - 1, W, H), to = obstacle_xy(obstacle, x, y, W, H);
            if (bo != to) {
                val = 0.0f;
                valid_v[g] = 1;
            } else {
                uint32_t bf = fluid_xy(fluid, x, y - 1, W, H), tf = fluid_xy(fluid, x, y, W, H);
                float dp = 0.0f;
                uint32_t bi = uint32_t((y - 1) * W + x), ti = uint32_t(y * W + x);
                if (p64) {
                    double d = 0.0;
                    if (bf && tf) d = p64[ti + W] - p64[bi + W];
                    else if (bf) d = -p64[bi + W] / double(theta(smoothed_guarded(sm, dens, fluid, ti, cells), sm[bi], target));
                    else if (tf) d = p64[ti + W] / double(theta(smoothed_guarded(sm, dens, fluid, bi, cells), sm[ti], target));
                    val -= float(d * double(inv_dx));
                } else {
                    if (bf && tf) dp = p[ti] - p[bi];
                    else if (bf) dp = -p[bi] / theta(smoothed_guarded(sm, dens, fluid, ti, cells), sm[bi], target);
                    else if (tf) dp = p[ti] / theta(smoothed_guarded(sm, dens, fluid, bi, cells), sm[ti], target);
                    val -= dp * inv_dx;
                }
            }
        }
        if (post) val += post_v[g] * ctl->dt;
        v[g] = val;
    }
}

// Velocity extrapolation: the four Jacobi sweeps of src/apic.rs:2266-2350 (it
// swaps buffers after each) on tiles of one face field (u: (W+1) x H, v: W x
// (H+1)) with a halo as wide as the sweeps of a launch, in shared memory; each
// sweep runs on a region one face smaller on each side than the one before,
// the last one on the tile, which is written out.  A neighbour outside the
// field reads as invalid, which is exactly the reference's x > 0 / x < width /
// y > 0 / y < height guards, and every face adds its valid neighbours in the
// reference's order (x-1, x+1, y-1, y+1) before the one division, so each
// sweep's values and flags are bit-identical to a sweep over the whole grid.
// A tile whose staged faces are all valid, or all invalid, is what the sweeps
// would leave it as: most of a large grid.
struct ExField {
    const float* in;
    const uint8_t* in_ok;
    float* out;
    uint8_t* out_ok;
    int w, h;          // faces per row, rows
    int tiles_x;       // tiles per row of tiles
};

template <int kRX>
__device__ __forceinline__ void ex_face(const float* val, const uint8_t* ok, int i, float* nv, uint8_t* nok) {
    if (ok[i]) { *nv = val[i]; *nok = 1; return; }
    float sum = 0.0f;
    uint32_t cnt = 0;
    if (ok[i - 1]) { sum += val[i - 1]; cnt++; }
    if (ok[i + 1]) { sum += val[i + 1]; cnt++; }
    if (ok[i - kRX]) { sum += val[i - kRX]; cnt++; }
    if (ok[i + kRX]) { sum += val[i + kRX]; cnt++; }
    if (cnt > 0) { *nv = sum / float(cnt); *nok = 1; }
    else { *nv = val[i]; *nok = 0; }
}

template <class T>
__global__ void __launch_bounds__(256) k_extrapolate(ExField fu, ExField fv, int tiles_u) {
    __shared__ float s_val[2][T::RX * T::RY];
    __shared__ uint8_t s_ok[2][T::RX * T::RY];
    const bool is_u = int(blockIdx.x) < tiles_u;
    const ExField& F = is_u ? fu : fv;
    const int t = is_u ? int(blockIdx.x) : int(blockIdx.x) - tiles_u;
    const int x0 = (t % F.tiles_x) * T::TX - T::N, y0 = (t / F.tiles_x) * T::TY - T::N;
    pdl_wait();
    bool some = false, all = true;  // of the staged faces inside the field: valid
#pragma unroll 4
    for (int i = threadIdx.x; i < T::RX * T::RY; i += 256) {
        const int gx = x0 + i % T::RX, gy = y0 + i / T::RX;
        float v = 0.0f;
        uint8_t k = 0;
        if (gx >= 0 && gx < F.w && gy >= 0 && gy < F.h) {
            const size_t g = size_t(gy) * F.w + gx;
            v = F.in[g];
            k = F.in_ok[g] != 0;  // (a caller may have written any byte; a sweep writes 1)
            some = some || k;
            all = all && k;
        }
        s_val[0][i] = v;
        s_ok[0][i] = k;
    }
    const bool mixed = __syncthreads_or(some) && !__syncthreads_and(all);
    int cur = 0;
    if (mixed) {
#pragma unroll
        for (int n = 1; n < T::N; ++n) {
            // faces outside the field stay invalid
            const int rx_n = T::RX - 2 * n, cells = rx_n * (T::RY - 2 * n);
            for (int j = threadIdx.x; j < cells; j += 256) {
                const int rx = n + j % rx_n, ry = n + j / rx_n, i = ry * T::RX + rx;
                const int gx = x0 + rx, gy = y0 + ry;
                float v = 0.0f;
                uint8_t k = 0;
                if (gx >= 0 && gx < F.w && gy >= 0 && gy < F.h) ex_face<T::RX>(s_val[cur], s_ok[cur], i, &v, &k);
                s_val[cur ^ 1][i] = v;
                s_ok[cur ^ 1][i] = k;
            }
            __syncthreads();
            cur ^= 1;
        }
    }
    for (int j = threadIdx.x; j < T::TX * T::TY; j += 256) {
        const int rx = T::N + j % T::TX, ry = T::N + j / T::TX, i = ry * T::RX + rx;
        const int gx = x0 + rx, gy = y0 + ry;
        if (gx >= F.w || gy >= F.h) continue;
        float v = s_val[cur][i];
        uint8_t k = s_ok[cur][i];
        if (mixed) ex_face<T::RX>(s_val[cur], s_ok[cur], i, &v, &k);
        const size_t g = size_t(gy) * F.w + gx;
        F.out[g] = v;
        F.out_ok[g] = k;
    }
}

__global__ void __launch_bounds__(256) k_smoothed_view(uint32_t cells, const float* __restrict__ sm,
                                                       const float* __restrict__ dens,
                                                       const uint32_t* __restrict__ fluid, float* __restrict__ out) {
    uint32_t c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c < cells) out[c] = smoothed_at(sm, dens, fluid, c);
}

}  // namespace

uint32_t seg_grid(uint32_t words) {
    uint32_t b = div_up(words, kSegWarps);
    // Levels of up to 2 M cells are latency bound: four CTAs per SM (fewer
    // block partials for the next kernel to sum) beat eight by 2% per PCG
    // iteration at 1024^2; a 4096^2 base level needs every warp slot for
    // bandwidth (eight: 955 vs 1206 us per iteration).
    const uint32_t cap = words <= 65536u ? uint32_t(kMaxRedBlocks) / 2u : uint32_t(kMaxRedBlocks);
    if (b > cap) b = cap;
    return b ? b : 1;
}

cudaError_t launch_finalize_faces(Scene& s, bool forces, bool gravity) {
    uint32_t nf = s.uf + s.vf;
    launch(s.use_pdl, k_faces, div_up(nf, 256), 256, 0, s.stream, s.uf, s.vf, int(s.W), int(s.H), s.acc_u, s.acc_uw, s.acc_v,
                                                    s.acc_vw, s.u, s.v, s.valid_u, s.valid_v, s.ext_u, s.ext_v,
                                                    s.lv[0].fluid, s.obstacle, s.ctl, s.props.gravity, 1,
                                                    forces ? 1 : 0, gravity ? 1 : 0);
    return cudaGetLastError();
}

cudaError_t launch_external_forces(Scene& s) {
    uint32_t nf = s.uf + s.vf;
    launch(s.use_pdl, k_faces, div_up(nf, 256), 256, 0, s.stream, s.uf, s.vf, int(s.W), int(s.H), s.acc_u, s.acc_uw, s.acc_v,
                                                    s.acc_vw, s.u, s.v, s.valid_u, s.valid_v, s.ext_u, s.ext_v,
                                                    s.lv[0].fluid, s.obstacle, s.ctl, s.props.gravity, 0, 1, 1);
    return cudaGetLastError();
}

static cudaError_t compact_level(Scene& s, int level, const uint32_t* obstacle) {
    Level& L = s.lv[level];
    if (level > 0 && L.words <= kOneWords) {
        launch(s.use_pdl, k_compact_one, 1, kOneThreads, 0, s.stream, static_cast<const uint32_t*>(L.fluid), L.words,
               L.seg, level, s.ctl);
        return cudaGetLastError();
    }
    if (L.words <= kOneWords) {
        launch(s.use_pdl, k_compact_base, 1, kOneThreads, 0, s.stream, L.fluid, obstacle, L.words, L.seg, L.w, s.ctl);
        return cudaGetLastError();
    }
    uint32_t nb = div_up(L.words, kCompactWords);
    if (nb == 0) nb = 1;  // the last block records the (empty) level's totals
    launch(s.use_pdl, k_compact_count, nb, 256, 0, s.stream, L.fluid, obstacle, L.words, s.scan_tmp);
    launch(s.use_pdl, k_compact_write, nb, 256, 0, s.stream, static_cast<const uint32_t*>(L.fluid), L.words,
           static_cast<const uint32_t*>(s.scan_tmp), L.seg, L.w, level, s.ctl);
    return cudaGetLastError();
}

cudaError_t launch_mask_level(Scene& s, int level) {
    k_mask_level<<<div_up(s.lv[level].padded, 256), 256, 0, s.stream>>>(s.lv[level]);
    return cudaGetLastError();
}
// Every level that the V-cycle's tile kernels may work on (those with a
// coarser one).
cudaError_t launch_tile_lists(Scene& s) {
    TileLists t;
    t.n = s.nlevels - 1;
    if (t.n < 1) return cudaSuccess;
    for (int l = 0; l < t.n; ++l) {
        t.lv[l] = s.lv[l];
        if (s.lv[l].tile_flags)
            launch(s.use_pdl, k_tile_flags, div_up(s.lv[l].ntiles, 256), 256, 0, s.stream, s.lv[l]);
    }
    launch(s.use_pdl, k_tile_lists, t.n, kOneThreads, 0, s.stream, t, s.ctl);
    return cudaGetLastError();
}
cudaError_t launch_base_lists(Scene& s) { return compact_level(s, 0, s.obstacle); }
cudaError_t launch_level_lists(Scene& s, int level) { return compact_level(s, level, nullptr); }

template <class T> static void smooth_density(Scene& s) {
    const uint32_t tiles_x = div_up(s.W, T::TX);
    launch(s.use_pdl, k_smooth_density<T>, tiles_x * div_up(s.H, T::TY), 256, 0, s.stream,
           static_cast<const uint32_t*>(s.lv[0].fluid), s.W, s.H, static_cast<const float*>(s.density), s.sm_a, tiles_x);
}

cudaError_t launch_build_pressure(Scene& s) {
    const Level& B = s.lv[0];
    uint32_t g = seg_grid(B.words);
    if (s.cells <= 512u * 512u) smooth_density<SweepTile<32, 8, 3>>(s);
    else smooth_density<SweepTile<64, 16, 3>>(s);
    launch(s.use_pdl, k_laplacian, g, kSegBlock, 0, s.stream, B.fluid, s.obstacle, B.seg, s.ctl, s.W, s.cells, s.dx, s.u, s.v,
                                               s.sm_a, s.density, B.res, B.diag, B.inv_diag, B.px, B.py);
    return cudaGetLastError();
}

// Levels of at most kTailWords mask words (4096 cells: 64^2 and below) are
// built together by one CTA; each larger level by a coarsening launch and
// its segment list.
cudaError_t launch_multilevel(Scene& s) {
    int l = 1;
    for (; l < s.nlevels && s.lv[l].words > kTailWords; ++l) {
        Level& c = s.lv[l];
        launch(s.use_pdl, k_coarsen, div_up(uint64_t(c.words) * 32, 256), 256, 0, s.stream, s.lv[l - 1], c);
        cudaError_t e = compact_level(s, l, nullptr);
        if (e != cudaSuccess) return e;
    }
    if (l < s.nlevels) {
        TailLevels t;
        t.first = l;
        t.n = s.nlevels;
        uint32_t groups = 0;
        for (int k = 0; k < s.nlevels; ++k) {
            t.lv[k] = s.lv[k];
            if (k + 1 < s.nlevels) groups += div_up(s.lv[k].ntiles, 32);
        }
        // up to 512^2 cells: a launch less
        t.tiles = groups <= kTailTileGroups ? 1 : 0;
        launch(s.use_pdl, k_coarsen_tail, 1, kOneThreads, 0, s.stream, t, s.ctl);
        if (t.tiles) return cudaGetLastError();
    }
    return launch_tile_lists(s);
}

cudaError_t launch_gradient(Scene& s, bool post) {
    uint32_t nf = s.uf + s.vf;
    launch(s.use_pdl, k_gradient, div_up(nf, 256), 256, 0, s.stream, s.uf, s.vf, int(s.W), int(s.H), 1.0f / s.dx, s.u, s.v,
                                                       s.valid_u, s.valid_v, s.lv[0].fluid, s.obstacle, s.pressure,
                                                       s.sm_a, s.density, s.post_u, s.post_v, s.ctl,
                                                       s.p64_valid ? s.p64 : nullptr, 1, post ? 1 : 0);
    return cudaGetLastError();
}

cudaError_t launch_post_forces(Scene& s) {
    uint32_t nf = s.uf + s.vf;
    launch(s.use_pdl, k_gradient, div_up(nf, 256), 256, 0, s.stream, s.uf, s.vf, int(s.W), int(s.H), 1.0f / s.dx, s.u, s.v,
                                                       s.valid_u, s.valid_v, s.lv[0].fluid, s.obstacle, s.pressure,
                                                       s.sm_a, s.density, s.post_u, s.post_v, s.ctl, nullptr,
                                                       0, 1);
    return cudaGetLastError();
}

template <class T> static void extrapolate(Scene& s, bool from_alt) {
    const int W = int(s.W), H = int(s.H);
    auto field = [](const float* in, const uint8_t* in_ok, float* out, uint8_t* out_ok, int w, int h) {
        return ExField{in, in_ok, out, out_ok, w, h, int(div_up(uint32_t(w), T::TX))};
    };
    const ExField fu = from_alt ? field(s.u_alt, s.valid_u_alt, s.u, s.valid_u, W + 1, H)
                                : field(s.u, s.valid_u, s.u_alt, s.valid_u_alt, W + 1, H);
    const ExField fv = from_alt ? field(s.v_alt, s.valid_v_alt, s.v, s.valid_v, W, H + 1)
                                : field(s.v, s.valid_v, s.v_alt, s.valid_v_alt, W, H + 1);
    const uint32_t tiles_u = uint32_t(fu.tiles_x) * div_up(uint32_t(fu.h), T::TY);
    const uint32_t tiles_v = uint32_t(fv.tiles_x) * div_up(uint32_t(fv.h), T::TY);
    launch(s.use_pdl, k_extrapolate<T>, tiles_u + tiles_v, 256, 0, s.stream, fu, fv, int(tiles_u));
}

// The reference's four sweeps as two launches of two sweeps each:
// u, v -> u_alt, v_alt -> u, v (the result ends where the next stages read it).
// Up to 512^2 cells the grid's tiles are few and a tile's rounds set the time:
// 32 x 8 tiles, three rounds a sweep; above, the halo's share of the traffic
// does: 64 x 16.  The four sweeps, 32 x 8 / 64 x 16 / 128 x 24 (every size before):
// 64^2 9.5 / 13.6 / 22.3 us, 256^2 10.5 / 15.7 / 26.8, 512^2 15.4 / 16.3 / 27.9,
// 1024^2 34.8 / 27.7 / 37.4, 4096^2 (noise) 510 / 348 / 350.
cudaError_t launch_extrapolate(Scene& s) {
    if (s.cells <= 512u * 512u) {
        extrapolate<SweepTile<32, 8, 2>>(s, false);
        extrapolate<SweepTile<32, 8, 2>>(s, true);
    } else {
        extrapolate<SweepTile<64, 16, 2>>(s, false);
        extrapolate<SweepTile<64, 16, 2>>(s, true);
    }
    return cudaGetLastError();
}

cudaError_t launch_smoothed_view(Scene& s, float* out) {
    k_smoothed_view<<<div_up(s.cells, 256), 256, 0, s.stream>>>(s.cells, s.sm_a, s.density, s.lv[0].fluid, out);
    return cudaGetLastError();
}

}  // namespace apic
