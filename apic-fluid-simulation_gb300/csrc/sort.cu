// sort.cu — Morton keys, stable LSD radix sort, particle permutation.
//
// Restates Apic::update_spatial_lookup (src/apic.rs:1043-1111): key = Morton
// code of the particle's clamped cell (:1049-1064), sort of (key, val = slot)
// pairs (:1066, rdst radix_sort_unstable over 4 x 8-bit levels, :220-227), then
// a gather of the nine particle fields by `val` with the tail lanes of the last
// chunk zero-filled (:1068-1104).  The reference leaves the order of equal keys
// to rdst; this sort is stable (equal keys keep ascending `val`), which is the
// order the oracle defines.
//
// One kernel counts every digit of the keys (k_sort_prepare); then a pass over
// one digit of up to 10 bits is one kernel (k_sort_pass) that reads each pair
// once and writes it once.  A tile ranks its keys stably with
// __match_any_sync, publishes its count of each digit value, and finds its
// place behind the tiles before it by adding up what they published
// ("decoupled look-back", Merrill and Garland, "Single-pass Parallel Prefix
// Scan with Decoupled Look-back", 2016, and its use in radix sorting by
// Adinets and Merrill, "Onesweep", 2022): a tile that knows its own place
// publishes the running total, so later tiles stop there.  Tiles take their
// numbers from a counter as they start, so a tile only waits for tiles that
// are running or done; the wait is bounded all the same, and a tile whose wait
// runs out counts the keys before it.  Only the bits below
// the bit length of the largest possible key are sorted: higher bits are zero
// for every key, so their passes would be identities.  The digit width is
// chosen per sort for the fewest passes (20-bit keys of a 1024^2 grid: two
// 10-bit passes), and the sorted pairs stay in the buffer the last pass wrote.
#include <cuda_runtime.h>

#include <algorithm>

#include "apic_device.cuh"
#include "apic_internal.h"

namespace apic {

namespace {

constexpr uint32_t kMaxBuckets = 1u << kMaxDigitBits;
constexpr int kSortThreads = 512;
constexpr int kSortWarps = kSortThreads / 32;
// Scratch words in front of the tiles' published counts: every digit's
// histogram (passes * buckets <= 3072) and a tile counter per pass.
constexpr uint32_t kSortHead = kSortHeadWords;
// A published count: the tile's own, with bit 31 the total up to and with it.
constexpr uint32_t kNotReady = 0xFFFFFFFFu, kInclusive = 0x80000000u;
constexpr int kLookback = 8;             // earlier tiles read at once
// Rounds of reads before a tile stops waiting and counts the keys before it
// itself (some 50 ms; a macro so that a test can let every wait run out).
#ifndef APIC_SORT_SPIN_LIMIT
#define APIC_SORT_SPIN_LIMIT (1u << 16)
#endif
constexpr uint32_t kSpinLimit = APIC_SORT_SPIN_LIMIT;

// Four particles per thread with 16-byte loads and stores: the particle
// arrays and the key buffers hold npad (a multiple of 8) lanes, so lanes
// n .. npad-1 get keys too, which the sort of n pairs never reads.  (The
// slots need no array: the first pass makes them up.)
__global__ void __launch_bounds__(256) k_morton_keys(const PartPtrs* __restrict__ pp, uint32_t n, CellSize cs, float max_x,
                                                     float max_y, uint32_t* __restrict__ keys,
                                                     uint32_t* __restrict__ head) {
    pdl_wait();
    clear_sort_head(head);
    const uint32_t i0 = 4u * (blockIdx.x * blockDim.x + threadIdx.x);
    if (i0 >= n) return;
    const float4 px = *reinterpret_cast<const float4*>(pp->f[PX] + i0);
    const float4 py = *reinterpret_cast<const float4*>(pp->f[PY] + i0);
    const float xs[4] = {px.x, px.y, px.z, px.w}, ys[4] = {py.x, py.y, py.z, py.w};
    uint32_t k[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const float gx = over_dx(xs[q], cs), gy = over_dx(ys[q], cs);  // Vec2x8 / f32x8: per-component division
        const uint32_t cx = uint32_t(trunc_x86(fmin_x86(fmax_x86(gx, 0.0f), max_x)));
        const uint32_t cy = uint32_t(trunc_x86(fmin_x86(fmax_x86(gy, 0.0f), max_y)));
        k[q] = morton(cx, cy);
    }
    *reinterpret_cast<uint4*>(keys + i0) = make_uint4(k[0], k[1], k[2], k[3]);
}

// Counts of every digit value of every pass, and the published counts' start
// value.  Keys come in nearly sorted order: a thread takes eight consecutive
// ones and adds a run of equal digits at once, and a warp whose threads all
// end with the same digit (the high ones) adds it once (a key at a time,
// 8.3 M keys took 43 us).
constexpr uint32_t kCountKeys = 8;
__global__ void __launch_bounds__(kSortThreads) k_sort_prepare(const uint32_t* __restrict__ keys, uint32_t n,
                                                               int passes, int dbits, uint32_t* __restrict__ head,
                                                               uint32_t state_words) {
    __shared__ uint32_t h[kMaxBuckets * 3];
    pdl_wait();
    const uint32_t nbk = 1u << dbits, mask = nbk - 1u, lane = threadIdx.x & 31u;
    for (uint32_t d = threadIdx.x; d < uint32_t(passes) * nbk; d += kSortThreads) h[d] = 0;
    uint4* state = reinterpret_cast<uint4*>(head + kSortHead);
    for (uint32_t i = blockIdx.x * kSortThreads + threadIdx.x; i < (state_words + 3u) / 4u;
         i += gridDim.x * kSortThreads)
        state[i] = make_uint4(kNotReady, kNotReady, kNotReady, kNotReady);
    __syncthreads();
    const bool aligned = (reinterpret_cast<uintptr_t>(keys) & 15u) == 0;  // a caller's buffer may not be
    const uint64_t step = uint64_t(gridDim.x) * kSortThreads * kCountKeys;
    // (whole warps stay in the loop: the vote below is the warp's)
    for (uint64_t w0 = (uint64_t(blockIdx.x) * kSortThreads + (threadIdx.x & ~31u)) * kCountKeys; w0 < n; w0 += step) {
        const uint64_t i0 = w0 + lane * kCountKeys;
        uint32_t k[kCountKeys];
        uint32_t live = 0;
        if (i0 + kCountKeys <= n && aligned) {
            const uint4 a = *reinterpret_cast<const uint4*>(keys + i0), b = *reinterpret_cast<const uint4*>(keys + i0 + 4);
            k[0] = a.x; k[1] = a.y; k[2] = a.z; k[3] = a.w;
            k[4] = b.x; k[5] = b.y; k[6] = b.z; k[7] = b.w;
            live = kCountKeys;
        } else {
#pragma unroll
            for (uint32_t j = 0; j < kCountKeys; ++j) {
                const bool ok = i0 + j < n;
                k[j] = ok ? keys[i0 + j] : 0u;
                live += ok ? 1u : 0u;
            }
        }
        for (int p = 0; p < passes; ++p) {
            uint32_t* hp = h + uint32_t(p) * nbk;
            uint32_t cur = (k[0] >> (p * dbits)) & mask, run = live > 0 ? 1u : 0u;
#pragma unroll
            for (uint32_t j = 1; j < kCountKeys; ++j) {
                const uint32_t d = (k[j] >> (p * dbits)) & mask;
                if (j < live && d != cur) {
                    atomicAdd(&hp[cur], run);
                    cur = d;
                    run = 0;
                }
                run += j < live ? 1u : 0u;
            }
            int same;
            __match_all_sync(0xffffffffu, cur, &same);
            if (same) {
                const uint32_t all = __reduce_add_sync(0xffffffffu, run);
                if (lane == 0) atomicAdd(&hp[cur], all);
            } else if (run) {
                atomicAdd(&hp[cur], run);
            }
        }
    }
    __syncthreads();
    for (uint32_t d = threadIdx.x; d < uint32_t(passes) * nbk; d += kSortThreads)
        if (h[d]) atomicAdd(&head[d], h[d]);
}

__device__ __forceinline__ uint32_t load_published(const uint32_t* p) {
    uint32_t v;
    asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void publish(uint32_t* p, uint32_t v) {
    asm volatile("st.relaxed.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

// One stable pass.  Bound by instructions (some 130 per 32 pairs) and by the
// waits between its steps, with 16 warps per CTA and two CTAs per SM: 1.05 M
// pairs 18 us, 8.3 M 59 us, where a histogram, three scan kernels and a
// scatter took 36 and 87.  kItems keys per thread; a thread looks after kPer
// consecutive digit values (two when there are 1024, else one).  iota >= 0:
// the values are the pair's index >> iota, not read from vals.  Shared
// memory (dynamic): per-warp counts of each digit (16 bits), their tile-wide
// start and global offset, the tile's pairs in sorted order.
template <int kItems, int kPer>
__global__ void __launch_bounds__(kSortThreads, 2) k_sort_pass(const uint32_t* __restrict__ keys,
                                                            const uint32_t* __restrict__ vals, uint32_t n, int shift,
                                                            int dbits, int pass, int iota, uint32_t* __restrict__ head,
                                                            uint32_t* __restrict__ okeys, uint32_t* __restrict__ ovals,
                                                            uint32_t* __restrict__ status) {
    constexpr uint32_t kTileKeys = uint32_t(kItems) * kSortThreads;
    extern __shared__ uint32_t sm[];
    const uint32_t nbk = 1u << dbits, mask = nbk - 1u;
    uint16_t* wh = reinterpret_cast<uint16_t*>(sm);              // [warp][digit]
    uint32_t* lstart = sm + kSortWarps * nbk / 2u;               // [digit]
    uint32_t* goff = lstart + nbk;                               // [digit]
    uint32_t* sk = goff + nbk;
    uint32_t* sv = sk + kTileKeys;
    __shared__ uint32_t s_tile;
    __shared__ unsigned long long s_scan[kSortWarps];
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    for (uint32_t i = threadIdx.x; i < kSortWarps * nbk / 2u; i += kSortThreads) sm[i] = 0u;
    pdl_wait();
    if (threadIdx.x == 0) s_tile = atomicAdd(head + 3072 + pass, 1u);
    __syncthreads();
    const uint32_t tile = s_tile, ntiles = gridDim.x;
    // calls that overlap on one scratch (apic_morton_sort_noalloc on two streams)
    // share its counters: a number past this launch's tiles has neither keys nor
    // published counts in the scratch
    if (tile >= ntiles) return;
    const uint32_t tile0 = tile * kTileKeys, base = tile0 + warp * (32u * kItems);
    uint32_t k[kItems], v[kItems], rk[kItems];
#pragma unroll
    for (int r = 0; r < kItems; ++r) {
        const uint32_t i = base + uint32_t(r) * 32u + lane;
        k[r] = i < n ? keys[i] : 0u;
        v[r] = iota >= 0 ? i >> iota : (i < n ? vals[i] : 0u);
    }
    const uint32_t d0 = threadIdx.x * uint32_t(kPer);
    const bool owner = d0 < nbk;
    uint32_t total_all[kPer];  // of this thread's digits over all tiles
#pragma unroll
    for (int j = 0; j < kPer; ++j) total_all[j] = owner ? head[uint32_t(pass) * nbk + d0 + uint32_t(j)] : 0u;
    uint16_t* mine = wh + warp * nbk;
#pragma unroll
    for (int r = 0; r < kItems; ++r) {
        const bool ok = base + uint32_t(r) * 32u + lane < n;
        const uint32_t d = ok ? (k[r] >> shift) & mask : kMaxBuckets;
        const uint32_t peers = __match_any_sync(0xffffffffu, d);
        const uint32_t before = ok ? mine[d] : 0u, below = uint32_t(__popc(peers & ((1u << lane) - 1u)));
        __syncwarp();
        if (ok && below == 0) mine[d] = uint16_t(before + uint32_t(__popc(peers)));
        __syncwarp();
        rk[r] = before + below;
    }
    __syncthreads();
    // this thread's digits: the warps' places within the digit, the tile's count
    uint32_t* state = head + kSortHead + (size_t(pass) * ntiles + tile) * nbk;
    // (all warps' counts first, two digits of a thread in one word: a loop of
    // reads behind writes is a chain of shared-memory latencies)
    uint32_t cnt[kPer];
    unsigned long long both = 0;  // count in the tile | count over all tiles << 32
    if constexpr (kPer == 2) {
        uint32_t run = 0;  // of both digits; a tile holds at most 4096 pairs
        if (owner) {
            uint32_t* col = sm + d0 / 2u;
            uint32_t c[kSortWarps];
#pragma unroll
            for (int w = 0; w < kSortWarps; ++w) c[w] = col[uint32_t(w) * (nbk / 2u)];
#pragma unroll
            for (int w = 0; w < kSortWarps; ++w) {
                col[uint32_t(w) * (nbk / 2u)] = run;
                run += c[w];
            }
        }
        cnt[0] = run & 0xffffu;
        cnt[1] = run >> 16;
    } else {
        uint32_t run = 0;
        if (owner) {
            uint32_t c[kSortWarps];
#pragma unroll
            for (int w = 0; w < kSortWarps; ++w) c[w] = wh[uint32_t(w) * nbk + d0];
#pragma unroll
            for (int w = 0; w < kSortWarps; ++w) {
                wh[uint32_t(w) * nbk + d0] = uint16_t(run);
                run += c[w];
            }
        }
        cnt[0] = run;
    }
#pragma unroll
    for (int j = 0; j < kPer; ++j) {
        if (owner) publish(state + d0 + j, tile == 0 ? cnt[j] | kInclusive : cnt[j]);
        both += (static_cast<unsigned long long>(total_all[j]) << 32) | cnt[j];
    }
    // exclusive sums over the digits of both
    unsigned long long x = both;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned long long y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= uint32_t(o)) x += y;
    }
    if (lane == 31) s_scan[warp] = x;
    __syncthreads();
    unsigned long long ex = x - both;
    for (uint32_t w = 0; w < warp; ++w) ex += s_scan[w];
    uint32_t local[kPer], global[kPer];
    {
        uint32_t l = uint32_t(ex), g = uint32_t(ex >> 32);
#pragma unroll
        for (int j = 0; j < kPer; ++j) {
            local[j] = l;
            global[j] = g;
            if (owner) lstart[d0 + j] = l;
            l += cnt[j];
            g += total_all[j];
        }
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < kItems; ++r) {
        if (base + uint32_t(r) * 32u + lane >= n) continue;
        const uint32_t d = (k[r] >> shift) & mask;
        const uint32_t at = lstart[d] + mine[d] + rk[r];
        sk[at] = k[r];
        sv[at] = v[r];
    }
    // look back: add up what the tiles before this one published, kLookback of
    // them at a time, until one has its running total
    bool lost = false;
    if (owner && tile > 0) {
        uint32_t sum[kPer], left[kPer];  // left: tiles still to add (0: done)
#pragma unroll
        for (int j = 0; j < kPer; ++j) {
            sum[j] = 0;
            left[j] = tile;
        }
        uint32_t spins = 0;
        for (;;) {
            bool open = false;
#pragma unroll
            for (int j = 0; j < kPer; ++j) {
                if (left[j] == 0) continue;
                const uint32_t* at = state + d0 + j - size_t(tile) * nbk;  // tile 0's
                uint32_t q[kLookback];
#pragma unroll
                for (int b = 0; b < kLookback; ++b)
                    q[b] = left[j] > uint32_t(b) ? load_published(at + size_t(left[j] - 1u - uint32_t(b)) * nbk)
                                                 : kNotReady;
                bool go = true;
#pragma unroll
                for (int b = 0; b < kLookback; ++b) {
                    if (!go || q[b] == kNotReady) {
                        go = false;
                        continue;
                    }
                    sum[j] += q[b] & ~kInclusive;
                    left[j] -= 1u;
                    if (q[b] & kInclusive) {
                        left[j] = 0;
                        go = false;
                    }
                }
                open = open || left[j] != 0;
            }
            if (!open) break;
            if (++spins > kSpinLimit) {
                lost = true;
                break;
            }
        }
        if (!lost) {
#pragma unroll
            for (int j = 0; j < kPer; ++j) {
                publish(state + d0 + j, (sum[j] + cnt[j]) | kInclusive);
                global[j] += sum[j];
            }
        }
    }
    if (owner) {
#pragma unroll
        for (int j = 0; j < kPer; ++j) goff[d0 + j] = global[j] - local[j];
    }
    const uint32_t here = min(kTileKeys, n - tile0);
    if (__syncthreads_or(lost)) {  // (never expected)
        for (uint32_t i = threadIdx.x; i < nbk; i += kSortThreads) sm[i] = 0u;  // (the warps' counts are used up)
        __syncthreads();
        for (uint32_t i = threadIdx.x; i < tile0; i += kSortThreads) atomicAdd(&sm[(keys[i] >> shift) & mask], 1u);
        __syncthreads();
        if (lost) {
#pragma unroll
            for (uint32_t j = 0; j < kPer; ++j) {
                const uint32_t d = d0 + j, own = (d + 1u < nbk ? lstart[d + 1u] : here) - lstart[d];
                publish(state + d, (sm[d] + own) | kInclusive);
                goff[d] += sm[d];
            }
        }
        __syncthreads();
    }
    for (uint32_t q = threadIdx.x; q < here; q += kSortThreads) {
        const uint32_t key = sk[q], pos = goff[(key >> shift) & mask] + q;
        if (pos >= n) {  // (scratch overwritten by an overlapping call)
            if (status) atomicOr(status, kStatusBounds);
            continue;
        }
        okeys[pos] = key;
        ovals[pos] = sv[q];
    }
}

}  // namespace

// Bit length of the largest P2G bin key (row-major cell index).
int bin_key_bits(const Scene& s) {
    uint32_t mx = s.cells > 0 ? s.cells - 1 : 0;
    int b = 0;
    while (b < 32 && (mx >> b)) ++b;
    return b;
}

static int key_bits(const Scene& s) {
    uint32_t mx = s.W ? s.W - 1 : 0, my = s.H ? s.H - 1 : 0;
    // Morton order is monotone in x and y, so the largest key is that of the
    // far corner (sides are limited to 65536, so 16 bits per axis suffice).
    uint32_t ex = mx & 0xFFFFu, ey = my & 0xFFFFu;
    auto expand = [](uint32_t v) {
        v = (v | (v << 8)) & 0x00FF00FFu;
        v = (v | (v << 4)) & 0x0F0F0F0Fu;
        v = (v | (v << 2)) & 0x33333333u;
        v = (v | (v << 1)) & 0x55555555u;
        return v;
    };
    uint32_t k = expand(ex) | (expand(ey) << 1);
    int b = 0;
    while (b < 32 && (k >> b)) ++b;
    return b;
}

// Digit width of an LSD sort over `bits` key bits: the fewest passes of at
// most kMaxDigitBits bits, split as evenly as possible.
static int digit_bits(int bits) {
    if (bits <= 0) return 0;
    int passes = (bits + kMaxDigitBits - 1) / kMaxDigitBits;
    return (bits + passes - 1) / passes;
}

// Tile size of a sort: small sorts take small tiles, for which the look-back
// is short and more SMs work; from 256 K pairs on 4096 pairs a tile.
constexpr uint32_t kTile2Pairs = 65536u, kTile4Pairs = 262144u;
static int tile_items(uint32_t n) { return n <= kTile2Pairs ? 2 : n <= kTile4Pairs ? 4 : 8; }
static uint32_t sort_tiles(uint32_t n) { return div_up(n, uint32_t(tile_items(n)) * kSortThreads); }
static int sort_passes(int bits, int dbits) { return dbits > 0 ? (bits + dbits - 1) / dbits : 0; }
static size_t pass_smem(int items, int dbits) {
    const size_t nbk = size_t(1) << dbits;
    return kSortWarps * nbk * 2 + 2 * nbk * 4 + 2 * size_t(items) * kSortThreads * 4;
}

template <int kItems>
static cudaError_t sort_pass(bool pdl, uint32_t tiles, cudaStream_t st, const uint32_t* k, const uint32_t* v,
                             uint32_t n, int shift, int dbits, int pass, int iota, uint32_t* head, uint32_t* ok,
                             uint32_t* ov, uint32_t* status) {
    auto kern = dbits > 9 ? k_sort_pass<kItems, 2> : k_sort_pass<kItems, 1>;
    // the limit is the kernel's largest, not this pass's: scenes are prepared on
    // several threads, and a limit that changes under another thread's graph
    // breaks that graph
    const size_t smem = pass_smem(kItems, dbits);
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         int(pass_smem(kItems, dbits > 9 ? kMaxDigitBits : 9)));
    if (e != cudaSuccess) return e;
    return launch(pdl, kern, tiles, kSortThreads, smem, st, k, v, n, shift, dbits, pass, iota, head, ok, ov, status);
}

static cudaError_t lsd_passes(uint32_t* keys, uint32_t* vals, uint32_t* keys_alt, uint32_t* vals_alt, uint32_t* head,
                              uint32_t n, int bits, int dbits, int iota, cudaStream_t st, bool pdl,
                              uint32_t** keys_out, uint32_t** vals_out, uint32_t* status) {
    uint32_t *k_in = keys, *v_in = vals, *k_out = keys_alt, *v_out = vals_alt;
    const int passes = sort_passes(bits, dbits), items = tile_items(n);
    const uint32_t tiles = sort_tiles(n);
    cudaError_t e = cudaSuccess;
    if (passes > 0)
        e = launch(pdl, k_sort_prepare, std::min(div_up(n, kSortThreads * kCountKeys), 304u), kSortThreads, 0, st,
                   static_cast<const uint32_t*>(k_in), n, passes, dbits, head,
                   uint32_t(passes) * tiles << dbits);
    for (int p = 0; p < passes && e == cudaSuccess; ++p) {
        auto pass = items == 2 ? sort_pass<2> : items == 4 ? sort_pass<4> : sort_pass<8>;
        e = pass(pdl, tiles, st, k_in, v_in, n, p * dbits, dbits, p, p == 0 ? iota : -1, head, k_out, v_out, status);
        std::swap(k_in, k_out);
        std::swap(v_in, v_out);
    }
    *keys_out = k_in;
    *vals_out = v_in;
    return e != cudaSuccess ? e : cudaGetLastError();
}

uint32_t sort_scratch_words(uint32_t n, int bits, int dbits) {
    if (n == 0) return kSortHead;
    return kSortHead + uint32_t(((size_t(sort_passes(bits, dbits)) * sort_tiles(n) << dbits) + 3) & ~size_t(3));
}
uint32_t sort_scratch_words(const Scene& s, uint32_t n) {
    const int m = key_bits(s), b = bin_key_bits(s);
    uint32_t words = 0;
    // (the largest counts of each tile size: fewer pairs may make more tiles)
    for (uint32_t k : {n, std::min(n, kTile2Pairs), std::min(n, kTile4Pairs)})
        words = std::max({words, sort_scratch_words(k, m, digit_bits(m)), sort_scratch_words(k, b, digit_bits(b))});
    return words;
}

cudaError_t radix_sort_pairs(uint32_t* keys, uint32_t* vals, uint32_t* keys_alt, uint32_t* vals_alt, uint32_t* scratch,
                             uint32_t n, int bits, int iota, cudaStream_t st, bool pdl, uint32_t** keys_out,
                             uint32_t** vals_out, uint32_t* status) {
    *keys_out = keys;
    *vals_out = vals;
    if (n == 0) return cudaSuccess;
    return lsd_passes(keys, vals, keys_alt, vals_alt, scratch, n, bits, digit_bits(bits), iota, st, pdl, keys_out,
                      vals_out, status);
}

bool radix_sort_in_alt(int bits) { return sort_passes(bits, digit_bits(bits)) % 2 == 1; }
int sort_digit_bits(int bits) { return digit_bits(bits); }

cudaError_t launch_sort(Scene& s) {
    if (s.n == 0) return cudaSuccess;
    float max_x = float(s.W > 0 ? s.W - 1 : 0), max_y = float(s.H > 0 ? s.H - 1 : 0);
    launch(s.use_pdl, k_morton_keys, div_up(s.n, 1024), 256, 0, s.stream, s.pp, s.n,
           CellSize{s.dx, exact_reciprocal(s.dx)}, max_x, max_y, s.keys, s.sort_scratch);
    // the sorted pairs stay where the last pass wrote them (no copy back)
    uint32_t *k_res, *v_res;
    cudaError_t e = radix_sort_pairs(s.keys, s.vals, s.keys_alt, s.vals_alt, s.sort_scratch, s.n, key_bits(s), 0,
                                     s.stream, s.use_pdl, &k_res, &v_res, &s.ctl->status);
    if (e != cudaSuccess) return e;
    return launch_permute(s, v_res);
}

// Where launch_sort leaves the sorted pairs of a scene (the number of digit
// passes is fixed by the grid size).
bool sort_result_in_alt(const Scene& s) { return radix_sort_in_alt(key_bits(s)); }

// The same sort with digits of the caller's choice, on a stream of the
// caller's (noalloc.cu).  Its kernels are programmatic dependents of one another,
// on the legacy stream too (20000 pairs 25.1 -> 19.5 us, 1000003 58.4 -> 53.3,
// with the counts of a digit's warps read before they are written back).
cudaError_t radix_sort_pairs_digits(uint32_t* keys, uint32_t* vals, uint32_t* keys_alt, uint32_t* vals_alt,
                                    uint32_t* scratch, uint32_t n, int bits, int dbits, cudaStream_t st) {
    uint32_t *k_res, *v_res;
    return lsd_passes(keys, vals, keys_alt, vals_alt, scratch, n, bits, dbits, 0, st, true, &k_res, &v_res,
                      nullptr);
}

// Bit length of the largest Morton key of a width x height grid.
int morton_key_bits(uint32_t width, uint32_t height) {
    Scene probe;
    probe.W = width;
    probe.H = height;
    return key_bits(probe);
}

}  // namespace apic
