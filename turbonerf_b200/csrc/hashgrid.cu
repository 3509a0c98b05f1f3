// Multiresolution hash-grid encoding (sm_100a): the upstream producer of sigma and rgb at the
// tiny-cuda-nn boundary of the reference (src/core/nerf-network.cu:27-124 builds tcnn's HashGrid
// with 16 levels of 2 features, 2^19 entries a level, base resolution 16 and per-level scale
// b = exp((ln 2048 A - ln 16) / 15), linear interpolation; its forward and backward run at
// :431-545 and :668-768). tcnn's source is not part of the reference tree, so this is the
// published algorithm (Mueller et al. 2022, "Instant neural graphics primitives with a
// multiresolution hash encoding", section 3):
//   level l has resolution N_l = floor(N_min b^l); a position x in [0,1]^3 falls in the cell
//   floor(x N_l) with in-cell coordinates f = x N_l - floor(x N_l); the level's feature vector is
//   the trilinear interpolation of the 8 corner vertices' entries; a vertex v indexes its entry
//   directly when the level's (N_l + 1)^3 vertices fit in the table (coarse levels), else by the
//   spatial hash (v_x * 1) xor (v_y * 2654435761) xor (v_z * 805459861) mod T.
// The backward scatters w_c * dL/dfeature into the corner entries' gradients (atomic adds) and
// records, once per entry, every entry a live sample touched: a bitmap and a list, which drive
// the gradient clearing before the next step (and tell which hash entries Adam will see).
//
// Layout: parameters [level][T][2] (one float2 per entry, level l at l T entries); features and
// their gradients [2 L][stride] (feature-major, coalesced per feature). The linear heads that
// stand in for tcnn's density and colour MLPs read the 2 L features of a sample:
//   density = b_s + w_s . f (raw network density; the losses apply the reference's exp
//   activation), rgb_c = sigmoid(b_c + W_c . f).
// Head parameters, after the hash entries: w_s[2L], b_s, then for c = r, g, b: W_c[2L], b_c.
#include <cmath>
#include <vector>

#include "tn_internal.cuh"

namespace tn {

constexpr int HG_F = 2;             // features a level
constexpr int HG_MAX_LEVELS = 16;   // levels
constexpr int HG_MAX_FEAT = HG_F * HG_MAX_LEVELS;

struct HashLevels {
    float scale[HG_MAX_LEVELS];     // N_l
    uint32_t res[HG_MAX_LEVELS];    // N_l
    uint32_t dense[HG_MAX_LEVELS];  // 1: the level's (N_l + 1)^3 vertices index their entries directly
    uint32_t n_levels;
    uint32_t log2_t;
};

// Per-level constants from the descriptor (host, double precision for b^l as the reference's
// host code computes b).
static int hash_levels(const tn_hashgrid_desc* d, HashLevels& H) {
    TN_REQUIRE(d != nullptr, TN_E_NULL, "hash-grid descriptor is NULL");
    TN_REQUIRE(d->n_levels >= 1 && d->n_levels <= (uint32_t)HG_MAX_LEVELS, TN_E_INVALID,
               "n_levels %u not in 1..%d", d->n_levels, HG_MAX_LEVELS);
    TN_REQUIRE(d->log2_hashmap_size >= 4 && d->log2_hashmap_size <= 24, TN_E_INVALID,
               "log2_hashmap_size %u not in 4..24", d->log2_hashmap_size);
    TN_REQUIRE(d->base_resolution >= 1.0f && d->per_level_scale >= 1.0f, TN_E_INVALID,
               "base_resolution and per_level_scale must be at least 1");
    const double T = (double)(1u << d->log2_hashmap_size);
    H.n_levels = d->n_levels;
    H.log2_t = d->log2_hashmap_size;
    for (uint32_t l = 0; l < (uint32_t)HG_MAX_LEVELS; ++l) {
        const double n = l < d->n_levels ? std::floor((double)d->base_resolution *
                                                      std::pow((double)d->per_level_scale, (double)l))
                                         : 1.0;
        TN_REQUIRE(n >= 1.0 && n < 16777216.0, TN_E_INVALID, "level %u resolution %.0f out of range", l, n);
        H.res[l] = (uint32_t)n;
        H.scale[l] = (float)n;
        H.dense[l] = (n + 1.0) * (n + 1.0) * (n + 1.0) <= T ? 1u : 0u;
    }
    return TN_OK;
}

__device__ __forceinline__ uint32_t hg_index(const HashLevels& H, int l, uint32_t x, uint32_t y, uint32_t z) {
    if (H.dense[l]) {
        const uint32_t r = H.res[l] + 1u;
        return x + r * (y + r * z);
    }
    return ((x * 1u) ^ (y * 2654435761u) ^ (z * 805459861u)) & ((1u << H.log2_t) - 1u);
}

// Cell and in-cell coordinate of one coordinate at a level; the cell is clamped to [0, N - 1],
// so that its upper corner is a vertex of the level (a coordinate of exactly 1 has f = 1).
__device__ __forceinline__ void hg_cell(float p, float scale, uint32_t res, uint32_t& i, float& f) {
    const float s = __fmul_rn(p, scale);
    const float fl = fminf(fmaxf(floorf(s), 0.0f), (float)(res - 1u));
    i = (uint32_t)fl;
    f = __fsub_rn(s, fl);
}

// A sample's cell at a level and its in-cell coordinates.
struct HashCell {
    uint32_t x, y, z;
    float fx, fy, fz;
};

__device__ __forceinline__ HashCell hg_locate(const HashLevels& H, int l, float px, float py, float pz) {
    HashCell c;
    hg_cell(px, H.scale[l], H.res[l], c.x, c.fx);
    hg_cell(py, H.scale[l], H.res[l], c.y, c.fy);
    hg_cell(pz, H.scale[l], H.res[l], c.z, c.fz);
    return c;
}

__device__ __forceinline__ bool hg_same(const HashCell& a, const HashCell& b) {
    return a.x == b.x && a.y == b.y && a.z == b.z;
}

// Corner k (bit 0: x + 1, bit 1: y + 1, bit 2: z + 1) of a cell: its entry and trilinear weight
// ((w_x w_y) w_z, each 1 - f or f).
__device__ __forceinline__ uint32_t hg_corner(const HashLevels& H, int l, const HashCell& c, int k) {
    return hg_index(H, l, c.x + (k & 1), c.y + ((k >> 1) & 1), c.z + ((k >> 2) & 1));
}

__device__ __forceinline__ void hg_weights(const HashCell& c, float (&w)[8]) {
    const float gx = __fsub_rn(1.0f, c.fx), gy = __fsub_rn(1.0f, c.fy), gz = __fsub_rn(1.0f, c.fz);
#pragma unroll
    for (int k = 0; k < 8; ++k)
        w[k] = __fmul_rn(__fmul_rn((k & 1) ? c.fx : gx, ((k >> 1) & 1) ? c.fy : gy), ((k >> 2) & 1) ? c.fz : gz);
}

__device__ __forceinline__ uint32_t live_count(uint32_t n, const uint32_t* n_dev) {
    return n_dev ? min(*n_dev, n) : n;
}

// RUN consecutive values from s0 (those below n; the others zero), as 16-byte groups when VEC.
template <int RUN, bool VEC>
__device__ __forceinline__ void hg_load_run(const float* __restrict__ p, uint32_t s0, uint32_t n, float (&v)[RUN]) {
    if (VEC && s0 + RUN <= n) {
#pragma unroll
        for (int q = 0; q < RUN / 4; ++q) {
            const float4 u = __ldg(reinterpret_cast<const float4*>(p + s0) + q);
            v[4 * q] = u.x;
            v[4 * q + 1] = u.y;
            v[4 * q + 2] = u.z;
            v[4 * q + 3] = u.w;
        }
    } else {
#pragma unroll
        for (int q = 0; q < RUN; ++q) v[q] = s0 + q < n ? __ldg(p + s0 + q) : 0.0f;
    }
}

constexpr int HG_THREADS = 256;

// One thread per (sample, level): the level's two features, sum over the corners in order of
// w_c * entry (fused multiply-adds).
__global__ void __launch_bounds__(HG_THREADS)
hg_encode_kernel(HashLevels H, uint32_t n, const uint32_t* __restrict__ n_dev, uint32_t pstride, uint32_t stride,
                 const float* __restrict__ pos, const float2* __restrict__ params, float* __restrict__ feat) {
    const uint32_t s = blockIdx.x * blockDim.x + threadIdx.x;
    const int l = blockIdx.y;
    if (s >= live_count(n, n_dev)) return;
    const HashCell c = hg_locate(H, l, pos[s], pos[s + pstride], pos[s + 2 * (size_t)pstride]);
    const float2* P = params + ((size_t)l << H.log2_t);
    float2 v[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) v[k] = __ldg(P + hg_corner(H, l, c, k));
    float w[8];
    hg_weights(c, w);
    float a0 = 0.0f, a1 = 0.0f;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        a0 = __fmaf_rn(w[k], v[k].x, a0);
        a1 = __fmaf_rn(w[k], v[k].y, a1);
    }
    feat[(size_t)(HG_F * l) * stride + s] = a0;
    feat[(size_t)(HG_F * l + 1) * stride + s] = a1;
}

// grads[e] += v for the four floats of an aligned pair of entries in one reduction.
__device__ __forceinline__ void red_pair(float2* p, float2 a, float2 b) {
    asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(p), "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y)
                 : "memory");
}

// Adds a cell's corner sums to the gradients. The two corners of an x edge are neighbours in the
// table, in one aligned pair, for every second x (directly indexed levels: entry e and e + 1 with e
// even; hashed levels: x even, where x and x + 1 differ in bit 0 of the hash alone): one 16-byte
// reduction instead of two 8-byte ones (pairs: the gradients are 16-byte aligned).
__device__ __forceinline__ void hg_flush(const HashLevels& H, int l, const HashCell& c, const float2 (&g)[8],
                                         float2* __restrict__ G, bool pairs) {
#pragma unroll
    for (int k = 0; k < 8; k += 2) {
        const uint32_t e0 = hg_corner(H, l, c, k), e1 = hg_corner(H, l, c, k + 1);
        if (pairs && (e0 ^ e1) == 1u) {
            const bool up = (e0 & 1u) == 0u;
            red_pair(G + (e0 & ~1u), up ? g[k] : g[k + 1], up ? g[k + 1] : g[k]);
        } else {
            atomicAdd(G + e0, g[k]);
            atomicAdd(G + e1, g[k + 1]);
        }
    }
}

// One thread per RUN consecutive samples and level: w_c * dL/dfeature summed in registers over the
// samples of a cell, then added to the corners' entries when the cell changes: samples follow each
// other along rays, so on the coarse half of the levels most of them stay in their cell. Bound by
// the L2's reductions (about 150 G a second). 2^18 samples, 16 levels of up to 2048: 85 us (110
// without the paired reductions), 234 us with one sample a thread and the lanes of a warp that
// share an entry added up in shared memory; on uniform positions only the pairing remains.
template <int RUN, bool VEC>
__global__ void __launch_bounds__(HG_THREADS)
hg_backward_kernel(HashLevels H, uint32_t n, const uint32_t* __restrict__ n_dev, uint32_t pstride, uint32_t stride,
                   const float* __restrict__ pos, const float* __restrict__ dfeat, float2* __restrict__ grads, bool pairs) {
    const uint32_t s0 = (blockIdx.x * HG_THREADS + threadIdx.x) * RUN;
    const int l = blockIdx.y;
    const uint32_t nl = live_count(n, n_dev);
    if (s0 >= nl) return;
    float px[RUN], py[RUN], pz[RUN], g0[RUN], g1[RUN];
    hg_load_run<RUN, VEC>(pos, s0, nl, px);
    hg_load_run<RUN, VEC>(pos + pstride, s0, nl, py);
    hg_load_run<RUN, VEC>(pos + 2 * (size_t)pstride, s0, nl, pz);
    hg_load_run<RUN, VEC>(dfeat + (size_t)(HG_F * l) * stride, s0, nl, g0);
    hg_load_run<RUN, VEC>(dfeat + (size_t)(HG_F * l + 1) * stride, s0, nl, g1);
    float2* G = grads + ((size_t)l << H.log2_t);
    HashCell cur;
    float2 sum[8];
#pragma unroll
    for (int q = 0; q < RUN; ++q) {
        if (s0 + q >= nl) break;
        const HashCell c = hg_locate(H, l, px[q], py[q], pz[q]);
        float w[8];
        hg_weights(c, w);
        const bool same = q > 0 && hg_same(c, cur);
        if (q > 0 && !same) hg_flush(H, l, cur, sum, G, pairs);
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            const float vx = __fmul_rn(w[k], g0[q]), vy = __fmul_rn(w[k], g1[q]);
            sum[k].x = same ? sum[k].x + vx : vx;
            sum[k].y = same ? sum[k].y + vy : vy;
        }
        cur = c;
    }
    hg_flush(H, l, cur, sum, G, pairs);
}

// Lists every entry a live sample touches once (the thread whose atomic or sets the entry's bit appends
// l T + idx), one thread per (sample, level); with ADD it adds the sample's gradients too, one launch for
// a short batch. A cell shared with the sample before, as along a ray, is that one's to list; bits already
// set are seen with a plain read and skip their atomic; the two corners of an x edge have theirs in one word
// for 31 of 32 x, read and set as one; a block's new entries take one counter atomic.
// Bound by the atomics that return and the random reads of the bitmap before them (28 of 43 stall cycles an
// issued instruction wait for them). The backward with its list, 2^18 samples of 16 levels along rays and uniform: 310 and
// 485 us; 467 and 590 where one kernel added and listed a sample a thread, 416 and 609 with this kernel
// one atomic a corner, lanes compared entry by entry and one counter atomic a warp. Listing inside
// the runs of hg_backward_kernel, edges together: 375 and 424, but 8000 samples 30 and 28 where this takes 22 and 25.
template <bool ADD>
__global__ void __launch_bounds__(HG_THREADS)
hg_touch_kernel(HashLevels H, uint32_t n, const uint32_t* __restrict__ n_dev, uint32_t pstride, uint32_t stride,
                const float* __restrict__ pos, const float* __restrict__ dfeat, float2* __restrict__ grads, bool pairs,
                uint32_t* __restrict__ bits, uint32_t* __restrict__ list, uint32_t* __restrict__ count) {
    __shared__ uint32_t warp_n[HG_THREADS / WARP];
    __shared__ uint32_t block_at;
    const uint32_t nl = live_count(n, n_dev);
    if (blockIdx.x * HG_THREADS >= nl) return;  // whole blocks
    const uint32_t s = blockIdx.x * HG_THREADS + threadIdx.x, at_s = min(s, nl - 1u);
    const int l = blockIdx.y;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const HashCell c = hg_locate(H, l, pos[at_s], pos[at_s + pstride], pos[at_s + 2 * (size_t)pstride]);
    HashCell before = c;
    before.x = __shfl_up_sync(FULL_MASK, c.x, 1);
    before.y = __shfl_up_sync(FULL_MASK, c.y, 1);
    before.z = __shfl_up_sync(FULL_MASK, c.z, 1);
    const bool head = s < nl && (lane == 0 || !hg_same(before, c));
    const uint32_t base = (uint32_t)l << H.log2_t;
    // the two corners of an x edge have their bits in one word for 31 of 32 x
    uint32_t e[8], word[8];
#pragma unroll
    for (int k = 0; k < 8; k += 2) {
        e[k] = base + hg_corner(H, l, c, k);
        e[k + 1] = base + hg_corner(H, l, c, k + 1);
        word[k] = head ? bits[e[k] >> 5] : ~0u;
        word[k + 1] = !head ? ~0u : (e[k] ^ e[k + 1]) < 32u ? word[k] : bits[e[k + 1] >> 5];
    }
    if (ADD && s < nl) {  // beside the words on their way
        const float g0 = dfeat[(size_t)(HG_F * l) * stride + s], g1 = dfeat[(size_t)(HG_F * l + 1) * stride + s];
        float w[8];
        hg_weights(c, w);
        float2 g[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) g[k] = make_float2(__fmul_rn(w[k], g0), __fmul_rn(w[k], g1));
        hg_flush(H, l, c, g, grads + base, pairs);
    }
    bool fresh[8];
#pragma unroll
    for (int k = 0; k < 8; k += 2) {
        const bool together = (e[k] ^ e[k + 1]) < 32u;
        uint32_t b0 = ~word[k] & (1u << (e[k] & 31u)), b1 = ~word[k + 1] & (1u << (e[k + 1] & 31u));
        const uint32_t set = together ? b0 | b1 : b0;
        if (set) {
            const uint32_t old = atomicOr(bits + (e[k] >> 5), set);
            b0 &= ~old;
            if (together) b1 &= ~old;
        }
        if (!together && b1) b1 &= ~atomicOr(bits + (e[k + 1] >> 5), b1);
        fresh[k] = b0 != 0u;
        fresh[k + 1] = b1 != 0u;
    }
    unsigned news[8];
    uint32_t total = 0;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        news[k] = __ballot_sync(FULL_MASK, fresh[k]);
        total += (uint32_t)__popc(news[k]);
    }
    if (lane == 0) warp_n[wid] = total;
    __syncthreads();
    if (threadIdx.x == 0) {
        uint32_t sum = 0;
#pragma unroll
        for (int w = 0; w < HG_THREADS / WARP; ++w) {
            const uint32_t v = warp_n[w];
            warp_n[w] = sum;
            sum += v;
        }
        block_at = sum ? atomicAdd(count, sum) : 0u;
    }
    __syncthreads();
    uint32_t at = block_at + warp_n[wid];
    const unsigned below = (1u << lane) - 1u;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        if (fresh[k]) list[at + (uint32_t)__popc(news[k] & below)] = e[k];
        at += (uint32_t)__popc(news[k]);
    }
}

// Zeroes the listed entries' gradients and bitmap words (several entries may share a word; all
// write zero).
__global__ void hg_clear_kernel(const uint32_t* __restrict__ list, const uint32_t* __restrict__ count, uint32_t max,
                                float2* __restrict__ grads, uint32_t* __restrict__ bits) {
    const uint32_t nl = min(*count, max);
    for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < nl; k += gridDim.x * blockDim.x) {
        const uint32_t e = list[k];
        grads[e] = make_float2(0.0f, 0.0f);
        if (bits) bits[e >> 5] = 0u;
    }
}

// Entries with a nonzero gradient (either feature), listed in no particular order: each thread
// takes 8 consecutive entries (four 16-byte loads), a block ranks its nonzero entries with a scan of
// the warps' counts and takes their places with one counter atomic.
constexpr int HG_NZ_THREADS = 256;
__global__ void __launch_bounds__(HG_NZ_THREADS)
hg_nonzero_kernel(uint32_t n_entries, const float4* __restrict__ grads, uint32_t* __restrict__ list,
                  uint32_t* __restrict__ count) {
    __shared__ uint32_t warp_n[HG_NZ_THREADS / WARP];
    __shared__ uint32_t block_at;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const uint32_t e0 = (blockIdx.x * HG_NZ_THREADS + threadIdx.x) * 8u;
    uint32_t mask = 0;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        if (e0 + 2u * q < n_entries) {  // n_entries is even: the pair's second entry exists too
            const float4 v = grads[e0 / 2u + q];
            if (v.x != 0.0f || v.y != 0.0f) mask |= 1u << (2 * q);
            if (v.z != 0.0f || v.w != 0.0f) mask |= 1u << (2 * q + 1);
        }
    }
    const uint32_t mine = (uint32_t)__popc(mask);
    uint32_t incl = mine;
#pragma unroll
    for (int d = 1; d < WARP; d <<= 1) {
        const uint32_t o = __shfl_up_sync(FULL_MASK, incl, d);
        if (lane >= d) incl += o;
    }
    if (lane == WARP - 1) warp_n[wid] = incl;
    __syncthreads();
    if (threadIdx.x == 0) {
        uint32_t t = 0;
        for (int w = 0; w < HG_NZ_THREADS / WARP; ++w) {
            const uint32_t c = warp_n[w];
            warp_n[w] = t;
            t += c;
        }
        block_at = t ? atomicAdd(count, t) : 0u;
    }
    __syncthreads();
    uint32_t at = block_at + warp_n[wid] + incl - mine;
    for (uint32_t m = mask; m; m &= m - 1u) list[at++] = e0 + (uint32_t)(__ffs(m) - 1);
}

// ---- linear heads (the stand-in for tcnn's density and colour MLPs) ------------------------
__device__ __forceinline__ float sigmoid(float z) { return 1.0f / (1.0f + expf(-z)); }

// One thread per sample: raw density and rgb ([3][ostride]) from the 2 L features ([2L][stride]).
__global__ void __launch_bounds__(256)
hg_heads_forward_kernel(uint32_t nf, uint32_t n, const uint32_t* __restrict__ n_dev, uint32_t stride,
                        const float* __restrict__ feat, const float* __restrict__ head, float* __restrict__ density,
                        float* __restrict__ rgb, uint32_t ostride) {
    const uint32_t s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= live_count(n, n_dev)) return;
    float z[4];
#pragma unroll
    for (int o = 0; o < 4; ++o) z[o] = __ldg(head + o * (nf + 1) + nf);
    for (uint32_t j = 0; j < nf; ++j) {
        const float f = feat[(size_t)j * stride + s];
#pragma unroll
        for (int o = 0; o < 4; ++o) z[o] = fmaf(__ldg(head + o * (nf + 1) + j), f, z[o]);
    }
    density[s] = z[0];
    if (rgb) {
#pragma unroll
        for (int c = 0; c < 3; ++c) rgb[(size_t)c * ostride + s] = sigmoid(z[c + 1]);
    }
}

// A warp takes 32 samples at a time, a grid apart: a thread per sample for dL/dfeature (written)
// and dz, then a lane per feature for the heads' parameter gradients, which adds dz_o f_j over the
// 32 samples from the warp's shared tile; summed over the block into partials[block][4]
// [HG_MAX_FEAT + 1] (head o's weights j < nf, then its bias at HG_MAX_FEAT; deterministic: fixed
// samples a warp, fixed lanes, fixed warps). 2^18 samples of the training step, beside a march on
// 64 SMs: 35 us; with a thread's 33 products through shared memory for every head and column sums
// by 231 threads 50 us; with all 132 sums in each thread's registers 120 us (spills, 8 warps an
// SM); 8 features loaded at a time instead of 16 47 us.
constexpr int HG_HEAD_THREADS = 256;
constexpr int HG_HEAD_BLOCKS_PER_SM = 4;
constexpr int HG_HEAD_GROUP = 16;  // features loaded at a time
constexpr int HG_HEAD_SLOTS = 4 * (HG_MAX_FEAT + 1);
static_assert(HG_MAX_FEAT == WARP, "one feature a lane");
__global__ void __launch_bounds__(HG_HEAD_THREADS, HG_HEAD_BLOCKS_PER_SM)
hg_heads_backward_kernel(uint32_t nf, uint32_t n, const uint32_t* __restrict__ n_dev, uint32_t stride,
                         const float* __restrict__ feat, const float* __restrict__ head,
                         const float* __restrict__ dL_ddensity, const float* __restrict__ dL_drgb,
                         float* __restrict__ dfeat, float* __restrict__ partials) {
    constexpr int NW = HG_HEAD_THREADS / WARP, PITCH = HG_MAX_FEAT + 1;
    __shared__ float4 w_s[HG_MAX_FEAT + 1];  // the heads' weights of a feature (zero past nf); last: the biases
    __shared__ float f_s[NW][WARP * PITCH];
    __shared__ float4 dz_s[NW][WARP];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    if (threadIdx.x <= HG_MAX_FEAT) {
        const uint32_t j = threadIdx.x == HG_MAX_FEAT ? nf : threadIdx.x, h = nf + 1;
        const bool on = j < nf || threadIdx.x == HG_MAX_FEAT;
        w_s[threadIdx.x] = on ? make_float4(head[j], head[h + j], head[2 * h + j], head[3 * h + j])
                              : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    }
    __syncthreads();
    const uint32_t nl = live_count(n, n_dev);
    float* const tile = f_s[wid];
    float acc[4] = {0.0f, 0.0f, 0.0f, 0.0f}, bias[4] = {0.0f, 0.0f, 0.0f, 0.0f};
    const uint32_t step = gridDim.x * HG_HEAD_THREADS;
    for (uint32_t s0 = blockIdx.x * HG_HEAD_THREADS + wid * WARP; s0 < nl; s0 += step) {  // whole warps
        const uint32_t s = s0 + lane;
        const bool live = s < nl;
        float4 z = w_s[HG_MAX_FEAT];
#pragma unroll 1
        for (int j0 = 0; j0 < HG_MAX_FEAT; j0 += HG_HEAD_GROUP) {
            float f[HG_HEAD_GROUP];
#pragma unroll
            for (int j = 0; j < HG_HEAD_GROUP; ++j)
                f[j] = live && j0 + j < (int)nf ? __ldg(feat + (size_t)(j0 + j) * stride + s) : 0.0f;
#pragma unroll
            for (int j = 0; j < HG_HEAD_GROUP; ++j) {
                const float4 w = w_s[j0 + j];
                z.y = fmaf(w.y, f[j], z.y);
                z.z = fmaf(w.z, f[j], z.z);
                z.w = fmaf(w.w, f[j], z.w);
                tile[lane * PITCH + j0 + j] = f[j];
            }
        }
        float4 dz = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (live) {
            const float yr = sigmoid(z.y), yg = sigmoid(z.z), yb = sigmoid(z.w);
            dz = make_float4(dL_ddensity[s], dL_drgb[s] * yr * (1.0f - yr), dL_drgb[(size_t)stride + s] * yg * (1.0f - yg),
                             dL_drgb[2 * (size_t)stride + s] * yb * (1.0f - yb));
        }
        dz_s[wid][lane] = dz;
#pragma unroll 8
        for (int j = 0; j < HG_MAX_FEAT; ++j) {
            const float4 w = w_s[j];
            const float g = fmaf(dz.w, w.w, fmaf(dz.z, w.z, fmaf(dz.y, w.y, dz.x * w.x)));
            if (live && j < (int)nf) dfeat[(size_t)j * stride + s] = g;
        }
        bias[0] += dz.x;
        bias[1] += dz.y;
        bias[2] += dz.z;
        bias[3] += dz.w;
        __syncwarp();
#pragma unroll 8
        for (int i = 0; i < WARP; ++i) {
            const float v = tile[i * PITCH + lane];
            const float4 d = dz_s[wid][i];
            acc[0] = fmaf(d.x, v, acc[0]);
            acc[1] = fmaf(d.y, v, acc[1]);
            acc[2] = fmaf(d.z, v, acc[2]);
            acc[3] = fmaf(d.w, v, acc[3]);
        }
        __syncwarp();
    }
#pragma unroll
    for (int o = 0; o < 4; ++o) {
        const float b = warp_sum(bias[o]);
        tile[o * PITCH + lane] = acc[o];
        if (lane == 0) tile[o * PITCH + HG_MAX_FEAT] = b;
    }
    __syncthreads();
    for (int i = threadIdx.x; i < HG_HEAD_SLOTS; i += HG_HEAD_THREADS) {
        float v = 0.0f;
#pragma unroll
        for (int w = 0; w < NW; ++w) v += f_s[w][i];
        partials[(size_t)blockIdx.x * HG_HEAD_SLOTS + i] = v;
    }
}

// The heads' gradients (head o, weight j < nf at o (nf + 1) + j, bias at o (nf + 1) + nf): one
// block a parameter sums the blocks' partials, each thread a strided run of them, then a fixed tree
// over the threads (deterministic).
constexpr int HG_FINISH_THREADS = 256;
__global__ void __launch_bounds__(HG_FINISH_THREADS)
hg_heads_grad_finish_kernel(uint32_t nf, uint32_t n_blocks, const float* __restrict__ partials,
                            float* __restrict__ grads) {
    __shared__ float warp_s[HG_FINISH_THREADS / WARP];
    const uint32_t k = blockIdx.x;
    const uint32_t o = k / (nf + 1), j = k % (nf + 1);
    const uint32_t slot = o * (HG_MAX_FEAT + 1) + (j < nf ? j : (uint32_t)HG_MAX_FEAT);
    float v = 0.0f;
    for (uint32_t b = threadIdx.x; b < n_blocks; b += HG_FINISH_THREADS) v += partials[(size_t)b * HG_HEAD_SLOTS + slot];
    v = warp_sum(v);
    if ((threadIdx.x & 31) == 0) warp_s[threadIdx.x >> 5] = v;
    __syncthreads();
    if (threadIdx.x == 0) {
        float t = 0.0f;
        for (int w = 0; w < HG_FINISH_THREADS / WARP; ++w) t += warp_s[w];
        grads[k] = t;
    }
}

// 16-byte groups: the base 16-byte aligned and the stride between rows a multiple of 4.
static bool hg_vec(const void* a, uint32_t a_stride, const void* b, uint32_t b_stride) {
    return ((((uintptr_t)a | (uintptr_t)b) & 15u) == 0) && ((a_stride | b_stride) & 3u) == 0;
}

static dim3 hg_grid(uint32_t n, uint32_t levels, int run) {
    return dim3((n + HG_THREADS * run - 1) / (HG_THREADS * run), levels);
}

int hashgrid_encode(cudaStream_t stream, const tn_hashgrid_desc* desc, uint32_t n, const uint32_t* n_dev,
                    uint32_t pstride, uint32_t stride, const float* pos, const float* params, float* features) {
    HashLevels H;
    int st = hash_levels(desc, H);
    if (st != TN_OK || n == 0) return st;
    hg_encode_kernel<<<hg_grid(n, H.n_levels, 1), HG_THREADS, 0, stream>>>(
        H, n, n_dev, pstride, stride, pos, reinterpret_cast<const float2*>(params), features);
    return check_launch("tn_hashgrid_encode");
}

int hashgrid_backward(cudaStream_t stream, const tn_hashgrid_desc* desc, uint32_t n, const uint32_t* n_dev,
                      uint32_t pstride, uint32_t stride, const float* pos, const float* dL_dfeatures, float* grads,
                      uint32_t* touched_bits, uint32_t* touched_list, uint32_t* touched_count) {
    HashLevels H;
    int st = hash_levels(desc, H);
    if (st != TN_OK || n == 0) return st;
    const bool pairs = ((uintptr_t)grads & 15u) == 0;
    float2* G = reinterpret_cast<float2*>(grads);
    const bool vec = hg_vec(pos, pstride, dL_dfeatures, stride);
#define TN_HG_BACKWARD(RUN, VEC)                                                                           \
    hg_backward_kernel<RUN, VEC><<<hg_grid(n, H.n_levels, RUN), HG_THREADS, 0, stream>>>(H, n, n_dev, pstride, \
                                                                                       stride, pos, dL_dfeatures, G, pairs)
#define TN_HG_TOUCH(ADD)                                                                                            \
    hg_touch_kernel<ADD><<<hg_grid(n, H.n_levels, 1), HG_THREADS, 0, stream>>>(                                      \
        H, n, n_dev, pstride, stride, pos, dL_dfeatures, G, pairs, touched_bits, touched_list, touched_count)
    // With a list, up to 2^17 (sample, level) pairs one launch adds and lists (1000 samples of 16 levels 15.4
    // us against 20.5 in two; 8000 uniform 25.3 against 27.7); past it the runs are worth their own (30,000 along
    // rays 50.2 against 46.1, 65,536 97 against 83).
    if (touched_bits && (uint64_t)n * H.n_levels <= (1u << 17)) {
        TN_HG_TOUCH(true);
        return check_launch("tn_hashgrid_backward");
    }
    // Eight samples a thread from 2^20 (sample, level) pairs on (2^18 samples, 16 levels: 85 us against
    // 89 with four), four below, where the GPU wants more threads (8000 samples: 5.9 against 9.1 us;
    // even at 64,000).
    if ((uint64_t)n * H.n_levels >= (1u << 20)) {
        if (vec) TN_HG_BACKWARD(8, true);
        else TN_HG_BACKWARD(8, false);
    } else {
        if (vec) TN_HG_BACKWARD(4, true);
        else TN_HG_BACKWARD(4, false);
    }
#undef TN_HG_BACKWARD
    if (touched_bits) TN_HG_TOUCH(false);
#undef TN_HG_TOUCH
    return check_launch("tn_hashgrid_backward");
}

int hashgrid_clear_touched(cudaStream_t stream, const uint32_t* touched_list, const uint32_t* touched_count,
                           uint32_t max_entries, float* grads, uint32_t* touched_bits) {
    hg_clear_kernel<<<num_sms() * 4, 256, 0, stream>>>(touched_list, touched_count, max_entries,
                                                       reinterpret_cast<float2*>(grads), touched_bits);
    int st = check_launch("tn_hashgrid_clear_touched");
    if (st == TN_OK)
        st = cuda_status(cudaMemsetAsync(const_cast<uint32_t*>(touched_count), 0, sizeof(uint32_t), stream),
                         "tn_hashgrid_clear_touched: count");
    return st;
}

// ---- the hash-grid network behind tn_network ------------------------------------------------
struct HashNet {
    tn_hashgrid_desc desc{};
    uint32_t n_features = 0;     // 2 L
    uint64_t n_hash = 0;         // hash parameters (floats): L T 2
    const float* params = nullptr;  // [hash | heads]
    float* feat = nullptr;       // [2L][cap] features of the last forward
    float* dfeat = nullptr;      // [2L][cap]
    float* qfeat = nullptr;      // [2L][qcap] features of density queries
    float* partials = nullptr;   // [blocks][HG_HEAD_SLOTS]
    uint32_t* list = nullptr;    // [L T]
    uint32_t* count = nullptr;   // [1]
    uint32_t cap = 0, qcap = 0;
    ~HashNet() {
        cudaFree(feat); cudaFree(dfeat); cudaFree(qfeat); cudaFree(partials);
        cudaFree(list); cudaFree(count);
    }
};

// Blocks of the heads' backward over up to n samples: all resident at once.
static uint32_t heads_blocks(uint32_t n) {
    return std::min((n + HG_HEAD_THREADS - 1) / HG_HEAD_THREADS, (uint32_t)(num_sms() * HG_HEAD_BLOCKS_PER_SM));
}

static const float* head_params(const HashNet* h) { return h->params + h->n_hash; }

static int hashnet_forward(void* user, tn_stream_t stream, uint32_t n, const uint32_t* n_dev, uint32_t stride,
                           const float* pos, const float* /*dir*/, float* density, float* rgb) {
    auto* h = static_cast<HashNet*>(user);
    cudaStream_t s = (cudaStream_t)stream;
    TN_REQUIRE(n <= h->cap && stride >= n, TN_E_INVALID, "hash-grid network: %u samples past its %u", n, h->cap);
    int st = hashgrid_encode(s, &h->desc, n, n_dev, stride, h->cap, pos, h->params, h->feat);
    if (st != TN_OK || n == 0) return st;
    hg_heads_forward_kernel<<<(n + 255) / 256, 256, 0, s>>>(h->n_features, n, n_dev, h->cap, h->feat,
                                                            head_params(h), density, rgb, stride);
    return check_launch("hash-grid network forward");
}

static int hashnet_density(void* user, tn_stream_t stream, uint32_t n, const uint32_t* n_dev, uint32_t stride,
                           const float* pos, float* density) {
    auto* h = static_cast<HashNet*>(user);
    cudaStream_t s = (cudaStream_t)stream;
    TN_REQUIRE(n <= h->qcap && stride >= n, TN_E_INVALID, "hash-grid density: %u queries past its %u", n,
               h->qcap);
    int st = hashgrid_encode(s, &h->desc, n, n_dev, stride, h->qcap, pos, h->params, h->qfeat);
    if (st != TN_OK || n == 0) return st;
    hg_heads_forward_kernel<<<(n + 255) / 256, 256, 0, s>>>(h->n_features, n, n_dev, h->qcap, h->qfeat,
                                                            head_params(h), density, nullptr, stride);
    return check_launch("hash-grid network density");
}

static int hashnet_backward(void* user, tn_stream_t stream, uint32_t n, const uint32_t* n_dev, uint32_t stride,
                            const float* pos, const float* /*dir*/, const float* dL_ddensity, const float* dL_drgb,
                            float* param_grads) {
    auto* h = static_cast<HashNet*>(user);
    cudaStream_t s = (cudaStream_t)stream;
    // the previous step's hash gradients (Adam has read them): a step touches most entries of the
    // fine levels, so one whole-array clear writes less than the entries' scattered sectors would
    const uint64_t entries = h->n_hash / HG_F;
    int st = cuda_status(cudaMemsetAsync(param_grads, 0, h->n_hash * sizeof(float), s), "hash-grid gradients");
    if (st == TN_OK) st = cuda_status(cudaMemsetAsync(h->count, 0, sizeof(uint32_t), s), "hash-grid count");
    if (st != TN_OK || n == 0) return st;
    const uint32_t blocks = heads_blocks(n);
    hg_heads_backward_kernel<<<blocks, HG_HEAD_THREADS, 0, s>>>(h->n_features, n, n_dev, stride, h->feat,
                                                                head_params(h), dL_ddensity, dL_drgb, h->dfeat,
                                                                h->partials);
    st = check_launch("hash-grid heads backward");
    if (st != TN_OK) return st;
    hg_heads_grad_finish_kernel<<<4 * (h->n_features + 1), HG_FINISH_THREADS, 0, s>>>(h->n_features, blocks,
                                                                                      h->partials,
                                                                                      param_grads + h->n_hash);
    st = check_launch("hash-grid heads gradients");
    if (st != TN_OK) return st;
    st = hashgrid_backward(s, &h->desc, n, n_dev, stride, h->cap, pos, h->dfeat, param_grads, nullptr, nullptr,
                           nullptr);
    if (st != TN_OK) return st;
    // the entries Adam will update: those with a nonzero gradient
    const uint32_t nz_blocks = (uint32_t)((entries + 8ull * HG_NZ_THREADS - 1) / (8ull * HG_NZ_THREADS));
    hg_nonzero_kernel<<<nz_blocks, HG_NZ_THREADS, 0, s>>>((uint32_t)entries, reinterpret_cast<const float4*>(param_grads),
                                                          h->list, h->count);
    return check_launch("hash-grid nonzero entries");
}

// A network over the parameters `params` ([hash entries | heads]) for batches of up to `cap`
// samples (positions with that stride) and density queries of up to `qcap`.
int hashnet_create(const tn_hashgrid_desc* desc, const float* params, uint32_t cap, uint32_t qcap, tn_network* out,
                   void** handle) {
    HashLevels H;
    int st = hash_levels(desc, H);
    if (st != TN_OK) return st;
    auto* h = new HashNet();
    h->desc = *desc;
    h->n_features = HG_F * desc->n_levels;
    h->n_hash = (uint64_t)desc->n_levels << (desc->log2_hashmap_size + 1);
    h->params = params;
    h->cap = cap;
    h->qcap = std::max(qcap, 1u);
    const uint64_t entries = h->n_hash / HG_F;
    const uint32_t blocks = heads_blocks(cap);
    st = cuda_status(cudaMalloc(&h->feat, (size_t)h->n_features * cap * sizeof(float)), "hash-grid features");
    if (st == TN_OK) st = cuda_status(cudaMalloc(&h->dfeat, (size_t)h->n_features * cap * sizeof(float)), "hash-grid dfeat");
    if (st == TN_OK)
        st = cuda_status(cudaMalloc(&h->qfeat, (size_t)h->n_features * h->qcap * sizeof(float)), "hash-grid query features");
    if (st == TN_OK)
        st = cuda_status(cudaMalloc(&h->partials, (size_t)std::max(blocks, 1u) * HG_HEAD_SLOTS * sizeof(float)),
                         "hash-grid partials");
    if (st == TN_OK) st = cuda_status(cudaMalloc(&h->list, (size_t)entries * sizeof(uint32_t)), "hash-grid list");
    if (st == TN_OK) st = cuda_status(cudaMalloc(&h->count, sizeof(uint32_t)), "hash-grid count");
    if (st == TN_OK) st = cuda_status(cudaMemset(h->count, 0, sizeof(uint32_t)), "hash-grid count");
    if (st != TN_OK) {
        delete h;
        return st;
    }
    out->user = h;
    out->activation = TN_ACT_DENSITY;
    out->forward = hashnet_forward;
    out->backward = hashnet_backward;
    out->density = hashnet_density;
    *handle = h;
    return TN_OK;
}

void hashnet_destroy(void* handle) { delete static_cast<HashNet*>(handle); }

// Entries with a nonzero gradient after the last backward (device count, and *list: the
// entries, in no particular order), for inspection and tests.
const uint32_t* hashnet_touched(void* handle, const uint32_t** list) {
    auto* h = static_cast<HashNet*>(handle);
    if (list) *list = h->list;
    return h->count;
}

}  // namespace tn

using namespace tn;

extern "C" {

int tn_hashgrid_n_params(const tn_hashgrid_desc* desc, uint64_t* n_hash, uint32_t* n_head) {
    HashLevels H;
    int st = hash_levels(desc, H);
    if (st != TN_OK) return st;
    if (n_hash) *n_hash = (uint64_t)desc->n_levels << (desc->log2_hashmap_size + 1);
    if (n_head) *n_head = 4 * (HG_F * desc->n_levels + 1);
    return TN_OK;
}

int tn_hashgrid_level_resolution(const tn_hashgrid_desc* desc, uint32_t level, uint32_t* resolution,
                                 int* dense) {
    HashLevels H;
    int st = hash_levels(desc, H);
    if (st != TN_OK) return st;
    TN_REQUIRE(level < desc->n_levels, TN_E_INVALID, "level %u past %u", level, desc->n_levels);
    if (resolution) *resolution = H.res[level];
    if (dense) *dense = (int)H.dense[level];
    return TN_OK;
}

int tn_hashgrid_encode(tn_stream_t stream, const tn_hashgrid_desc* desc, uint32_t n, const uint32_t* n_dev,
                       uint32_t stride, const float* pos, const float* params, float* features) {
    TN_NONNULL(pos); TN_NONNULL(params); TN_NONNULL(features);
    TN_REQUIRE(stride >= n, TN_E_INVALID, "stride %u < n %u", stride, n);
    return hashgrid_encode((cudaStream_t)stream, desc, n, n_dev, stride, stride, pos, params, features);
}

int tn_hashgrid_backward(tn_stream_t stream, const tn_hashgrid_desc* desc, uint32_t n, const uint32_t* n_dev,
                         uint32_t stride, const float* pos, const float* dL_dfeatures, float* grads,
                         uint32_t* touched_bits, uint32_t* touched_list, uint32_t* touched_count) {
    TN_NONNULL(pos); TN_NONNULL(dL_dfeatures); TN_NONNULL(grads);
    TN_REQUIRE(stride >= n, TN_E_INVALID, "stride %u < n %u", stride, n);
    TN_REQUIRE((touched_bits == nullptr) == (touched_list == nullptr) &&
                   (touched_list == nullptr) == (touched_count == nullptr),
               TN_E_INVALID, "touched_bits, touched_list and touched_count go together");
    return hashgrid_backward((cudaStream_t)stream, desc, n, n_dev, stride, stride, pos, dL_dfeatures, grads,
                             touched_bits, touched_list, touched_count);
}

int tn_hashgrid_clear_touched(tn_stream_t stream, const uint32_t* touched_list, const uint32_t* touched_count,
                              uint32_t max_entries, float* grads, uint32_t* touched_bits) {
    TN_NONNULL(touched_list); TN_NONNULL(touched_count); TN_NONNULL(grads);
    return hashgrid_clear_touched((cudaStream_t)stream, touched_list, touched_count, max_entries, grads,
                                  touched_bits);
}

}  // extern "C"
