// What new tags set up on every level, in a few launches over all levels at once:
// the solver's lists and words, and the buffers that have to hold 0 again.
//
// On small grids this is launches, each of them a dependent kernel of
// microseconds of latency for less of work: level by level it took about ten a
// level (encode, restrict, words, split words, items, count, scan, write, clears).
// Here a launch covers all levels, its blocks dealt out by the prefix sums in its
// parameters, a group's words, split words, items and count come from one reading
// of its codes, and the launches are programmatic dependents of one another.
// set_tags: 32^3 on 3 levels 103 -> 23 us, 64^3 on 4 151 -> 28, 256 x 64 x 256 on 4
// 189 -> 49, 256^3 on 6 330 -> 132.
#pragma once

#include "coarse.cuh"
#include "smooth_block.cuh"

namespace flub {

constexpr int kSetupMaxLevels = 12;
constexpr int kSetupThreads = 256;  // groups of 8 cells per block

struct SetupLevel {
    Dims D;
    const uint8_t *code;
    uint16_t *sw, *sws;  // stencil words, and colour-split (NULL: not kept)
    uint32_t *items;     // item words (NULL: not kept)
    int *act, *act_n;    // active groups, ascending, and their number
    int first;           // the level's first block
    bool part;           // items with kItemPart: level 0
};

struct SetupParams {
    SetupLevel lv[kSetupMaxLevels];
    int n, blocks;  // levels with nz % 8 == 0, blocks of all
    int *bcount;    // active groups per block, then their exclusive sums within a level
};

template <typename P>
__device__ __forceinline__ int setup_level(const P &p, int block) {
    int l = 0;
    while (l + 1 < p.n && block >= p.lv[l + 1].first) l++;
    return l;
}

// One thread per group: its 8 stencil words, the same split by colour, its two
// item words; per block the number of active groups.
__global__ void __launch_bounds__(kSetupThreads) k_setup_words(const __grid_constant__ SetupParams P) {
    setup_open();
    const SetupLevel &L = P.lv[setup_level(P, blockIdx.x)];
    const Dims D = L.D;
    const int g = ((int)blockIdx.x - L.first) * kSetupThreads + (int)threadIdx.x, ng = (int)(D.n() >> 3);
    bool fluid = false;
    if (g < ng) {
        int i, j, kg;
        group_ijk(g, D, i, j, kg);
        const uint4 u = words8_from_codes<true>(L.code, D, i, j, kg << 3, g << 3);
        fluid = words_have_fluid(u);
        *reinterpret_cast<uint4 *>(L.sw + ((int64_t)g << 3)) = u;
        const uint32_t wd[4] = {u.x, u.y, u.z, u.w};
        const int p = (i + j) & 1;
        if (L.sws) {
            // natural cell (i, j, k) -> element k >> 1 of row (i, j) in half (i + j + k) & 1
            const int hz = D.nz >> 1, hn = (int)(D.n() >> 1), h = (i * D.ny + j) * hz + 4 * kg;
            const uint2 a = make_uint2(__byte_perm(u.x, u.y, 0x5410), __byte_perm(u.z, u.w, 0x5410));  // k even
            const uint2 b = make_uint2(__byte_perm(u.x, u.y, 0x7632), __byte_perm(u.z, u.w, 0x7632));  // k odd
            *reinterpret_cast<uint2 *>(L.sws + h) = p ? b : a;
            *reinterpret_cast<uint2 *>(L.sws + hn + h) = p ? a : b;
        }
        if (L.items) {
            uint32_t out[2];
            item_words<4>(wd, D, i, j, kg << 3, L.part, out);
            L.items[g] = out[0];
            L.items[ng + g] = out[1];
        }
    }
    const int total = __syncthreads_count(fluid);
    if (threadIdx.x == 0) P.bcount[blockIdx.x] = total;
}

// Exclusive sums of a level's block counts in place, the total to *act_n: one block a level.
__global__ void __launch_bounds__(1024) k_setup_scan(const __grid_constant__ SetupParams P) {
    __shared__ int wsum[32];
    setup_open();
    const SetupLevel &L = P.lv[blockIdx.x];
    const int nb = ((int)blockIdx.x + 1 < P.n ? P.lv[blockIdx.x + 1].first : P.blocks) - L.first;
    int *c = P.bcount + L.first;
    const int per = (nb + 1023) / 1024, b0 = min(nb, (int)threadIdx.x * per), b1 = min(nb, b0 + per);
    int s = 0;
    for (int b = b0; b < b1; b++) s += c[b];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int in = s;  // inclusive over the warp
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, in, o);
        if (lane >= o) in += v;
    }
    if (lane == 31) wsum[warp] = in;
    __syncthreads();
    if (warp == 0) {
        int w = wsum[lane];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int v = __shfl_up_sync(0xffffffffu, w, o);
            if (lane >= o) w += v;
        }
        wsum[lane] = w;
        if (lane == 31) *L.act_n = w;
    }
    __syncthreads();
    int run = in - s + (warp > 0 ? wsum[warp - 1] : 0);
    for (int b = b0; b < b1; b++) {
        const int v = c[b];
        c[b] = run;
        run += v;
    }
}

// The active groups, ascending.
__global__ void __launch_bounds__(kSetupThreads) k_setup_write(const __grid_constant__ SetupParams P) {
    __shared__ int wcount[kSetupThreads / 32];
    setup_open();
    const SetupLevel &L = P.lv[setup_level(P, blockIdx.x)];
    const int g = ((int)blockIdx.x - L.first) * kSetupThreads + (int)threadIdx.x;
    const bool f = g < (int)(L.D.n() >> 3) && group_has_fluid(load_codes8<true>(L.code + ((int64_t)g << 3)));
    const unsigned m = __ballot_sync(0xffffffffu, f);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (lane == 0) wcount[warp] = __popc(m);
    __syncthreads();
    int at = P.bcount[blockIdx.x] + __popc(m & ((1u << lane) - 1u));
    for (int w = 0; w < warp; w++) at += wcount[w];
    if (f) L.act[at] = g;
}

// The tiles of the blocked smoothing's levels that hold a fluid cell, in any
// order (they do not depend on each other).  One block per tile; *n is 0 before.
struct TileLevel {
    Dims D;
    const uint8_t *code;
    int ti, ntj, ntk, first;
    uint32_t *tiles;
    int *count;
};

struct TileParams {
    TileLevel lv[kSetupMaxLevels];
    int n;
};

__global__ void __launch_bounds__(128) k_setup_tiles(const __grid_constant__ TileParams P) {
    setup_open();
    const TileLevel &L = P.lv[setup_level(P, blockIdx.x)];
    const Dims D = L.D;
    const int tile = (int)blockIdx.x - L.first, tk = tile % L.ntk, tq = tile / L.ntk;
    const int ib = (tq / L.ntj) * L.ti, jb = (tq % L.ntj) * kTJb, kb = L.ntk > 1 ? tk * kKB : 0;
    const int kn = L.ntk > 1 ? min(kKB, D.nz - kb) : D.nz;
    bool any = false;
    for (int e = threadIdx.x; e < L.ti * kTJb * kn; e += blockDim.x) {
        const int k = e % kn, row = e / kn, i = ib + row / kTJb, j = jb + row % kTJb;
        if (i < D.nx && j < D.ny) any |= L.code[((int64_t)i * D.ny + j) * D.nz + kb + k] == kCodeFluid;
    }
    if (__syncthreads_or(any) && threadIdx.x == 0)
        L.tiles[atomicAdd(L.count, 1)] = (uint32_t)(tq / L.ntj) | (uint32_t)(tq % L.ntj) << 11 | (uint32_t)tk << 22;
}

// Buffers to clear, in units of 16 bytes.
constexpr int kClearMax = 5 * kSetupMaxLevels + 1, kClearChunk = 16 * kSetupThreads;
struct ClearRange {
    uint4 *p;
    unsigned n;
    int first;  // the range's first block
};
struct ClearParams {
    ClearRange lv[kClearMax];
    int n;
};

__global__ void __launch_bounds__(kSetupThreads) k_setup_clear(const __grid_constant__ ClearParams P) {
    setup_open();
    const ClearRange &R = P.lv[setup_level(P, blockIdx.x)];
    const int64_t base = (int64_t)((int)blockIdx.x - R.first) * kClearChunk + threadIdx.x;
#pragma unroll
    for (int u = 0; u < kClearChunk / kSetupThreads; u++)
        if (base + u * kSetupThreads < R.n) R.p[base + u * kSetupThreads] = make_uint4(0u, 0u, 0u, 0u);
}

// k_restrict_codes for fine rows of whole 8-cell groups: four coarse cells a
// thread.  With solid 0, air 1 and fluid 2 the bitwise or of the 8 children has bit
// 0 for air and bit 1 for fluid.
__global__ void __launch_bounds__(256) k_restrict_codes8(const uint8_t *cf, uint8_t *cc, Dims C) {
    setup_open();
    const int n4 = (int)(C.n() >> 2);
    for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < n4; q += gridDim.x * blockDim.x) {
        int I, J, K4;
        group_ijk(q, Dims{C.nx, C.ny, C.nz << 1}, I, J, K4);  // the coarse grid read as 4-cell groups
        const int fz = 2 * C.nz, fy = 2 * C.ny;
        const uint8_t *r = cf + ((int64_t)(2 * I) * fy + 2 * J) * fz + 8 * K4;
        const uint2 a = load_codes8<true>(r), b = load_codes8<true>(r + fz),
                    c = load_codes8<true>(r + (int64_t)fy * fz), d = load_codes8<true>(r + (int64_t)fy * fz + fz);
        const uint32_t x = a.x | b.x | c.x | d.x, y = a.y | b.y | c.y | d.y;
        const uint32_t v = __byte_perm(x | (x >> 8), y | (y >> 8), 0x6420);
        const uint32_t air = v & 0x01010101u;
        reinterpret_cast<uint32_t *>(cc)[q] = air | (v & 0x02020202u & ~(air << 1));
    }
}

}  // namespace flub
