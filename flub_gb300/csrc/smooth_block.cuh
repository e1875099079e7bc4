// Several red-black half-sweeps of a level in one launch, by tiles.
//
// On levels of a few hundred thousand cells a half-sweep is two to three
// microseconds of launch, dependent loads and drain for a fraction of a
// microsecond of work, and the reference schedule runs 6 << l iterations per
// side at level l.  Here a block loads a tile of the level with a halo of S
// cells (z, r and item words, split by colour) into shared memory and runs S
// half-sweeps on it, each on a region one cell smaller, so that after the last
// one the tile itself is right; the halo cells it updates on the way are what
// the neighbouring blocks compute, bit for bit.  One launch of S = 4 replaces
// four, at the price of 2.6 times the updates at 4 x 8 x 64.
//
// A tile is TI x kTJb rows of up to kKB cells; along k the halo is 8 cells, and
// levels with rows of at most kKB + 16 cells have none.  Threads own V cells of
// one colour in a row and walk along i, so that a half-sweep reads each row of
// the other colour once for its three uses along i.  The output goes to
// another buffer than the input (neighbouring tiles still read it); tiles
// without fluid are not in the list, and both buffers hold 0 there.
//
// Bound by shared-memory bandwidth in the sweeps (half of a launch) and by the
// load's latency before them.  Measured per half-sweep, four in a launch, dam
// layout / full of fluid: 64^3 2.2 / 3.2 -> 1.25 / 1.2 us, 52 x 36 x 44 and
// its like (rows of 4 k cells, scalar sweeps before) 2.7 -> 1.3 us.
#pragma once

#include "coarse.cuh"
#include "store.cuh"

namespace flub {

constexpr int kBlockThreads = 512;
constexpr int kTJb = 8, kKB = 64, kKHalo = 8;

enum BlockMode { kBlockFromZero = 0, kBlockPlain = 1, kBlockProlong = 2 };

// What a half-sweep has to know of an item (V cells of one colour in a row),
// in one word per colour: a nibble per cell with its diagonal count (0: never
// updated), kItemAny when a count is not 0, kItemSolid when a neighbour does not
// count although it lies in the domain, kItemAir when one is air, and at level 0,
// whose residual can hold anything off the fluid, kItemPart when some counts are 0 and
// others not.  Built once by set_tags; an
// item without kItemSolid needs no stencil words: a neighbour outside the
// domain is replaced by the cell itself, whose term is then 0.
constexpr uint32_t kAllCount = 0x1554u;  // sw_ns of a cell whose six neighbours all count
constexpr uint32_t kItemAny = 1u << 16, kItemSolid = 1u << 17, kItemAir = 1u << 18,
                   kItemPart = 1u << 19;

struct BlockArgs {
    Dims D;
    const uint32_t *tiles;        // tiles that hold fluid: ti | tj << 11 | tk << 22
    const int *tiles_n;           // their number
    const uint32_t *items;        // item words: colour 0 of every item of the level, then colour 1
    const uint16_t *cw;           // stencil words, natural order
    const void *r, *zin, *zc;     // residual, input z (not kBlockFromZero), next level's z (kBlockProlong)
    void *zout;
    float zc_scale;
    int mode, first_odd;  // first_odd: the odd colour is updated first (pre-smoothing)
    int ks;               // floats of one colour per row in shared memory
};

// Bytes of shared memory for tiles of TI planes with halo h, items of V cells.
static inline size_t block_smem(int ti, int h, int ks, int V) {
    const size_t cells = (size_t)(ti + 2 * h) * (kTJb + 2 * h) * ks;
    return 64 + 2 * cells * (4 + 4) + 2 * cells / V * 4;
}

// V consecutive values of a natural row (aligned to V values).
template <int V, typename T>
__device__ __forceinline__ void ld_nat(const T *p, float *o) {
    if constexpr (V == 4)
        St<T>::ld4_in(p, o);
    else
        St<T>::ld2_in(p, o);
}
template <int V, typename T>
__device__ __forceinline__ void st_nat(T *p, const float *v) {
    if constexpr (V == 4) {
        St<T>::st4(p, v);
    } else {
#pragma unroll
        for (int m = 0; m < V; m++) St<T>::st(p + m, v[m]);
    }
}

// z + (r + L z) / d on V cells of one colour (coarse_half's sequence); a
// neighbour that does not count holds the cell's own value.
template <int V>
__device__ __forceinline__ void block_update(uint32_t item, float *xc, const float *ip, const float *im,
                                             const float *jp, const float *jm, const float *va, const float *vb,
                                             const float *r, const float2 *lut) {
    static_assert(V % 2 == 0, "two cells at a time");
    constexpr int h = 1;
#pragma unroll
    for (int m = 0; m < V; m += 2) {
        const F2 x = f2(xc[m], xc[m + h]);
        F2 s = f2_add(f2_sub(f2(ip[m], ip[m + h]), x), f2_sub(f2(im[m], im[m + h]), x));
        s = f2_add(s, f2_add(f2_sub(f2(jp[m], jp[m + h]), x), f2_sub(f2(jm[m], jm[m + h]), x)));
        s = f2_add(s, f2_add(f2_sub(f2(va[m], va[m + h]), x), f2_sub(f2(vb[m], vb[m + h]), x)));
        const float2 l0 = lut[(item >> (4 * m)) & 7u], l1 = lut[(item >> (4 * (m + h))) & 7u];
        const F2 a = f2_add(f2(r[m], r[m + h]), s), y = f2(l0.x, l1.x), q0 = f2_mul(a, y);
        f2_get(f2_sub(x, f2_fma(f2_fma(q0, f2(l0.y, l1.y), a), y, q0)), xc[m], xc[m + h]);
    }
}

// FP16 levels: a value as its storage holds it.
template <typename T>
__device__ __forceinline__ float as_stored(float v) {
    if constexpr (std::is_same<T, __half>::value) return __half2float(__float2half_rn(v));
    return v;
}

// T: storage of r, z and zc (float, or __half in mixed precision: each update
// is rounded to it).  TI: planes of a tile.  S: half-sweeps.  kAnyR: level 0, whose
// residual can hold anything off the fluid (elsewhere the restriction leaves 0); its
// test in the other levels' kernels cost 1 % of a solve on rows of 4 k cells.
template <int V, typename T, int TI, int S, bool kAnyR>
__global__ void __launch_bounds__(kBlockThreads, 1) k_smooth_block(const BlockArgs A, unsigned long long *kc) {
    constexpr int RI = TI + 2 * S, RJ = kTJb + 2 * S;
    extern __shared__ __align__(16) unsigned char block_smem_[];
    pdl_open();
    const Dims D = A.D;
    const int KS = A.ks, half = RI * RJ * KS, ihalf = half / V, irow = KS / V;
    float2 *lut = reinterpret_cast<float2 *>(block_smem_);
    float *z0 = reinterpret_cast<float *>(block_smem_ + 64), *z1 = z0 + half, *r0 = z1 + half;
    uint32_t *w0 = reinterpret_cast<uint32_t *>(r0 + 2 * half);
    if (threadIdx.x < 8)
        lut[threadIdx.x] = make_float2(threadIdx.x ? __fdiv_rn(-1.0f, (float)threadIdx.x) : 0.0f, (float)threadIdx.x);
    // the list entry together with the count it is valid under (the list is as
    // long as the grid is wide)
    uint32_t tile = __ldg(A.tiles + blockIdx.x);
    const int total = *A.tiles_n;
    const int lsegs = D.nz / (2 * V), litems = D.nx * D.ny * lsegs;
    bool waited = false;
    for (int t = blockIdx.x; t < total; t += gridDim.x) {
        const int ib = (int)(tile & 2047u) * TI, jb = (int)((tile >> 11) & 2047u) * kTJb, kb = (int)(tile >> 22) * kKB;
        const int kout = min(D.nz <= kKB + 2 * kKHalo ? D.nz : kKB, D.nz - kb);
        const int kr = max(0, kb - kKHalo), kw = min(D.nz, kb + kout + kKHalo) - kr;
        const int segs = kw / (2 * V);
        // workers: groups of `segs` threads, one row each at a time
        const int worker = threadIdx.x / segs, seg = threadIdx.x - worker * segs, workers = kBlockThreads / segs;
        const int rows = worker < workers ? RI * RJ : 0;
        // four rows of a worker at a time, so that their loads are in flight together
        constexpr int U = 4;
        // row -> the item's offset in a half, in the level's items and cells; false outside the domain
        auto place = [&](int row, int &at, int &par, int &le, int &i, int &j) {
            i = ib - S + row / RJ;
            j = jb - S + row % RJ;
            at = row * KS + seg * V;
            par = (i + j) & 1;
            le = (i * D.ny + j) * lsegs + kr / (2 * V) + seg;
            return row < RI * RJ && i >= 0 && i < D.nx && j >= 0 && j < D.ny;
        };
        if (!waited) {
            pdl_wait(kc);
            waited = true;
        }
        const T *gr = static_cast<const T *>(A.r), *gz = static_cast<const T *>(A.zin), *gc = static_cast<const T *>(A.zc);
        for (int q = worker; q < rows; q += U * workers) {
            float zn[U][2 * V], rn[U][2 * V];
            uint32_t we[U], wo[U];
#pragma unroll
            for (int u = 0; u < U; u++) {
                we[u] = wo[u] = 0u;
#pragma unroll
                for (int m = 0; m < 2 * V; m++) zn[u][m] = rn[u][m] = 0.0f;
                int at, par, le, i, j;
                if (!place(q + u * workers, at, par, le, i, j)) continue;
                const int c = le * (2 * V);
                we[u] = __ldg(A.items + le);
                wo[u] = __ldg(A.items + litems + le);
                ld_nat<V>(gr + c, rn[u]);
                ld_nat<V>(gr + c + V, rn[u] + V);
                if (A.mode != kBlockFromZero) {
                    ld_nat<V>(gz + c, zn[u]);
                    ld_nat<V>(gz + c + V, zn[u] + V);
                }
            }
#pragma unroll
            for (int u = 0; u < U; u++) {
                const int row = q + u * workers;
                if (row >= RI * RJ) break;
                int at, par, le, i, j;
                const bool in = place(row, at, par, le, i, j);
                float ze[V], zo[V], re[V], ro[V];
#pragma unroll
                for (int m = 0; m < V; m++) {
                    ze[m] = par ? zn[u][2 * m + 1] : zn[u][2 * m];
                    zo[m] = par ? zn[u][2 * m] : zn[u][2 * m + 1];
                    re[m] = par ? rn[u][2 * m + 1] : rn[u][2 * m];
                    ro[m] = par ? rn[u][2 * m] : rn[u][2 * m + 1];
                }
                if (kAnyR && ((we[u] | wo[u]) & kItemPart)) {
                    // 0 on the cells that are never updated: their factor 0 would turn a
                    // caller's infinity there into NaN, and an air cell's z is read
#pragma unroll
                    for (int m = 0; m < V; m++) {
                        re[m] = (we[u] >> (4 * m)) & 7u ? re[m] : 0.0f;
                        ro[m] = (wo[u] >> (4 * m)) & 7u ? ro[m] : 0.0f;
                    }
                }
                if (A.mode == kBlockProlong && in) {
                    // z stays 0 on the cells that are never updated
                    float cv[V];
                    ld_nat<V>(gc + ((i >> 1) * (D.ny >> 1) + (j >> 1)) * (D.nz >> 1) + (kr >> 1) + V * seg, cv);
#pragma unroll
                    for (int m = 0; m < V; m++) {
                        const float add = __fmul_rn(cv[m], A.zc_scale);
                        ze[m] = (we[u] >> (4 * m)) & 7u ? __fadd_rn(ze[m], add) : 0.0f;
                        zo[m] = (wo[u] >> (4 * m)) & 7u ? __fadd_rn(zo[m], add) : 0.0f;
                    }
                }
                w0[row * irow + seg] = we[u];
                w0[ihalf + row * irow + seg] = wo[u];
                st_vec<V>(z0 + at, ze);
                st_vec<V>(z1 + at, zo);
                st_vec<V>(r0 + at, re);
                st_vec<V>(r0 + half + at, ro);
            }
        }
        __syncthreads();
#pragma unroll
        for (int s = 0; s < S; s++) {
            constexpr int kJ = RJ - 2, kI = RI - 2;
            const int nj = kJ - 2 * s, ni = kI - 2 * s;  // rows updated along j and i
            const int slices = workers / nj, chunk = (ni + slices - 1) / slices;
            const int sl = worker / nj, rj = s + 1 + worker - sl * nj, j = jb - S + rj;
            // this worker's rows, those in the domain
            const int a0 = max(s + 1 + sl * chunk, S - ib);
            const int a1 = min(min(s + 1 + (sl + 1) * chunk, s + 1 + ni), D.nx - ib + S);
            const bool odd = ((s & 1) == 0) == (A.first_odd != 0);
            float *zu = odd ? z1 : z0;
            const float *zv = odd ? z0 : z1, *ru = r0 + (odd ? half : 0);
            const uint32_t *wu = w0 + (odd ? ihalf : 0);
            if (worker < workers && sl < slices && a0 < a1 && j >= 0 && j < D.ny) {
                int at = (a0 * RJ + rj) * KS + seg * V;
                float im[V], va[V], ip[V];
                ld_vec<V>(ib - S + a0 > 0 ? zv + at - RJ * KS : zu + at, im);
                ld_vec<V>(zv + at, va);
                for (int ri = a0; ri < a1; ri++, at += RJ * KS) {
                    const int i = ib - S + ri;
                    const uint32_t item = wu[(ri * RJ + rj) * irow + seg];
                    ld_vec<V>(i + 1 < D.nx ? zv + at + RJ * KS : zu + at, ip);
                    if (item & kItemAny) {
                        float jp[V], jm[V], vb[V], xc[V], rr[V];
                        ld_vec<V>(j + 1 < D.ny ? zv + at + KS : zu + at, jp);
                        ld_vec<V>(j > 0 ? zv + at - KS : zu + at, jm);
                        ld_vec<V>(zu + at, xc);
                        ld_vec<V>(ru + at, rr);
                        // q: the cells sit at odd k offsets; their k neighbours are va and, one further, vb.
                        // At the ends of the region the cell itself: a wall, or in the part of the halo that is
                        // wrong by then
                        const bool q = (odd ? 1 : 0) ^ ((i + j) & 1);
                        const bool end = q ? seg == segs - 1 : seg == 0;
                        const float e = end ? zu[q ? at + V - 1 : at] : zv[q ? at + V : at - 1];
#pragma unroll
                        for (int m = 0; m < V; m++) {
                            const float up = m + 1 < V ? va[m + 1 < V ? m + 1 : m] : e;
                            const float dn = m > 0 ? va[m > 0 ? m - 1 : m] : e;
                            vb[m] = q ? up : dn;
                        }
                        if (item & kItemSolid) {
                            // solids next to it: the neighbours that do not count become the cell itself
                            const uint16_t *w = A.cw + (int64_t)(i * D.ny + j) * D.nz + kr + 2 * V * seg + (q ? 1 : 0);
                            float ti[V], tm[V], tj[V], tn[V], ta[V], tb[V];
#pragma unroll
                            for (int m = 0; m < V; m++) {
                                const uint32_t ns = sw_ns(__ldg(w + 2 * m));
                                ti[m] = ns & 4u ? ip[m] : xc[m];
                                tm[m] = ns & 16u ? im[m] : xc[m];
                                tj[m] = ns & 64u ? jp[m] : xc[m];
                                tn[m] = ns & 256u ? jm[m] : xc[m];
                                ta[m] = ns & (q ? 4096u : 1024u) ? va[m] : xc[m];
                                tb[m] = ns & (q ? 1024u : 4096u) ? vb[m] : xc[m];
                            }
                            block_update<V>(item, xc, ti, tm, tj, tn, ta, tb, rr, lut);
                        } else {
                            block_update<V>(item, xc, ip, im, jp, jm, va, vb, rr, lut);
                        }
#pragma unroll
                        for (int m = 0; m < V; m++) xc[m] = as_stored<T>(xc[m]);
                        st_vec<V>(zu + at, xc);
                    }
#pragma unroll
                    for (int m = 0; m < V; m++) {
                        im[m] = va[m];
                        va[m] = ip[m];
                    }
                }
            }
            __syncthreads();
            if (std::is_same<T, __half>::value && s == 0 && A.mode == kBlockProlong) {
                // the first half-sweep read the prolonged values unrounded, as
                // the sweep fused with the prolongation does; from here on the
                // colour it did not update is what its storage would hold
                float *zr = odd ? z0 : z1;
                for (int q = worker; q < rows; q += workers) {
                    float v[V];
                    ld_vec<V>(zr + q * KS + seg * V, v);
#pragma unroll
                    for (int m = 0; m < V; m++) v[m] = as_stored<T>(v[m]);
                    st_vec<V>(zr + q * KS + seg * V, v);
                }
                __syncthreads();
            }
        }
        // the tile, in natural order
        const int so = kout / (2 * V), skip = (kb - kr) / (2 * V);
        for (int row = worker; row < (seg >= skip && seg < skip + so ? TI * kTJb : 0) && worker < workers;
             row += workers) {
            const int a = row / kTJb, b = row % kTJb, i = ib + a, j = jb + b;
            if (i >= D.nx || j >= D.ny) continue;
            const int at = ((a + S) * RJ + b + S) * KS + seg * V, par = (i + j) & 1;
            float ev[V], od[V], n[2 * V];
            ld_vec<V>(z0 + at, ev);
            ld_vec<V>(z1 + at, od);
#pragma unroll
            for (int m = 0; m < V; m++) {
                n[2 * m] = par ? od[m] : ev[m];
                n[2 * m + 1] = par ? ev[m] : od[m];
            }
            T *o = static_cast<T *>(A.zout) + (i * D.ny + j) * D.nz + kr + 2 * V * seg;
            st_nat<V>(o, n);
            st_nat<V>(o + V, n + V);
        }
        if (t + (int)gridDim.x < total) {
            tile = __ldg(A.tiles + t + gridDim.x);
            __syncthreads();  // the next tile overwrites what this one reads
        }
    }
    if (!waited) pdl_wait(kc);
}

// The item words of the 2 V cells of a row from k0 on, from their stencil words
// (two in each element of wd).  part: kItemPart is kept.
template <int V>
__device__ __forceinline__ void item_words(const uint32_t (&wd)[V], const Dims D, int i, int j, int k0, bool part,
                                           uint32_t (&out)[2]) {
    const int par = (i + j) & 1;
    uint32_t ab[2] = {0u, 0u};  // of the cells k0 + 0, 2, .. and k0 + 1, 3, ..
    int updated[2] = {0, 0};
#pragma unroll
    for (int m = 0; m < 2 * V; m++) {
        const uint32_t w = (wd[m >> 1] >> (16 * (m & 1))) & 0xffffu;
        const int k = k0 + m;
        if ((w & 3u) != kCodeFluid) continue;
        const uint32_t ns = sw_ns(w), d = __popc(ns);
        uint32_t inside = kAllCount;  // the neighbours that lie in the domain
        if (i + 1 >= D.nx) inside &= ~4u;
        if (i == 0) inside &= ~16u;
        if (j + 1 >= D.ny) inside &= ~64u;
        if (j == 0) inside &= ~256u;
        if (k + 1 >= D.nz) inside &= ~1024u;
        if (k == 0) inside &= ~4096u;
        uint32_t &o = ab[m & 1];
        o |= d << (4 * (m >> 1));
        if (d) {
            o |= kItemAny;
            updated[m & 1]++;
        }
        if (d && ns != inside) o |= kItemSolid;
        if (d && (w & kAllCount)) o |= kItemAir;  // the low bit of a neighbour's code
    }
#pragma unroll
    for (int c = 0; c < 2; c++)
        if (part && updated[c] > 0 && updated[c] < V) ab[c] |= kItemPart;
    out[0] = par ? ab[1] : ab[0];
    out[1] = par ? ab[0] : ab[1];
}

// The item words of a level whose rows are not whole 8-cell groups (V = 2).
template <int V>
__global__ void __launch_bounds__(256) k_block_items(const uint16_t *cw, Dims D, bool part, uint32_t *items) {
    setup_open();
    const int lsegs = D.nz / (2 * V), n = D.nx * D.ny * lsegs;
    for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < n; e += gridDim.x * blockDim.x) {
        const int seg = e % lsegs, row = e / lsegs, j = row % D.ny, i = row / D.ny;
        uint32_t wd[V], out[2];
#pragma unroll
        for (int m = 0; m < V; m++) wd[m] = reinterpret_cast<const uint32_t *>(cw)[(int64_t)e * V + m];
        item_words<V>(wd, D, i, j, 2 * V * seg, part, out);
        items[e] = out[0];
        items[n + e] = out[1];
    }
}

}  // namespace flub
