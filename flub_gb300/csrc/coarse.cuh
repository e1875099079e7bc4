// The coarse part of the V-cycle, from a level of at most 65,536 cells down to
// the bottom and back, in ONE launch.
//
// Below that size a red-black half-sweep is microseconds of launch latency for
// a fraction of a microsecond of work, and the reference schedule runs 6 << l
// iterations per side at level l (multigrid/mgpcg.py:296-349).  Levels of more
// than kBlockCells cells are split over a thread-block cluster, each block
// holding a slab of i-planes in its shared memory; levels of at most that many
// run in block 0 alone, with block barriers.
//
// What bounds a half-sweep is its chain -- shared loads, nine dependent FP32
// operations, the store, the barrier -- and the issue slots of one SM, so the
// sweeps keep everything but the neighbours in registers:
//   - z is stored split by colour (as smooth_split.cuh does at level 0): a
//     thread owns V cells of each colour in one row, reads the other colour's
//     four neighbour rows as one vector each and has its k neighbours but one
//     in registers already;
//   - a cell's six "neighbour counts" flags are weights 2 or 0 in one byte
//     each, expanded to a float by one byte permute, so walls, solids and air
//     cost no branch: the sum of the six terms comes out doubled, which is
//     exact, and is halved inside the FMA that adds r;
//   - the division by the diagonal count is Markstein's FMA correction with
//     the cell's 1/d in a register.
// Same FP32 operations in the same order as the other smoothing kernels, cell
// by cell, so the V-cycle is bit-identical.
//
// Measured per half-sweep (slope over the iteration count, full grids / the dam
// layout), against one cluster barrier per half-sweep on natural-order z with
// six scalar neighbour loads a cell: 32^3 2.1 / 1.4 -> 0.47 / 0.41 us, 16^3 in
// one block 0.40 -> 0.37 / 0.23 us, 64 x 16 x 64 in one launch each 2.6 -> 0.6
// us.  At 32^3 the exchange of planes is 0.27 us of it.  What a launch costs
// beside its half-sweeps (reading words and residual, changing levels) is
// latency as well, so its loads are issued in batches and the correction that
// the whole cluster prolongates from block 0 is copied row by row first: 21.1
// -> 19.2 us on three levels from 32^3.
//
// A block stores its first and last plane of each half-sweep into the
// neighbouring blocks' ghost planes (distributed shared memory) and waits for
// its own (CoarseSync).  Cluster barriers come only where the levels change
// hands between the cluster and block 0; all blocks run the same sequence of
// them.
#pragma once

#include <cuda_fp16.h>

#include <type_traits>

#include "mg_kernels.cuh"
#include "smooth8.cuh"

namespace flub {

constexpr int kCoarseThreads = 256;  // 255 registers a thread: see coarse_level
constexpr int kCoarseMaxLevels = 12;
constexpr int kBlockCells = 4096;  // cells of a level one block holds: 16 per thread
constexpr int64_t kCoarseMaxCells = 16 * kBlockCells;  // of the first level
constexpr int kCoarseLut = 16;     // byte offset of the diagonal counts' table, after the mbarrier pair
constexpr int kCoarseFixed = 16 + 8 * 8;  // bytes in front of the levels
constexpr int kZeroPad = 8;        // zeros in front of each half: the k neighbour outside the domain

// Offset of row (plane p, j) in a half of z: each plane has a zero row after
// its last, which is also the row before the next plane's first, and a ghost
// plane on either side (zero at the ends of the domain), so that every
// neighbour row is at a fixed distance and reads 0 outside the domain.
__host__ __device__ __forceinline__ int coarse_row(int p, int j, int ny, int hz) {
    return kZeroPad + ((p + 1) * (ny + 1) + j) * hz;
}

struct CoarseLevel {
    Dims D;
    int abs_level;       // level index in the full hierarchy (sets 6 << l)
    int P;               // i-planes per block (D.nx when block 0 holds the level)
    int V;               // cells of one colour per thread item: 4, 2 or 1, dividing nz / 2
    int off_z, off_r;    // shared-memory byte offsets: z (two halves), r (natural order)
    int off_w;           // and: the cells' weights (natural order)
    int hn;              // floats per half of z
    uint32_t div_seg, div_ny, div_nz;  // for coarse_div by nz / 2 / V, ny and nz
    int half;            // a level that the storage types define as FP16 (see coarse_level)
    const uint16_t *cw;  // stencil words of the level, natural order
};

struct CoarseParams {
    int nl, nd;  // levels, and how many of them are split over the cluster (the first nd)
    CoarseLevel lv[kCoarseMaxLevels];
    int off_v;              // residual scratch of the restriction
    const float *r_top;     // residual of the first level (global)
    float *z_top;           // its final correction (global)
    const __half *r_top_h;  // FP16 instead of r_top / z_top when not NULL (mixed precision)
    __half *z_top_h;
    int nu;        // red-black iterations per side at every level (< 0: 6 << level, the reference's)
    int nbottom;   // iterations of each of the two bottom orders (3 in the reference)
    float rscale;  // restriction scale (1 in the reference)
    // bottom64: the bottom level is smoothed in FP64 (z as doubles at byte
    // offset off_zd; r converted exactly from FP32), the result rounded to FP32
    // once for the prolongation.  No reference counterpart: the reference
    // smooths the bottom in FP32 (multigrid/mgpcg.py:319-336).
    int bottom64, off_zd;
    int *status;  // set when a wait on a neighbouring block runs out (NULL: not reported)
};

// n / d for 0 <= n < 2^16 with m = coarse_div_by(d): a multiplication instead of
// the division sequence, whose code would be a good part of a level's set-up.
__host__ __forceinline__ uint32_t coarse_div_by(int d) {
    return d > 1 ? (uint32_t)((uint64_t(1) << 32) / (uint64_t)d) + 1u : 0u;
}
__device__ __forceinline__ int coarse_div(int n, uint32_t m) { return m ? (int)__umulhi((uint32_t)n, m) : n; }

// ---------------------------------------------------------------- cluster primitives
__device__ __forceinline__ unsigned cluster_rank() {
    unsigned r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}

__device__ __forceinline__ void cluster_barrier() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// Address of this block's shared-memory location p in block `rank`.
__device__ __forceinline__ uint32_t remote_addr(const void *p, unsigned rank) {
    uint32_t a;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;"
                 : "=r"(a)
                 : "r"((uint32_t)__cvta_generic_to_shared(p)), "r"(rank));
    return a;
}

__device__ __forceinline__ void remote_store(uint32_t a, float v) {
    asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(a), "f"(v) : "memory");
}

// Store into another block's shared memory that counts its bytes on that
// block's mbarrier.
template <int V>
__device__ __forceinline__ void remote_store_async(uint32_t a, uint32_t mbar, const float *v) {
    if (V == 4)
        asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v4.f32 [%0], {%1, %2, %3, %4}, [%5];" ::"r"(a),
                     "f"(v[0]), "f"(v[1 % V]), "f"(v[2 % V]), "f"(v[3 % V]), "r"(mbar)
                     : "memory");
    else if (V == 2)
        asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v2.f32 [%0], {%1, %2}, [%3];" ::"r"(a),
                     "f"(v[0]), "f"(v[1 % V]), "r"(mbar)
                     : "memory");
    else
        asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.f32 [%0], %1, [%2];" ::"r"(a), "f"(v[0]),
                     "r"(mbar)
                     : "memory");
}

// The exchange of ghost planes between neighbouring blocks.  After a
// half-sweep (and after a prolongation) a block has stored its first and last
// plane into its neighbours' ghosts; it goes on when its own ghosts' bytes
// have arrived.  Two mbarriers take turns: a neighbour may be one exchange
// ahead, never two, since its next one needs this block's planes, and those
// are stored after this block has read the ghosts they are computed from
// (which also keeps the ghosts from being overwritten too early).  A cluster
// barrier instead would have to wait for the remote stores first: measured on
// 16 blocks, 128 16-byte stores to each side, 950 cycles against 520.
struct CoarseSync {
    uint32_t mb, ml, mr;  // shared addresses of the mbarrier pair: this block's, its left and right neighbours'
    uint32_t h;           // exchanges so far
    bool dead;            // a wait ran out: the others do not wait any more
    int *status;
};

constexpr int kCoarseWaitTries = 1 << 14;

__device__ __forceinline__ void exchange_open(const CoarseSync &S, uint32_t bytes) {
    if (threadIdx.x == 0)
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(S.mb + 8u * (S.h & 1u)), "r"(bytes)
                     : "memory");
}

// The first warp polls; a block barrier after it holds the others.
__device__ __forceinline__ void exchange_wait(CoarseSync &S) {
    const uint32_t mb = S.mb + 8u * (S.h & 1u), parity = (S.h >> 1) & 1u;
    S.h++;
    if (threadIdx.x >= 32 || S.dead) return;
    for (int n = 0; n < kCoarseWaitTries; n++) {
        uint32_t ok;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(ok)
            : "r"(mb), "r"(parity)
            : "memory");
        if (ok) return;
    }
    S.dead = true;
    if (S.status) *S.status = FLUB_ERR_TIMEOUT;
}

__device__ __forceinline__ float remote_load(uint32_t a) {
    float v;
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(a) : "memory");
    return v;
}

template <int V>
__device__ __forceinline__ void ld_vec(const float *p, float *o) {
    if (V == 4) {
        const float4 a = *reinterpret_cast<const float4 *>(p);
        o[0] = a.x; o[1 % V] = a.y; o[2 % V] = a.z; o[3 % V] = a.w;
    } else if (V == 2) {
        const float2 a = *reinterpret_cast<const float2 *>(p);
        o[0] = a.x; o[1 % V] = a.y;
    } else {
        o[0] = *p;
    }
}

template <int V>
__device__ __forceinline__ void st_vec(float *p, const float *v) {
    if (V == 4)
        *reinterpret_cast<float4 *>(p) = make_float4(v[0], v[1 % V], v[2 % V], v[3 % V]);
    else if (V == 2)
        *reinterpret_cast<float2 *>(p) = make_float2(v[0], v[1 % V]);
    else
        *p = v[0];
}

// ---------------------------------------------------------------- a thread's cells
// 2 V consecutive cells of row (i, j): V of each colour (colour 0: i + j + k
// even).  Cell m of colour c sits at k = 2 V kg + 2 m + q, q = (c + i + j) & 1;
// of its k neighbours one is the other colour's cell m, the other its cell
// m - 1 (q == 0) or m + 1 (q == 1).
template <int V>
struct CoarseItem {
    float z[2][V], r[2][V];
    float y[2][V];           // -1 / diagonal count; 0 for a cell never updated
    uint32_t d[V];           // the diagonal counts as upper halves of floats: even cell in the low 16 bits, odd high
    uint32_t ml[2][V];       // weight bytes of the i+, i-, j+, j- neighbours (0x40 counts, 0 does not)
    uint32_t mk[V];          // bytes 0, 1: of the k neighbours "cell m" and "the other" of the even cell; 2, 3: odd
    int o, oe[2];            // float offsets in a half: the cells, and (by colour) the one k neighbour outside them
    uint32_t gl, gr;  // the cells' copies in the neighbouring blocks' ghost planes (half 0; 0: none)
    int par, at;      // (i + j) & 1; the item's first cell in natural order (of this block's planes)
    bool on;          // holds a cell that is updated
};

// 2.0f where byte b of m is 0x40, else 0.0f.  kKeep: the compiler may keep the
// 48 weights of an item in registers across the half-sweeps; otherwise they
// are expanded again each time, which it could not know to be cheaper than
// spilling them.
template <bool kKeep>
__device__ __forceinline__ float coarse_weight(uint32_t m, int b) {
    const uint32_t sel = 0x0444u | ((uint32_t)b << 12);
    uint32_t r;
    if (kKeep)
        r = __byte_perm(m, 0u, sel);
    else
        asm volatile("prmt.b32 %0, %1, 0, %2;" : "=r"(r) : "r"(m), "r"(sel));
    return __uint_as_float(r);
}

// The diagonal count of cell m of colour COL.
template <int COL>
__device__ __forceinline__ float coarse_diag(uint32_t d) {
    return __uint_as_float(COL ? d & 0xffff0000u : d << 16);
}

// Pairs of FP32 values for the two-wide FP32 instructions (each rounds both
// halves to nearest, as the one-wide ones do): half the issue slots.
struct F2 {
    unsigned long long v;
};
__device__ __forceinline__ F2 f2(float a, float b) {
    F2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ void f2_get(F2 x, float &a, float &b) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(x.v));
}
__device__ __forceinline__ F2 f2_add(F2 a, F2 b) {
    F2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
__device__ __forceinline__ F2 f2_sub(F2 a, F2 b) {
    F2 r;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
__device__ __forceinline__ F2 f2_mul(F2 a, F2 b) {
    F2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
__device__ __forceinline__ F2 f2_fma(F2 a, F2 b, F2 c) {
    F2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
    return r;
}

// r + L z of the item's V cells of colour COL (lap_at's operation order), two
// cells at a time (V == 1: the second half is idle).
template <int V, int COL, bool kKeep>
__device__ __forceinline__ void coarse_residual(const CoarseItem<V> &t, const float *zs, int hn, const float *r,
                                                int ps, int rs, float *a) {
    const float *zo = zs + (1 - COL) * hn + t.o;
    float ip[V], im[V], jp[V], jm[V], vb[V];
    ld_vec<V>(zo + ps, ip);
    ld_vec<V>(zo - ps, im);
    ld_vec<V>(zo + rs, jp);
    ld_vec<V>(zo - rs, jm);
    const bool q = (COL + t.par) & 1;
    const float e = zs[(1 - COL) * hn + t.oe[COL]];
#pragma unroll
    for (int m = 0; m < V; m++) {
        const float up = m + 1 < V ? t.z[1 - COL][m + 1 < V ? m + 1 : m] : e;
        const float dn = m > 0 ? t.z[1 - COL][m > 0 ? m - 1 : m] : e;
        vb[m] = q ? up : dn;
    }
#pragma unroll
    for (int m = 0; m < V; m += 2) {
        constexpr int h = V > 1 ? 1 : 0;
        const uint32_t l0 = t.ml[COL][m], l1 = t.ml[COL][m + h], k0 = t.mk[m], k1 = t.mk[m + h];
        const F2 xc = f2(t.z[COL][m], t.z[COL][m + h]);
        auto w2 = [&](uint32_t x, uint32_t y, int b) { return f2(coarse_weight<kKeep>(x, b), coarse_weight<kKeep>(y, b)); };
        // each term is exact (weight 2 or 0), so the FMA rounds the sum of the
        // pair once, as adding the two terms would
        F2 s = f2_fma(w2(l0, l1, 0), f2_sub(f2(ip[m], ip[m + h]), xc),
                      f2_mul(w2(l0, l1, 1), f2_sub(f2(im[m], im[m + h]), xc)));
        s = f2_add(s, f2_fma(w2(l0, l1, 2), f2_sub(f2(jp[m], jp[m + h]), xc),
                             f2_mul(w2(l0, l1, 3), f2_sub(f2(jm[m], jm[m + h]), xc))));
        s = f2_add(s, f2_fma(w2(k0, k1, 2 * COL), f2_sub(f2(t.z[1 - COL][m], t.z[1 - COL][m + h]), xc),
                             f2_mul(w2(k0, k1, 2 * COL + 1), f2_sub(f2(vb[m], vb[m + h]), xc))));
        f2_get(f2_fma(f2(0.5f, 0.5f), s, f2(r[m], r[m + h])), a[m], a[m + h]);
    }
}

// A value as FP16 storage holds it.
__device__ __forceinline__ float half_stored(float v) { return __half2float(__float2half_rn(v)); }

// z += (r + L z) / d on the item's cells of colour COL, the quotient by
// Markstein's FMA correction with y = -1/d: q0 = a y, -q = q0 + (a + d q0) y.
// For d = 1..6 that is IEEE a / d for every finite a but ties between two
// denormals at d = 6, so it needs no guard; a branch here cost 100 ns of a 350 ns
// half-sweep.  (tests/test_coarse_div.py checks every finite a >= 0 for d = 3, 5 and 6
// and every 61st for the powers of two; the operations are odd in a.)  A cell
// that is never updated has y = d = 0: its z stays 0.
template <int V, int COL, bool kKeep, bool kHalf>
__device__ __forceinline__ void coarse_half(CoarseItem<V> &t, float *zs, int hn, int ps, int rs) {
    constexpr int h = V > 1 ? 1 : 0;
    float a[V];
    coarse_residual<V, COL, kKeep>(t, zs, hn, t.r[COL], ps, rs, a);
#pragma unroll
    for (int m = 0; m < V; m += 2) {
        const F2 aa = f2(a[m], a[m + h]), y = f2(t.y[COL][m], t.y[COL][m + h]);
        const F2 d = f2(coarse_diag<COL>(t.d[m]), coarse_diag<COL>(t.d[m + h])), q0 = f2_mul(aa, y);
        f2_get(f2_sub(f2(t.z[COL][m], t.z[COL][m + h]), f2_fma(f2_fma(q0, d, aa), y, q0)), t.z[COL][m],
               t.z[COL][m + h]);
    }
    if (kHalf)
#pragma unroll
        for (int m = 0; m < V; m++) t.z[COL][m] = half_stored(t.z[COL][m]);
    st_vec<V>(zs + COL * hn + t.o, t.z[COL]);
}

// The item's cells of colour c (all of them, also of items that are never
// updated: the neighbour counts the plane's bytes) into the neighbours' ghosts.
template <int V>
__device__ __forceinline__ void coarse_push(const CoarseItem<V> &t, const CoarseSync &S, int c, int hn) {
    const uint32_t mb = 8u * (S.h & 1u);
    if (t.gl) remote_store_async<V>(t.gl + c * hn * 4, S.ml + mb, t.z[c]);
    if (t.gr) remote_store_async<V>(t.gr + c * hn * 4, S.mr + mb, t.z[c]);
}

// Masks of a cell from its stencil word for the FP64 bottom: bits 0-5
// neighbour (+i, -i, +j, -j, +k, -k) in the domain and not solid; 6-11 that
// neighbour is air; 12 the cell is fluid.
__device__ __forceinline__ uint32_t bottom_mask(uint32_t w) {
    uint32_t m = (w & 3u) == kCodeFluid ? 1u << 12 : 0u;
#pragma unroll
    for (int q = 0; q < 6; q++) {
        const uint32_t c = sw_code(w, q + 1);
        m |= (c != kCodeSolid ? 1u << q : 0u) | (c == kCodeAir ? 64u << q : 0u);
    }
    return m;
}

// ---------------------------------------------------------------- FP64 bottom
// No reference counterpart (the reference smooths its bottom level in FP32).
// The red-black Gauss-Seidel update of the other levels, z_c + (r + L z) / d
// with L z the sum over non-solid neighbours of (z_n - z_c), z_n = 0 for air,
// is in exact arithmetic (r + sum of the fluid neighbours' z) / d: the z_c
// terms cancel.  The bottom uses that form, which takes 6 FP64 additions and
// the division where the other takes 14 operations (this GPU issues FP64 at a
// small fraction of its FP32 rate, and the bottom runs on one SM): neighbours
// summed in the order i+, i-, j+, j-, k+, k- onto r, each non-fluid one adding
// +0.0, IEEE double rounding at each operation.  The oracle's FP64 bottom
// (oracle_bottom_half64) is the same sequence.

// a / d for d = 1..6, rounded to nearest as __ddiv_rn(a, d), by Markstein's
// FMA correction of a * RN(1/d) (P. Markstein, IBM J. Res. Dev. 34(1), 1990):
// two FMAs and a product instead of an FP64 division, which GB300 issues
// slowly.  tests/test_div6_exhaustive.py checks it bit for bit against IEEE
// division on 2^28 random doubles per d with |a| in [2^-900, 2^900] and on the
// zeros (which return a * RN(1/d), a zero of a's sign); other inputs take
// __ddiv_rn.
// The range is looked at in the bits of a, and d is put together from bits: an FP64
// comparison or conversion takes the FP64 pipe as long as an addition, and the pipe
// is what bounds a bottom full of fluid: with two FP64 comparisons and the
// conversion a half-sweep of 16^3 cells took 1.5 us longer (a V(2,2) cycle of 64^3 on
// 3 levels in mixed precision 182 us, now 157).
__device__ __forceinline__ double ddiv_small_rn(double a, int d) {
    const double y = d == 1 ? 1.0 : d == 2 ? 0.5 : d == 3 ? 1.0 / 3.0 : d == 4 ? 0.25 : d == 5 ? 0.2 : 1.0 / 6.0;
    const double dd = __hiloint2double(d == 1   ? 0x3ff00000
                                       : d == 2 ? 0x40000000
                                       : d == 3 ? 0x40080000
                                       : d == 4 ? 0x40100000
                                       : d == 5 ? 0x40140000
                                                : 0x40180000,
                                       0);
    const uint32_t hi = (uint32_t)__double2hiint(a) & 0x7fffffffu;
    const double q0 = __dmul_rn(a, y);
    if (hi - (123u << 20) < (1800u << 20)) return __fma_rn(__fma_rn(-q0, dd, a), y, q0);  // |a| in [2^-900, 2^900)
    if ((hi | (uint32_t)__double2loint(a)) == 0u) return q0;
    return __ddiv_rn(a, (double)d);
}

constexpr int kBottomPairs = kBlockCells / 2 / kCoarseThreads;

// Each thread owns up to kBottomPairs pairs of k-adjacent cells, one of each colour.
struct BottomCache {
    int idx[kBottomPairs];      // index of the pair's even-k cell, -1 if unused
    uint32_t msk[kBottomPairs];  // low 16 bits: even cell, high 16 bits: odd cell
    float r0[kBottomPairs], r1[kBottomPairs];
    int upd0;  // bit q: in phase 0 the odd-k cell of pair q is updated
};

// Whether the cell of stencil word w is updated.
__device__ __forceinline__ bool bottom_updated(uint32_t w) { return (w & 3u) == kCodeFluid && sw_ns(w) != 0u; }

// r + the fluid neighbours' z of cell c (mask m), in the order above.  All six
// neighbours are loaded (an excluded one reads the cell itself) so the loads
// issue together.
__device__ __forceinline__ double bottom_sum64(const double *z, int c, uint32_t m, double rc, int si, int sj) {
    const double zip = z[(m & 1u) ? c + si : c], zim = z[(m & 2u) ? c - si : c];
    const double zjp = z[(m & 4u) ? c + sj : c], zjm = z[(m & 8u) ? c - sj : c];
    const double zkp = z[(m & 16u) ? c + 1 : c], zkm = z[(m & 32u) ? c - 1 : c];
    // neighbour q is fluid: in the domain and not solid (bit q), not air (bit q + 6)
    const uint32_t fl = (m & 63u) & ~((m >> 6) & 63u);
    double s = rc;
    s = __dadd_rn(s, (fl & 1u) ? zip : 0.0);
    s = __dadd_rn(s, (fl & 2u) ? zim : 0.0);
    s = __dadd_rn(s, (fl & 4u) ? zjp : 0.0);
    s = __dadd_rn(s, (fl & 8u) ? zjm : 0.0);
    s = __dadd_rn(s, (fl & 16u) ? zkp : 0.0);
    return __dadd_rn(s, (fl & 32u) ? zkm : 0.0);
}

// Barrier among the first nthr threads (whole warps): the block's when all
// take part, else named barrier 1.
__device__ __forceinline__ void coarse_sync(int nthr) {
    if (nthr >= kCoarseThreads)
        __syncthreads();
    else
        asm volatile("bar.sync 1, %0;" ::"r"(nthr) : "memory");
}

__device__ __forceinline__ void bottom_half64(double *z, const BottomCache &tc, const Dims D, int phase, int nthr) {
    const int si = D.ny * D.nz, sj = D.nz;
#pragma unroll
    for (int q = 0; q < kBottomPairs; q++) {
        const int c = tc.idx[q];
        if (c < 0) continue;
        const bool odd = (((tc.upd0 >> q) & 1) != 0) == (phase == 0);
        const uint32_t m = odd ? (tc.msk[q] >> 16) : (tc.msk[q] & 0xffffu);
        const int cu = c + (odd ? 1 : 0);
        const double rc = (double)(odd ? tc.r1[q] : tc.r0[q]);
        double zn = 0.0;
        const int d = __popc(m & 63u);
        if ((m & (1u << 12)) && d != 0) zn = ddiv_small_rn(bottom_sum64(z, cu, m, rc, si, sj), d);
        z[cu] = zn;
    }
    coarse_sync(nthr);
}

// Where a thread has several of the FP64 bottom's pairs, those with a cell that is
// updated are listed before the wait on the previous kernel and dealt out from the
// list: the FP64 pipe takes as long for a warp with one such pair as for a full one,
// and a warp's pairs run one after the other.  V(2,2) cycles in mixed precision, dam /
// full of fluid: 96 x 48 x 48 on 3 levels 114 -> 91 / 153 -> 154 us, 64^3 on 3 levels
// 104 -> 85 / 160 -> 161, 128^3 on 4 levels 144 -> 124 / 228 -> 228.
// list: room for an index per pair and their number.
__device__ __forceinline__ void bottom_list(int *list, const uint16_t *cw, int npairs) {
    const uint32_t *words = reinterpret_cast<const uint32_t *>(cw);
    int *listed = list + npairs;
    if (threadIdx.x == 0) *listed = 0;
    __syncthreads();
    const int lane = threadIdx.x & 31;
    uint32_t next = __ldg(words + threadIdx.x);
#pragma unroll 1
    for (int t = threadIdx.x; t - lane < npairs; t += kCoarseThreads) {  // whole warps
        const uint32_t w2 = next;
        next = t + kCoarseThreads < npairs ? __ldg(words + t + kCoarseThreads) : 0u;
        const bool on = bottom_updated(w2 & 0xffffu) || bottom_updated(w2 >> 16);
        const unsigned who = __ballot_sync(0xffffffffu, on);
        int at = 0;
        if (lane == 0) at = atomicAdd(listed, __popc(who));
        at = __shfl_sync(0xffffffffu, at, 0) + __popc(who & ((1u << lane) - 1u));
        if (on) list[at] = t;
    }
}

// The bottom's 2 x nbottom red-black iterations in FP64, starting from z = 0,
// then z rounded to FP32 into the split halves.  Not inlined: its FP64
// registers would otherwise count against the FP32 sweeps.  list: bottom_list's,
// of a bottom with more pairs than threads.
__device__ __noinline__ void coarse_bottom64(double *zd, float *zs, const float *r, int hn, const uint16_t *cw,
                                             const Dims D, int nbottom, const int *list) {
    const int n = (int)D.n(), hz = D.nz >> 1, npairs = n >> 1;
    const bool deal = npairs > kCoarseThreads;
    for (int q = threadIdx.x; q < n; q += blockDim.x) zd[q] = 0.0;
    const uint32_t *words = reinterpret_cast<const uint32_t *>(cw);
    const int total = deal ? list[npairs] : npairs;
    BottomCache tc;
    tc.upd0 = 0;
#pragma unroll
    for (int q = 0; q < kBottomPairs; q++) {
        const int e = threadIdx.x + q * kCoarseThreads;
        tc.idx[q] = -1;
        tc.msk[q] = 0;
        tc.r0[q] = tc.r1[q] = 0.0f;
        if (e < total) {
            const int t = deal ? list[e] : e, c = 2 * t, qq = t / hz, j = qq % D.ny, i = qq / D.ny;
            const uint32_t w2 = __ldg(words + t);
            tc.idx[q] = c;
            tc.msk[q] = bottom_mask(w2 & 0xffffu) | (bottom_mask(w2 >> 16) << 16);
            tc.r0[q] = r[c];
            tc.r1[q] = r[c + 1];
            // phase 0 updates (i+j+k) odd cells: the odd-k cell iff i+j is even
            if (((i + j) & 1) == 0) tc.upd0 |= 1 << q;
        }
    }
    __syncthreads();
    const int w = (total + 31) & ~31, nthr = w < kCoarseThreads ? w : kCoarseThreads;
    if ((int)threadIdx.x < nthr)
        for (int it = 0; it < 2 * nbottom; it++) {
            const int first = it < nbottom ? 0 : 1;
            bottom_half64(zd, tc, D, first, nthr);
            bottom_half64(zd, tc, D, 1 - first, nthr);
        }
    __syncthreads();
    for (int q = threadIdx.x; q < n; q += blockDim.x) {
        const int k = q % D.nz, row = q / D.nz, j = row % D.ny, i = row / D.ny;
        zs[((i + j + k) & 1) * hn + coarse_row(i, j, D.ny, hz) + (k >> 1)] = __double2float_rn(zd[q]);
    }
    __syncthreads();
}

// ---------------------------------------------------------------- one level
enum CoarseMode { kCoarseDown = 0, kCoarseBottom = 1, kCoarseUp = 2 };

// A cell's weights, built once per launch from its stencil word (the levels'
// set-up, twice per launch, then is a load): ml as in CoarseItem; k the bytes
// of the k neighbours "cell m" and "the other" in the low half (k even: the
// pair's own cell above, then the one below), the diagonal count in the high.
struct __align__(8) CoarseWeights {
    uint32_t ml, k;
};

__device__ __forceinline__ CoarseWeights coarse_weights(uint32_t w, int odd_k) {
    const uint32_t ns = (w & 3u) == kCodeFluid ? sw_ns(w) : 0u;
    const uint32_t kp = (ns >> 10) & 1u, km = (ns >> 12) & 1u;
    CoarseWeights c;
    c.ml = ((ns & 4u) << 4) | ((ns & 16u) << 10) | ((ns & 64u) << 16) | ((ns & 256u) << 22);
    c.k = ((odd_k ? km : kp) << 6) | ((odd_k ? kp : km) << 14) | ((uint32_t)__popc(ns) << 16);
    return c;
}

// Level t on the blocks that hold it: down -- pre-smoothing from zero and the
// restriction; bottom -- both bottom orders; up -- the prolongation and
// post-smoothing.  Levels t < P.nd are split over the cluster: every block
// calls this, and neighbours exchange their planes after each half-sweep.  The
// others are block 0's alone.  One function serves both, so that a level's
// code is already in the instruction cache when the next level needs it: the
// first pass through it costs microseconds.
//
// kWide: the threads hold 16 cells each instead of 8, for levels of more than
// 2048 cells a block.  With 256 threads of 255 registers nothing spills in the
// sweeps; 512 threads of 128 hold the same cells and were slower (16^3 full of
// fluid in one block 0.41 against 0.36 us a half-sweep, 8^3 0.19 against 0.12,
// 32^3 on 16 blocks 0.54 against 0.41).
//
// kHalf: a level of a mixed-precision V-cycle that is FP16 at scale 8^-l
// (mixed.cuh).  Its values are held as floats, rounded where the level-by-level
// sweeps store them -- every update, the colour that the first half-sweep after
// the prolongation read unrounded, the coarse residual -- with the same scales
// between levels, so the V-cycle is bit-identical.
template <int V, bool kWide, bool kHalf = false>
__device__ __noinline__ CoarseSync coarse_level(const CoarseParams &P, int t, int mode, unsigned char *smem,
                                                unsigned rank, CoarseSync S) {
    constexpr int Q = (kWide ? 8 : 4) / V;  // items per thread
    constexpr bool kKeep = V == 4 && !kWide;
    const CoarseLevel &L = P.lv[t];
    const Dims D = L.D;
    const bool dist = t < P.nd;
    const int hz = D.nz >> 1, segs = hz / V, ps = (D.ny + 1) * hz, hn = L.hn;
    const int i0 = dist ? (int)rank * L.P : 0;
    const int np = max(0, min(L.P, D.nx - i0));
    const int items = np * D.ny * segs;
    float *zs = reinterpret_cast<float *>(smem + L.off_z);
    const float *R = reinterpret_cast<const float *>(smem + L.off_r);
    const CoarseWeights *W = reinterpret_cast<const CoarseWeights *>(smem + L.off_w);
    const float2 *lut = reinterpret_cast<const float2 *>(smem + kCoarseLut);
    // the 2 V values from natural cell c on, by colour (par: (i + j) & 1)
    auto by_colour = [&](const float *src, int par, float o[2][V]) {
        float n[2 * V];
        ld_vec<V>(src, n);
        ld_vec<V>(src + V, n + V);
#pragma unroll
        for (int m = 0; m < V; m++) {
            o[0][m] = par ? n[2 * m + 1] : n[2 * m];
            o[1][m] = par ? n[2 * m] : n[2 * m + 1];
        }
    };
    CoarseItem<V> it[Q];
#pragma unroll
    for (int s = 0; s < Q; s++) {
        CoarseItem<V> &x = it[s];
        const int e = threadIdx.x + s * kCoarseThreads;
        x.o = -1;
        x.on = false;
        x.gl = x.gr = 0u;
        if (e >= items) continue;
        const int row = coarse_div(e, L.div_seg), kg = e - row * segs;
        const int il = coarse_div(row, L.div_ny), j = row - il * D.ny, i = i0 + il;
        x.o = coarse_row(il, j, D.ny, hz) + V * kg;
        x.at = row * D.nz + 2 * V * kg;
        x.par = (i + j) & 1;
        // the k neighbour outside the item: below it for the colour that starts at its first cell
        const int lo = kg > 0 ? x.o - 1 : 0, hi = kg + 1 < segs ? x.o + V : 0;
        x.oe[0] = x.par ? hi : lo;
        x.oe[1] = x.par ? lo : hi;
        if (dist) {
            // plane 0 is also the left block's ghost plane P + 1, plane np - 1 the right block's ghost plane 0
            if (il == 0 && i > 0) x.gl = remote_addr(zs + x.o + L.P * ps, rank - 1);
            if (il == np - 1 && i + 1 < D.nx) x.gr = remote_addr(zs + x.o - L.P * ps, rank + 1);
        }
        by_colour(R + x.at, x.par, x.r);
#pragma unroll
        for (int m = 0; m < V; m++) x.mk[m] = x.d[m] = 0u;
#pragma unroll
        for (int c = 0; c < 2; c++) {
            ld_vec<V>(zs + c * hn + x.o, x.z[c]);
            const CoarseWeights *wc = W + x.at + ((c + x.par) & 1);
#pragma unroll
            for (int m = 0; m < V; m++) {
                const CoarseWeights w = wc[2 * m];
                const float2 yd = lut[w.k >> 16];
                x.ml[c][m] = w.ml;
                x.mk[m] |= (w.k & 0xffffu) << (16 * c);
                x.d[m] |= (__float_as_uint(yd.y) >> 16) << (16 * c);
                x.y[c][m] = yd.x;
                if (w.k < 0x10000u) x.r[c][m] = 0.0f;
                x.on |= w.k >= 0x10000u;
            }
        }
    }
    const int nw = (items + 31) & ~31, nthr = nw >= kCoarseThreads ? kCoarseThreads : nw;
    // bytes of one colour of the ghost planes that have a neighbour
    const uint32_t ghost = (uint32_t)(D.ny * hz) * 4u * ((i0 > 0 ? 1 : 0) + (i0 + np < D.nx ? 1 : 0));
    const bool work = (int)threadIdx.x < nthr;  // whole warps
    if (mode == kCoarseUp) {
        // z += z_{t+1}[I/2] on the cells that are updated (mgpcg.py:113-116; the
        // others stay 0).  The parents of cell m of either colour are the same
        // coarse cell: (i / 2, j / 2, V kg + m).
        const CoarseLevel &C = P.lv[t + 1];
        const float *zc = reinterpret_cast<const float *>(smem + C.off_z);
        const int chz = C.D.nz >> 1;
        int chn = C.hn;  // floats per half of zc, whose first plane is this block's
        if (dist && t + 1 == P.nd) {
            // the coarse level is in block 0: a copy of this block's planes first,
            // whole rows at a time (every block reads from the one)
            const int first = coarse_row(i0 >> 1, 0, C.D.ny, chz);
            const int len = ((np >> 1) * (C.D.ny + 1)) * chz;
            float *v = reinterpret_cast<float *>(smem + P.off_v);
            for (int q = threadIdx.x; q < 2 * len; q += kCoarseThreads) {
                const int h = q >= len ? 1 : 0, x = q - h * len;
                v[q] = remote_load(remote_addr(zc + h * C.hn + first + x, 0));
            }
            __syncthreads();
            zc = v - coarse_row(0, 0, C.D.ny, chz);
            chn = len;
        }
#pragma unroll
        for (int s = 0; s < Q; s++) {
            CoarseItem<V> &x = it[s];
            if (x.o < 0) continue;
            const int e = threadIdx.x + s * kCoarseThreads;
            const int row = coarse_div(e, L.div_seg), kg = e - row * segs;
            const int il = coarse_div(row, L.div_ny), j = row - il * D.ny, I = (i0 + il) >> 1, J = j >> 1;
            const float *pc = zc + coarse_row(il >> 1, J, C.D.ny, chz);
            float add[V];
#pragma unroll
            for (int m = 0; m < V; m++) {
                const int K = V * kg + m;
                add[m] = pc[((I + J + K) & 1) * chn + (K >> 1)];
                if (kHalf) add[m] = __fmul_rn(half_stored(add[m]), 8.0f);
            }
#pragma unroll
            for (int c = 0; c < 2; c++) {
#pragma unroll
                for (int m = 0; m < V; m++)
                    if (x.y[c][m] != 0.0f) x.z[c][m] = __fadd_rn(x.z[c][m], add[m]);
                st_vec<V>(zs + c * hn + x.o, x.z[c]);
                coarse_push<V>(x, S, c, hn);
            }
        }
        if (dist && np > 0) {
            exchange_open(S, 2u * ghost);
            exchange_wait(S);
        }
        __syncthreads();
    }
    // phase 0 updates the odd colour, phase 1 the even one (mgpcg.py:72-86)
    auto half = [&](auto col) {
        constexpr int COL = decltype(col)::value;
#pragma unroll
        for (int s = 0; s < Q; s++)
            if (it[s].on) coarse_half<V, COL, kKeep, kHalf>(it[s], zs, hn, ps, hz);
        if (dist) {
            exchange_open(S, ghost);
#pragma unroll
            for (int s = 0; s < Q; s++) coarse_push<V>(it[s], S, COL, hn);
            exchange_wait(S);
        }
        coarse_sync(nthr);
    };
    const int iters = mode == kCoarseBottom ? 2 * P.nbottom : (P.nu < 0 ? 6 << L.abs_level : P.nu);
    const uint32_t h_end = S.h + 2u * (uint32_t)iters;  // also on the threads without items
    if (work) {
        // odd then even; post-smoothing, and the bottom's second part, skip the
        // first odd half-sweep and append one
        for (int part = 0; part < (mode == kCoarseBottom ? 2 : 1); part++) {
            const bool even_first = mode == kCoarseUp || part == 1;
            bool skip = even_first;
            for (int n = mode == kCoarseBottom ? P.nbottom : iters; n > 0; n--) {
                if (!skip) half(std::integral_constant<int, 1>{});
                half(std::integral_constant<int, 0>{});
                if (kHalf && skip && mode == kCoarseUp)
#pragma unroll
                    for (int s = 0; s < Q; s++)
#pragma unroll
                        for (int m = 0; m < V; m++) it[s].z[1][m] = half_stored(it[s].z[1][m]);
                skip = false;
            }
            if (even_first) half(std::integral_constant<int, 1>{});
        }
    }
    if (dist) S.h = h_end;
    __syncthreads();
    if (mode != kCoarseDown) return S;
    // residual r + L z (r alone off the fluid), then each coarse fluid cell sums
    // its 8 children in (i, j, k) order and scales (mgpcg.py:94-101 as a gather)
    float *v = reinterpret_cast<float *>(smem + P.off_v);
#pragma unroll
    for (int s = 0; s < Q; s++) {
        const CoarseItem<V> &x = it[s];
        if (x.o < 0) continue;
        float res[2][V], a[2][V], n[2 * V];
        by_colour(R + x.at, x.par, res);
        coarse_residual<V, 0, false>(x, zs, hn, res[0], ps, hz, a[0]);
        coarse_residual<V, 1, false>(x, zs, hn, res[1], ps, hz, a[1]);
#pragma unroll
        for (int m = 0; m < V; m++) {
            // r itself where no neighbour counts: r + 0 z would turn an infinity there into NaN
            const float v0 = x.y[0][m] != 0.0f ? a[0][m] : res[0][m], v1 = x.y[1][m] != 0.0f ? a[1][m] : res[1][m];
            n[2 * m] = x.par ? v1 : v0;
            n[2 * m + 1] = x.par ? v0 : v1;
        }
        st_vec<V>(v + x.at, n);
        st_vec<V>(v + x.at + V, n + V);
    }
    __syncthreads();
    {
        const CoarseLevel &C = P.lv[t + 1];
        const bool remote = dist && t + 1 == P.nd;
        float *Rc = reinterpret_cast<float *>(smem + C.off_r);
        const int cyz = C.D.ny * C.D.nz, nc = (np >> 1) * cyz, sj = D.nz, si = D.ny * D.nz;
        for (int q = threadIdx.x; q < nc; q += kCoarseThreads) {
            const int cr = coarse_div(q, C.div_nz), K = q - cr * C.D.nz, Il = coarse_div(cr, C.div_ny), J = cr - Il * C.D.ny;
            const int g = q + (i0 >> 1) * cyz;  // global coarse cell
            float s = 0.0f;
            if ((__ldg(C.cw + g) & 3u) == kCodeFluid) {
                const float *vc = v + ((2 * Il) * D.ny + 2 * J) * D.nz + 2 * K;
                s = vc[0];
                s = __fadd_rn(s, vc[1]);
                s = __fadd_rn(s, vc[sj]);
                s = __fadd_rn(s, vc[sj + 1]);
                s = __fadd_rn(s, vc[si]);
                s = __fadd_rn(s, vc[si + 1]);
                s = __fadd_rn(s, vc[si + sj]);
                s = __fadd_rn(s, vc[si + sj + 1]);
                s = kHalf ? half_stored(__fmul_rn(s, 0.125f * P.rscale)) : __fmul_rn(s, P.rscale);
            }
            if (remote)
                remote_store(remote_addr(Rc + g, 0), s);
            else
                Rc[q] = s;
        }
        if (remote)
            cluster_barrier();
        else
            __syncthreads();
    }
    return S;
}

template <int kV, bool kMixed>
__device__ __forceinline__ CoarseSync coarse_dispatch(const CoarseParams &P, int t, int mode, unsigned char *smem,
                                                      unsigned rank, CoarseSync S) {
    const int V = kV ? kV : P.lv[t].V;
    if (kMixed && P.lv[t].half) return coarse_level<4, true, true>(P, t, mode, smem, rank, S);  // rows of 8 cells
    if (V == 4) {
        if (P.lv[t].P * P.lv[t].D.ny * P.lv[t].D.nz > 8 * kCoarseThreads)
            return coarse_level<kV ? kV : 4, true>(P, t, mode, smem, rank, S);
        return coarse_level<kV ? kV : 4, false>(P, t, mode, smem, rank, S);
    }
    if (V == 2) return coarse_level<kV ? kV : 2, true>(P, t, mode, smem, rank, S);
    return coarse_level<kV ? kV : 1, true>(P, t, mode, smem, rank, S);
}

// Grid: one cluster (P.nd > 0), or one block.  kV = 4: every level has V = 4 (nz a
// multiple of 8 down to the bottom); the general kernel also holds the code
// for shorter items, which costs it registers.  kMixed: there are levels of kind half.
template <int kV, bool kMixed>
__global__ void __launch_bounds__(kCoarseThreads, 1) k_coarse_vcycle(const __grid_constant__ CoarseParams P,
                                                                     unsigned long long *kc) {
    extern __shared__ __align__(16) unsigned char coarse_smem[];
    unsigned char *smem = coarse_smem;
    pdl_open();
    const unsigned rank = P.nd > 0 ? cluster_rank() : 0u;
    uint64_t *mbar = reinterpret_cast<uint64_t *>(smem);  // the mbarrier pair: the first 16 bytes
    CoarseSync S = {};
    S.mb = (uint32_t)__cvta_generic_to_shared(mbar);
    S.status = P.status;
    if (P.nd > 0) {
        if (threadIdx.x == 0) {
            asm volatile("mbarrier.init.shared.b64 [%0], 1;" ::"r"(S.mb) : "memory");
            asm volatile("mbarrier.init.shared.b64 [%0], 1;" ::"r"(S.mb + 8u) : "memory");
            asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        }
        if (rank > 0) S.ml = remote_addr(mbar, rank - 1);
        if (rank + 1 < gridDim.x) S.mr = remote_addr(mbar, rank + 1);
    }
    // z = 0 everywhere, ghost planes and pads included
    for (int t = 0; t < P.nl; t++) {
        if (t >= P.nd && rank != 0) break;
        float4 *z = reinterpret_cast<float4 *>(smem + P.lv[t].off_z);
        for (int q = threadIdx.x; q < P.lv[t].hn / 2; q += kCoarseThreads) z[q] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
    // what no earlier kernel of the solve writes: -1/d and d, and the weights
    if (threadIdx.x < 8) {
        const float d = (float)threadIdx.x;
        reinterpret_cast<float2 *>(smem + kCoarseLut)[threadIdx.x] =
            make_float2(threadIdx.x ? __fdiv_rn(-1.0f, d) : 0.0f, d);
    }
    for (int t = 0; t < P.nl; t++) {
        if (t >= P.nd && rank != 0) break;
        const CoarseLevel &L = P.lv[t];
        if (P.bottom64 && t + 1 == P.nl) {
            // no weights: their place takes the list of the bottom's pairs (block 0 holds it)
            const int npairs = (int)(L.D.n() >> 1);
            if (npairs > kCoarseThreads) bottom_list(reinterpret_cast<int *>(smem + L.off_w), L.cw, npairs);
            break;
        }
        const int first = t < P.nd ? (int)rank * L.P : 0, yz = L.D.ny * L.D.nz;
        const int pairs = (max(0, min(L.P, L.D.nx - first)) * yz) >> 1;
        const uint32_t *w2 = reinterpret_cast<const uint32_t *>(L.cw) + ((first * yz) >> 1);
        CoarseWeights *W = reinterpret_cast<CoarseWeights *>(smem + L.off_w);
        // a block has at most 8 pairs a thread: all loads first
        constexpr int U = kBlockCells / 2 / kCoarseThreads;
        uint32_t w[U];
#pragma unroll
        for (int u = 0; u < U; u++) {
            const int q = threadIdx.x + u * kCoarseThreads;
            w[u] = q < pairs ? __ldg(w2 + q) : 0u;
        }
#pragma unroll
        for (int u = 0; u < U; u++) {
            const int q = threadIdx.x + u * kCoarseThreads;
            if (q >= pairs) break;
            const CoarseWeights a = coarse_weights(w[u] & 0xffffu, 0), b = coarse_weights(w[u] >> 16, 1);
            *reinterpret_cast<uint4 *>(W + 2 * q) = make_uint4(a.ml, a.k, b.ml, b.k);
        }
    }
    pdl_wait(kc);
    const CoarseLevel &T = P.lv[0];
    const int i0 = P.nd > 0 ? (int)rank * T.P : 0, yz = T.D.ny * T.D.nz;
    const int own = max(0, min(T.P, T.D.nx - i0)) * yz, base = i0 * yz;
    {
        float *R = reinterpret_cast<float *>(smem + T.off_r);
        constexpr int U = 8;
        for (int q0 = threadIdx.x; q0 < own; q0 += U * kCoarseThreads) {
            float v[U];
#pragma unroll
            for (int u = 0; u < U; u++) {
                const int q = q0 + u * kCoarseThreads;
                v[u] = q >= own ? 0.0f : (P.r_top_h ? __half2float(P.r_top_h[base + q]) : P.r_top[base + q]);
            }
#pragma unroll
            for (int u = 0; u < U; u++)
                if (q0 + u * kCoarseThreads < own) R[q0 + u * kCoarseThreads] = v[u];
        }
    }
    if (P.nd > 0)
        cluster_barrier();  // the ghosts are zeroed before a neighbour stores into them
    else
        __syncthreads();
    // levels 0 .. b - 1 down, the bottom b, then up; one call site, so that the
    // level code is held once and inlined
    const int b = P.nl - 1;
    for (int n = 0; n <= 2 * b; n++) {
        const int t = n <= b ? n : 2 * b - n;
        const int mode = n < b ? kCoarseDown : (n == b ? kCoarseBottom : kCoarseUp);
        if (t < P.nd) {
            // block 0 has finished the levels below
            if (mode == kCoarseUp && t == P.nd - 1 && P.nd < P.nl) cluster_barrier();
            S = coarse_dispatch<kV, kMixed>(P, t, mode, smem, rank, S);
        } else if (rank == 0) {
            if (mode == kCoarseBottom && P.bottom64)
                coarse_bottom64(reinterpret_cast<double *>(smem + P.off_zd),
                                reinterpret_cast<float *>(smem + P.lv[t].off_z),
                                reinterpret_cast<const float *>(smem + P.lv[t].off_r), P.lv[t].hn, P.lv[t].cw,
                                P.lv[t].D, P.nbottom, reinterpret_cast<const int *>(smem + P.lv[t].off_w));
            else
                S = coarse_dispatch<kV, kMixed>(P, t, mode, smem, 0u, S);
        }
    }
    // the first level's correction in natural order
    const float *zs = reinterpret_cast<const float *>(smem + T.off_z);
    const int hz = T.D.nz >> 1;
    for (int q = threadIdx.x; q < own; q += kCoarseThreads) {
        const int row = coarse_div(q, T.div_nz), k = q - row * T.D.nz, il = coarse_div(row, T.div_ny), j = row - il * T.D.ny;
        const float z = zs[((i0 + il + j + k) & 1) * T.hn + coarse_row(il, j, T.D.ny, hz) + (k >> 1)];
        if (P.z_top_h)
            P.z_top_h[base + q] = __float2half_rn(z);
        else
            P.z_top[base + q] = z;
    }
    if (P.nd > 0) cluster_barrier();  // no block leaves while another may still store into it
}

// Stencil words of every cell of a level, natural order, for any nz (the same
// words as words8_from_codes).
__global__ void __launch_bounds__(256) k_cell_words(const uint8_t *code, uint16_t *cw, Dims D) {
    setup_open();
    const int n = (int)D.n(), sj = D.nz, si = D.ny * D.nz;
    for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < n; c += gridDim.x * blockDim.x) {
        const int k = c % D.nz, j = (c / D.nz) % D.ny, i = c / si;
        auto nb = [&](bool in, int off, int q) -> uint32_t {
            return in ? (uint32_t)code[c + off] << (2 * q) : 0u;
        };
        cw[c] = (uint16_t)((uint32_t)code[c] | nb(i + 1 < D.nx, si, 1) | nb(i > 0, -si, 2) | nb(j + 1 < D.ny, sj, 3) |
                           nb(j > 0, -sj, 4) | nb(k + 1 < D.nz, 1, 5) | nb(k > 0, -1, 6));
    }
}

}  // namespace flub
