// Red-black smoothing of the large levels on colour-split storage.
//
// In natural order (k fastest) the cells of one colour alternate along k, so
// a half-sweep that updates one colour still moves whole rows: half of every
// neighbour row it loads and half of the row it stores belong to the colour it
// does not update.  Inside the V-cycle the vectors of these levels are therefore
// kept split by colour: a buffer of n values holds the even cells ((i + j + k) even)
// in its first half and the odd cells in its second half, each half laid out
// [i][j][k / 2].  Natural cell (i, j, k) is element k >> 1 of row (i, j) in the
// half of parity (i + j + k) & 1, and
//   - its i and j neighbours (other colour) have the SAME index in the other
//     half's rows (i +- 1, j) and (i, j +- 1);
//   - its k neighbours are elements (k >> 1) - 1 + q and (k >> 1) + q of the
//     other half's row (i, j), with q = k & 1;
//   - its parent on the next level is (i >> 1, j >> 1, k >> 1) in natural order.
// An 8-cell group of the active lists (natural k = 8 kg .. 8 kg + 7) is
// elements 4 kg .. 4 kg + 3 of the row in each half.
//
// One lane updates the 4 cells of the active colour in one active group: one
// item word (smooth_block.cuh: the diagonal counts of the 4 cells, and whether
// a solid is next to any), 16-byte loads of their r and z and of the other
// colour's four neighbour rows and own row, one 16-byte store -- all of it data
// the update uses.  The arithmetic is block_update: smooth_cell's operations,
// cell by cell in the reference's order (multigrid/mgpcg.py:72-86), so results
// are bit-identical to the natural-order kernels.
//
// z is 0 on every cell off the fluid, in both buffers, so an air neighbour
// needs no test, and a solid or a wall is the cell itself (its term is 0).  What
// bounds a half-sweep up to 256^3, where the buffers sit in L2, is issue: a
// word per cell, decoded with a branch per cell wherever one of the 4 is not
// interior, took ~400 instructions an item, and a warp of 32 rows nearly always
// has such an item.  With the item word only items next to a solid load their
// stencil words; the prolongation, which adds the correction to air as well, does
// so next to air too.
// A half-sweep of 128^3 (FP32, dam break / full): 1.9 / 3.3 us, in natural order
// 3.0 / 6.7.  Whole projections with these levels in natural order (FLUB_NO_SPLIT=1)
// and as they are: 128^3 sphere in mixed precision 8.8 and 7.1 ms, 256^3 dam break 15.9
// and 12.7, 256 x 64 x 256 3.72 and 3.44, 104 x 72 x 88 2.11 and 1.88.
//
// Modes of one half-sweep (phase 0 updates the odd cells, phase 1 the even):
//   kFirst    first pre-smoothing half-sweep (phase 0, from zero): reads the
//             natural residual rn, writes both halves of the split residual
//             rs (0 on cells that are never updated) and z = r / d on the odd
//             cells; the even cells are not touched (the next half-sweep runs
//             kOwnZero).
//   kOwnZero  second half-sweep of the first iteration: the updated cells'
//             own z is 0 and is not read.
//   kInPlace  z updated in place.
//   kProlong  first post-smoothing half-sweep (phase 1): reads zin + zc[I/2]
//             (multigrid/mgpcg.py:113-116) and writes both halves of zout:
//             the updated even cells and the odd cells of the group with the
//             prolongation added (0 off the fluid).
//   kLast     last post-smoothing half-sweep (phase 0): writes the group's 8
//             cells to the natural-order output zn, the even cells
//             passed through (0 off the fluid).
// Only the groups of the active list are visited; the other groups of the
// split buffers are never read for a value that enters a fluid cell's update.
#pragma once

#include "smooth8.cuh"
#include "smooth_block.cuh"

namespace flub {

enum SplitMode { kFirst = 0, kOwnZero = 1, kInPlace = 2, kProlong = 3, kLast = 4 };

struct SplitArgs {
    Dims D;
    const int *act, *act_n;     // active 8-cell groups of the level
    const uint16_t *sws;        // stencil words, colour-split
    const uint32_t *items;      // item words (smooth_block.cuh) of every group: colour 0, then colour 1
    const void *rn;             // kFirst: natural residual (TRN)
    void *rs;                   // colour-split residual (TR): written by kFirst, read by the others
    const void *zin;            // kProlong: colour-split input z (TZI)
    void *z;                    // colour-split z (TZ), in place / output
    const void *zc;             // kProlong: next level's correction, natural order (TC)
    float zc_scale;
    void *zn;                   // kLast: natural-order output (TC)
    // kLast: z.r of the CG step folded in (mgpcg.py:401, 451): dot 1 --
    // zr_old = z.r and p = z (the solve's prologue), dot 2 -- beta = z.r /
    // zr_old, zr_old = z.r (each iteration), dot 3 -- the flexible beta =
    // (z.r - z.r_old) / zr_old of the mixed-precision solve; 0 -- none.  rdot
    // and rold are natural-order FP32 vectors; zscaled: the CG's z is
    // st->zscale times the V-cycle's output (mixed precision).  The per-group
    // sums are k8_dot_zr's / k8_dot_zr_flex's.
    int dot, zscaled;
    const float *rdot, *rold;
    float *pinit;
    MgState *st;
    double *partials;
};

__device__ __forceinline__ uint32_t word4_at(uint2 w, int m) {
    const uint32_t v = m < 2 ? w.x : w.y;
    return (m & 1) ? (v >> 16) : (v & 0xffffu);
}

// Register bound of 4 blocks of 256 threads per SM: 55 to 64 registers.  No array
// here is indexed by q, the parity of the updated cells' k: as an index it made
// the compiler select among all elements for each (the last half-sweep took 600
// instructions an item, now 310; 256^3-sized levels 17 -> 12 us, 512 x 256 x 256
// with the dot product 123 -> 101 us and 54 -> 51 us in place, of DRAM traffic worth
// 87 and 41).  More blocks, fewer, or two groups a lane with their loads issued
// together measured no better.
template <int kMode, typename TRN, typename TR, typename TZI, typename TZ, typename TC>
__global__ void __launch_bounds__(256, 4)
    k_smooth_split(const SplitArgs A, int phase, unsigned long long *kc) {
    __shared__ float2 lut[8];  // -1/d and d
    pdl_open();
    const Dims D = A.D;
    const int hz = D.nz >> 1;             // split row length
    const int hn = (int)(D.n() >> 1);     // elements per half
    const int sj = hz, si = D.ny * hz;    // split strides of j and i
    const int col = 1 - phase;            // colour of the updated cells: 1 odd, 0 even
    const int uoff = col ? hn : 0, voff = col ? 0 : hn;
    const TR *rs = static_cast<const TR *>(A.rs);
    TZ *z = static_cast<TZ *>(A.z);
    const int total = *A.act_n;
    const int stride = gridDim.x * blockDim.x;
    int t = blockIdx.x * blockDim.x + threadIdx.x;
    int g_next = t < total ? __ldg(A.act + t) : 0;
    // the list and the first words do not depend on the previous kernel
    const uint32_t *items = A.items + (col ? (int)(D.n() >> 3) : 0), *other = A.items + (col ? 0 : (int)(D.n() >> 3));
    uint32_t it_next = t < total ? __ldg(items + g_next) : 0u;
    if (threadIdx.x < 8)
        lut[threadIdx.x] = make_float2(threadIdx.x ? __fdiv_rn(-1.0f, (float)threadIdx.x) : 0.0f, (float)threadIdx.x);
    __syncthreads();
    pdl_wait(kc);
    const unsigned nb = working_blocks(total);
    if (kMode == kLast && A.dot && blockIdx.x >= nb) return;
    double zr = 0.0, zro = 0.0;  // kLast with A.dot: this thread's parts of z.r and z.r_old
    const float zsc = (kMode == kLast && A.dot && A.zscaled) ? A.st->zscale : 1.0f;
    for (; t < total; t += stride) {
        const int g = g_next;
        const int tn = t + stride;
        g_next = tn < total ? __ldg(A.act + tn) : 0;
        int i, j, kg;
        group_ijk(g, D, i, j, kg);
        const int h = (i * D.ny + j) * hz + 4 * kg;  // split index of the group's first element
        const int q = (col + i + j) & 1;             // updated cell m sits at natural k = 8 kg + 2 m + q
        const uint32_t item = it_next;
        it_next = tn < total ? __ldg(items + g_next) : 0u;
        float rr[4];
        if (kMode == kFirst) {
            // natural residual row -> both halves of the split residual
            float rv[8];
            St<TRN>::ld8_any(static_cast<const TRN *>(A.rn) + ((size_t)g << 3), rv);
            const int p = (i + j) & 1;  // natural cell m is even when (p + m) is even
            float re[4], ro[4];
#pragma unroll
            for (int m = 0; m < 8; m++) {
                if (((p + m) & 1) == 0) re[m >> 1] = rv[m];
                else ro[m >> 1] = rv[m];
            }
            // 0 where the smoothing never updates: the split residual is read
            // for those cells as well
            const uint32_t ov = __ldg(other + g);
#pragma unroll
            for (int m = 0; m < 4; m++) {
                const uint32_t se = col ? ov : item, so = col ? item : ov;
                if (!((se >> (4 * m)) & 7u)) re[m] = 0.0f;
                if (!((so >> (4 * m)) & 7u)) ro[m] = 0.0f;
            }
            TR *rsw = static_cast<TR *>(A.rs);
            St<TR>::st4(rsw + h, re);
            St<TR>::st4(rsw + hn + h, ro);
            float out[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
            for (int m = 0; m < 4; m++) rr[m] = col ? ro[m] : re[m];
            const float zero[4] = {0.f, 0.f, 0.f, 0.f};
            block_update<4>(item, out, zero, zero, zero, zero, zero, zero, rr, lut);
            St<TZ>::st4(z + uoff + h, out);
            continue;
        }
        St<TR>::ld4_in(rs + uoff + h, rr);
        const bool hip = i + 1 < D.nx, him = i > 0, hjp = j + 1 < D.ny, hjm = j > 0;
        const bool hkm = kg > 0, hkp = 4 * kg + 4 < hz;
        // operands: own z, the other colour's row (i, j) with the element before
        // (q = 0) or after it (q = 1), and its four neighbour rows
        float xc[4] = {0.f, 0.f, 0.f, 0.f}, edge;
        float zip[4] = {0.f, 0.f, 0.f, 0.f}, zim[4] = {0.f, 0.f, 0.f, 0.f};
        float zjp[4] = {0.f, 0.f, 0.f, 0.f}, zjm[4] = {0.f, 0.f, 0.f, 0.f};
        float vc[4];
        if (kMode == kProlong) {
            const TZI *zi = static_cast<const TZI *>(A.zin);
            const TC *zc = static_cast<const TC *>(A.zc);
            const float s = A.zc_scale;
            const int cy = D.ny >> 1;  // the coarse level is nx/2 x ny/2 x hz, natural order
            // coarse row (I, J) at K = 4 kg .. 4 kg + 3: the parents of elements h .. h + 3
            auto crow = [&](int ii, int jj, float o[4]) {
                St<TC>::ld4_in(zc + ((size_t)((ii >> 1) * cy + (jj >> 1)) * hz + 4 * kg), o);
            };
            float cc[4], cn[4] = {0.f, 0.f, 0.f, 0.f};
            crow(i, j, cc);
            St<TZI>::ld4(zi + uoff + h, xc);
            St<TZI>::ld4(zi + voff + h, vc);
#pragma unroll
            for (int m = 0; m < 4; m++) {
                xc[m] = __fadd_rn(xc[m], __fmul_rn(cc[m], s));
                vc[m] = __fadd_rn(vc[m], __fmul_rn(cc[m], s));
            }
            auto row = [&](bool in, int off, int ii, int jj, float o[4]) {
                if (in) {
                    St<TZI>::ld4(zi + voff + h + off, o);
                    crow(ii, jj, cn);
                }
#pragma unroll
                for (int m = 0; m < 4; m++) o[m] = in ? __fadd_rn(o[m], __fmul_rn(cn[m], s)) : xc[m];
            };
            row(hip, si, i + 1, j, zip);
            row(him, -si, i - 1, j, zim);
            row(hjp, sj, i, j + 1, zjp);
            row(hjm, -sj, i, j - 1, zjm);
            const int eo = q ? 4 : -1;
            edge = q ? xc[3] : xc[0];
            if (q ? hkp : hkm)
                edge = __fadd_rn(
                    St<TZI>::ld(zi + voff + h + eo),
                    __fmul_rn(St<TC>::ld_in(zc + (size_t)((i >> 1) * cy + (j >> 1)) * hz + 4 * kg + eo), s));
        } else {
            // a neighbour row outside the domain is replaced by the cells
            // themselves: their terms are then 0
            if (kMode != kOwnZero) St<TZ>::ld4(z + uoff + h, xc);
            St<TZ>::ld4(z + voff + h, vc);
            if (kMode != kOwnZero) {
                St<TZ>::ld4(hip ? z + voff + h + si : z + uoff + h, zip);
                St<TZ>::ld4(him ? z + voff + h - si : z + uoff + h, zim);
                St<TZ>::ld4(hjp ? z + voff + h + sj : z + uoff + h, zjp);
                St<TZ>::ld4(hjm ? z + voff + h - sj : z + uoff + h, zjm);
            } else {  // own z is 0, whatever the buffer holds
                if (hip) St<TZ>::ld4(z + voff + h + si, zip);
                if (him) St<TZ>::ld4(z + voff + h - si, zim);
                if (hjp) St<TZ>::ld4(z + voff + h + sj, zjp);
                if (hjm) St<TZ>::ld4(z + voff + h - sj, zjm);
            }
            edge = (q ? hkp : hkm) ? St<TZ>::ld(z + voff + h + (q ? 4 : -1)) : (q ? xc[3] : xc[0]);
        }
        float out[4], vo[4], va[4], vb[4];  // va: the k neighbours inside the group's row, vb the others
#pragma unroll
        for (int m = 0; m < 4; m++) {
            va[m] = vc[m];
            vb[m] = q ? (m < 3 ? vc[m < 3 ? m + 1 : m] : edge) : (m > 0 ? vc[m > 0 ? m - 1 : m] : edge);
            out[m] = xc[m];
            vo[m] = vc[m];
        }
        if (item & (kMode == kProlong ? kItemSolid | kItemAir : kItemSolid)) {
            // solids next to it: the neighbours that do not count become the cell
            // itself; air is 0 in z, but not after the prolongation's addition
            const uint2 ws = __ldg(reinterpret_cast<const uint2 *>(A.sws + uoff + h));
#pragma unroll
            for (int m = 0; m < 4; m++) {
                const uint32_t cw = word4_at(ws, m), ns = sw_ns(cw);
                auto fix = [&](float &v, uint32_t bit) {
                    if (!(ns & bit)) v = xc[m];
                    else if (kMode == kProlong && (cw & bit)) v = 0.0f;
                };
                fix(zip[m], 4u);
                fix(zim[m], 16u);
                fix(zjp[m], 64u);
                fix(zjm[m], 256u);
                fix(va[m], q ? 4096u : 1024u);
                fix(vb[m], q ? 1024u : 4096u);
            }
        }
        block_update<4>(item, out, zip, zim, zjp, zjm, va, vb, rr, lut);
        if (kMode == kProlong) {
            // 0 where a cell is never updated: the addition left the correction there
            const uint32_t ov = __ldg(other + g);
#pragma unroll
            for (int m = 0; m < 4; m++) {
                if (!((item >> (4 * m)) & 7u)) out[m] = 0.0f;
                if (!((ov >> (4 * m)) & 7u)) vo[m] = 0.0f;
            }
        }
        if (kMode == kLast) {
            // natural row of the group: updated cell m at offset 2 m + q, the
            // other colour's element m at 2 m + 1 - q
            float o8[8];
#pragma unroll
            for (int m = 0; m < 4; m++) {
                o8[2 * m] = q ? vo[m] : out[m];
                o8[2 * m + 1] = q ? out[m] : vo[m];
            }
            St<TC>::st8_any(static_cast<TC *>(A.zn) + ((size_t)g << 3), o8);
            if (A.dot) {
                float zv[8], rv[8];
                St<float>::ld8_wide(A.rdot + ((size_t)g << 3), rv);
#pragma unroll
                for (int m = 0; m < 8; m++) zv[m] = A.zscaled ? __fmul_rn(o8[m], zsc) : o8[m];
                zr += dot8_ff(zv, rv);
                if (A.dot == 3) {
                    float ov[8];
                    St<float>::ld8_wide(A.rold + ((size_t)g << 3), ov);
                    zro += dot8_ff(zv, ov);
                }
                if (A.dot == 1) St<float>::st8_wide(A.pinit + ((size_t)g << 3), zv);
            }
        } else {
            St<TZ>::st4(z + uoff + h, out);
            if (kMode == kProlong) St<TZ>::st4(z + voff + h, vo);
        }
    }
    if (kMode == kLast && A.dot) {
        // the grid's z.r in FP64 (deterministic two-level reduction) and the
        // CG scalars, as k8_dot_zr sets them
            if (A.dot == 3) {
            const double bo = block_sum_red(zro);
            __syncthreads();
            if (threadIdx.x == 0) A.partials[kMaxRedBlocks + blockIdx.x] = bo;
        }
        double tot;
        if (finish_partials(zr, A.partials, &A.st->ticket, &tot, nb)) {
            double t2 = 0.0;
            if (A.dot == 3) {
                __syncthreads();
                for (unsigned q = threadIdx.x; q < nb; q += blockDim.x)
                    t2 += __ldcg(&A.partials[kMaxRedBlocks + q]);
                t2 = block_sum_red(t2);
            }
            if (threadIdx.x == 0) {
                if (A.dot == 1) {
                    A.st->zr_old = tot;
                } else {
                    const double beta = (A.dot == 3 ? tot - t2 : tot) / (A.st->zr_old + A.st->eps);
                    A.st->beta = beta;
                    A.st->zr_old = tot;
                    if (!isfinite(beta)) A.st->status = FLUB_ERR_BREAKDOWN;
                }
            }
        }
    }
}

}  // namespace flub
