// Residual + restriction (multigrid/mgpcg.py:94-101, written as a gather) on
// groups of 8 fine cells: four lanes produce 4 consecutive coarse cells
// (I, J, K0..K0+3) from the four fine rows (2I + ii, 2J + jj), k = 2 K0 .. 2 K0
// + 7, each one 8-cell group read with vector loads.  Per coarse cell the 8
// children are summed in the reference's order (ii, jj, kk), kk fastest, with
// the same FP32 operations as the scalar k_restrict, so results are
// bit-identical.
#pragma once

#include "cg8.cuh"
#include "smooth_block.cuh"
#include "store.cuh"

namespace flub {

// (r + L z) on the 8 cells of fine group g (L z is 0 at non-fluid cells),
// neighbour codes from the stencil words (sw, or the codes when sw is NULL).
// kNC: r and z may be read through the read-only path (see smooth8_pass).
template <bool kNC, typename TR, typename TZ>
__device__ __forceinline__ void residual_row8(const TR *__restrict__ r, const TZ *__restrict__ z,
                                              const uint8_t *__restrict__ code, const uint16_t *__restrict__ sw,
                                              const Dims D, int g, float out[8]) {
    int i, j, kg;
    group_ijk(g, D, i, j, kg);
    const int k0 = kg << 3;
    const int sj = D.nz, si = D.ny * D.nz;
    const int c0 = g << 3;
    float rv[8];
    if (kNC) St<TR>::ld8_in(r + c0, rv); else St<TR>::ld8_cg(r + c0, rv);
    const uint4 wd = load_words8(sw, code, D, i, j, k0, c0);
    if (!words_have_fluid(wd)) {
#pragma unroll
        for (int m = 0; m < 8; m++) out[m] = __fadd_rn(rv[m], 0.0f);
        return;
    }
    const bool hip = i + 1 < D.nx, him = i > 0, hjp = j + 1 < D.ny, hjm = j > 0;
    const bool hkp = k0 + 8 < D.nz, hkm = k0 > 0;
    float xc[8], xip[8], xim[8], xjp[8], xjm[8];
    auto ld8 = [&](const TZ *p, float o[8]) {
        if (kNC) St<TZ>::ld8_in(p, o); else St<TZ>::ld8_cg(p, o);
    };
    auto ld1 = [&](const TZ *p) { return kNC ? St<TZ>::ld_in(p) : St<TZ>::ld_cg(p); };
#pragma unroll
    for (int m = 0; m < 8; m++) xip[m] = xim[m] = xjp[m] = xjm[m] = 0.0f;
    float xkm = 0.0f, xkp = 0.0f;
    ld8(z + c0, xc);
    if (hip) ld8(z + c0 + si, xip);
    if (him) ld8(z + c0 - si, xim);
    if (hjp) ld8(z + c0 + sj, xjp);
    if (hjm) ld8(z + c0 - sj, xjm);
    if (hkm) xkm = ld1(z + c0 - 1);
    if (hkp) xkp = ld1(z + c0 + 8);
#pragma unroll
    for (int m = 0; m < 8; m++) {
        float lz = 0.0f;
        const uint32_t w = word_at(wd, m);
        if (sw_code(w, 0) == kCodeFluid)
            lz = sw_nbsum(w, xc[m], xip[m], xim[m], xjp[m], xjm[m], m < 7 ? xc[m + 1] : xkp, m > 0 ? xc[m - 1] : xkm);
        out[m] = __fadd_rn(rv[m], lz);
    }
}

// The same with z on colour-split storage (smooth_split.cuh) and item words
// (smooth_block.cuh) in place of stencil words; r is in natural order and may be
// a caller's array.  Cells k = 2m ("a") are one colour of the row and k = 2m + 1
// ("b") the other: the neighbours of a in the rows around are elements of the
// half that b is in, and its k neighbours b's elements m - 1 and m.  A neighbour
// outside the domain is the cell itself, air holds 0, and only a group next to
// a solid loads its stencil words, so the sums have no branch per cell.
template <typename TR, typename TZ>
__device__ __forceinline__ void residual_row8_split(const TR *__restrict__ r, const TZ *__restrict__ z,
                                                    const uint16_t *__restrict__ sw,
                                                    const uint32_t *__restrict__ items, const Dims D, int g,
                                                    float out[8]) {
    int i, j, kg;
    group_ijk(g, D, i, j, kg);
    const int hz = D.nz >> 1, hn = (int)(D.n() >> 1), ng = (int)(D.n() >> 3);
    const int sj = hz, si = D.ny * hz;
    const int h = (i * D.ny + j) * hz + 4 * kg;
    const int p = (i + j) & 1;  // the colour of a: 0 even
    const TZ *za = z + (p ? hn : 0) + h, *zb = z + (p ? 0 : hn) + h;
    const uint32_t ia = __ldg(items + (p ? ng : 0) + g), ib = __ldg(items + (p ? 0 : ng) + g);
    float rv[8], a[4], b[4], n[4][4];
    St<TR>::ld8_any(r + ((size_t)g << 3), rv);
    St<TZ>::ld4_in(za, a);
    St<TZ>::ld4_in(zb, b);
    const bool hip = i + 1 < D.nx, him = i > 0, hjp = j + 1 < D.ny, hjm = j > 0;
#pragma unroll
    for (int half = 0; half < 2; half++) {
        // x: the half's cells, y: the other's; its k neighbours are y[m] and y[m - 1] (a) or y[m + 1] (b)
        const TZ *zx = half ? zb : za, *zy = half ? za : zb;
        const float *x = half ? b : a, *y = half ? a : b;
        const uint32_t item = half ? ib : ia;
        St<TZ>::ld4_in(hip ? zy + si : zx, n[0]);
        St<TZ>::ld4_in(him ? zy - si : zx, n[1]);
        St<TZ>::ld4_in(hjp ? zy + sj : zx, n[2]);
        St<TZ>::ld4_in(hjm ? zy - sj : zx, n[3]);
        float u[4], v[4];
#pragma unroll
        for (int m = 0; m < 4; m++) u[m] = y[m];
        if (half) {
            v[0] = y[1]; v[1] = y[2]; v[2] = y[3];
            v[3] = 4 * kg + 4 < hz ? St<TZ>::ld_in(zy + 4) : x[3];
        } else {
            v[0] = kg > 0 ? St<TZ>::ld_in(zy - 1) : x[0];
            v[1] = y[0]; v[2] = y[1]; v[3] = y[2];
        }
        if (item & kItemSolid) {
            const uint4 w = __ldg(reinterpret_cast<const uint4 *>(sw + ((size_t)g << 3)));
#pragma unroll
            for (int m = 0; m < 4; m++) {
                const uint32_t ns = sw_ns(word_at(w, 2 * m + half));
                if (!(ns & 4u)) n[0][m] = x[m];
                if (!(ns & 16u)) n[1][m] = x[m];
                if (!(ns & 64u)) n[2][m] = x[m];
                if (!(ns & 256u)) n[3][m] = x[m];
                if (!(ns & (half ? 4096u : 1024u))) u[m] = x[m];
                if (!(ns & (half ? 1024u : 4096u))) v[m] = x[m];
            }
        }
#pragma unroll
        for (int m = 0; m < 4; m++) {
            float lz = __fadd_rn(0.0f, __fadd_rn(__fsub_rn(n[0][m], x[m]), __fsub_rn(n[1][m], x[m])));
            lz = __fadd_rn(lz, __fadd_rn(__fsub_rn(n[2][m], x[m]), __fsub_rn(n[3][m], x[m])));
            lz = __fadd_rn(lz, __fadd_rn(__fsub_rn(u[m], x[m]), __fsub_rn(v[m], x[m])));
            if (!((item >> (4 * m)) & 7u)) lz = 0.0f;
            out[2 * m + half] = __fadd_rn(rv[2 * m + half], lz);
        }
    }
}

// Coarse level C (fine = 2C).  Work items: the coarse half-groups of 4 cells
// (I, J, 4 K4 .. 4 K4 + 3): with a coarse active list, the 2 halves of every
// listed coarse group (the coarse cells outside the list are not fluid and keep
// r_c = 0, cleared at set_tags and never written otherwise); without one, every
// half-group.  Four lanes share an item, lane 8 q + u of a warp computing the
// residual of fine row (2I + ii, 2J + jj), q = 2 ii + jj, of the warp's item u
// -- a quarter of the registers and four times the lanes of one thread per
// item, to hide memory latency, and eight consecutive lanes on consecutive
// groups of one row, so that a 16-byte load of theirs is one 128-byte line (with
// the four rows on adjacent lanes it is four, and the L1's throughput bound the
// kernel).  The 8 children of each coarse cell are then summed in the
// reference's order (ii, jj, kk), kk fastest: a transpose over the four lanes
// gives lane q every child of coarse cell q.  Figures at k_restrict8_split.
// out_scale: restriction scale (times 1/8 between FP16 levels at 8^-l).
// Grid: one-dimensional, grid-stride by warps (all lanes of a warp run the same
// iterations, so the shuffles see every lane).
// bid / nblk: this block's index and the number of blocks sharing the loop.
// pdl: called at the start of a kernel launched with programmatic dependent
// launch; the item count is read first, then pdl_wait(kc).
// residual(g, v): the residual of the 8 cells of fine group g.
template <typename TRO, typename Residual>
__device__ __forceinline__ void restrict8_pass(TRO *__restrict__ rc, const uint8_t *__restrict__ cc, const Dims C,
                                               float out_scale, const int *__restrict__ act,
                                               const int *__restrict__ act_n, int bid, int nblk, bool pdl,
                                               unsigned long long *kc, Residual residual) {
    const Dims F{2 * C.nx, 2 * C.ny, 2 * C.nz};
    const int nh = (int)(C.n() >> 2);  // coarse half-groups of 4 cells
    const int items = act ? 2 * *act_n : nh;
    const int fz8 = F.nz >> 3;
    const int lane = threadIdx.x & 31, q = lane >> 3;
    const bool q0 = q & 1, q1 = q & 2;
    const int stride = nblk * (blockDim.x >> 2);  // items
    // half-group index of item it, read one round ahead
    auto entry = [&](int it) { return it < items ? (act ? 2 * __ldg(act + (it >> 1)) + (it & 1) : it) : 0; };
    int it = bid * (blockDim.x >> 2) + ((threadIdx.x & ~31) >> 2) + (lane & 7), h_next = entry(it);
    if (pdl) pdl_wait(kc);
    for (; it - (lane & 7) < items; it += stride) {
        const bool valid = it < items;
        const int h = h_next;
        h_next = entry(it + stride);
        const int c0 = h << 2;  // first coarse cell
        const uint32_t codes4 = valid ? __ldg(reinterpret_cast<const uint32_t *>(cc + c0)) : 0u;
        float v[8];
#pragma unroll
        for (int m = 0; m < 8; m++) v[m] = 0.0f;
        // a listed group is worth its rows; without a list, only with a fluid cell among the 4
        if (valid && (act || (codes4 & 0x02020202u) != 0u)) {
            // (I, J, K4) of the half-group: the coarse grid read as 4-cell groups
            int I, J, K4;
            group_ijk(h, Dims{C.nx, C.ny, C.nz << 1}, I, J, K4);  // C.nz / 4 half-groups per row
            residual(((2 * I + (q >> 1)) * F.ny + 2 * J + (q & 1)) * fz8 + K4, v);  // fine group at k = 8 K4
        }
        // lane q holds its row's pairs (v[2m], v[2m + 1]) for every coarse cell m
        // and is to hold the pairs of m = q from the rows 0..3: bit 0, then bit 1
        float w[4][2], t[4][2];  // w[2 k + r]: row (q & 2) + r's pair for m = 2 k + (q & 1)
#pragma unroll
        for (int k = 0; k < 2; k++)
#pragma unroll
            for (int e = 0; e < 2; e++) {
                const float lo = v[4 * k + e], hi = v[4 * k + 2 + e];
                const float keep = q0 ? hi : lo, got = __shfl_xor_sync(0xffffffffu, q0 ? lo : hi, 8);
                w[2 * k][e] = q0 ? got : keep;
                w[2 * k + 1][e] = q0 ? keep : got;
            }
#pragma unroll
        for (int r = 0; r < 2; r++)
#pragma unroll
            for (int e = 0; e < 2; e++) {
                const float lo = w[r][e], hi = w[2 + r][e];
                const float keep = q1 ? hi : lo, got = __shfl_xor_sync(0xffffffffu, q1 ? lo : hi, 16);
                t[r][e] = q1 ? got : keep;
                t[2 + r][e] = q1 ? keep : got;
            }
        float s = __fadd_rn(t[0][0], t[0][1]);
#pragma unroll
        for (int u = 1; u < 4; u++) s = __fadd_rn(__fadd_rn(s, t[u][0]), t[u][1]);
        s = ((codes4 >> (8 * q)) & 0xffu) == kCodeFluid ? __fmul_rn(s, out_scale) : 0.0f;
        if (valid) St<TRO>::st(rc + c0 + q, s);
    }
}

template <typename TRI, typename TZI, typename TRO>
__global__ void __launch_bounds__(256, 4) k_restrict8(const TRI *rf, const TZI *zf,
                                                      const uint8_t *__restrict__ cf, const uint16_t *__restrict__ swf,
                                                      TRO *__restrict__ rc,
                                                      const uint8_t *__restrict__ cc, Dims C, float out_scale,
                                                      const int *__restrict__ act, const int *__restrict__ act_n,
                                                      unsigned long long *kc) {
    pdl_open();
    const Dims F{2 * C.nx, 2 * C.ny, 2 * C.nz};
    restrict8_pass(rc, cc, C, out_scale, act, act_n, blockIdx.x, gridDim.x, true, kc,
                   [&](int g, float *v) { residual_row8<true>(rf, zf, cf, swf, F, g, v); });
}

// Restriction out of a level whose pre-smoothed z is colour-split
// (smooth_split.cuh); r is the natural-order residual.  512 x 256 x 256 with 31 M
// fluid cells: 127 -> 81 us (32 -> 15 M shared/L1 wavefronts and 70 -> 50 M warp
// instructions), 0.32 GB of DRAM traffic.
template <typename TRI, typename TZI, typename TRO>
__global__ void __launch_bounds__(256, 4) k_restrict8_split(const TRI *rf, const TZI *zf,
                                                            const uint32_t *__restrict__ items,
                                                            const uint16_t *__restrict__ swf, TRO *__restrict__ rc,
                                                            const uint8_t *__restrict__ cc, Dims C, float out_scale,
                                                            const int *__restrict__ act,
                                                            const int *__restrict__ act_n, unsigned long long *kc) {
    pdl_open();
    const Dims F{2 * C.nx, 2 * C.ny, 2 * C.nz};
    restrict8_pass(rc, cc, C, out_scale, act, act_n, blockIdx.x, gridDim.x, true, kc,
                   [&](int g, float *v) { residual_row8_split(rf, zf, swf, items, F, g, v); });
}

}  // namespace flub
