// The part of a CG iteration between two V-cycles in two launches of one cluster
// each, for grids of at most 65,536 cells (multigrid/mgpcg.py:410-461):
// k_cg_small_dir takes z.r -> beta, x += alpha p and p = z + beta p, k_cg_small_res A p
// with p.Ap -> alpha, r -= alpha A p and r.r with the convergence test.
//
// On such a grid each of the four kernels (k8_dot_zr, k8_update_xp, k8_matvec_pap,
// k8_update_r_rr) is a launch, a few loads and a reduction through global memory --
// partials, fence, ticket, the last block's sums: 5 to 6 microseconds a reduction
// for less than one of work.  Here at most 16 blocks hold the grid in registers,
// one or two 8-cell groups a thread, A p never leaves them, a reduction is a block's
// sum, one value stored in every other block's shared memory and a cluster
// barrier, and what the V-cycle does not write (r, x, p) is loaded while it still
// runs.  32^3: 20 -> 8 us an iteration; above 65,536 cells the vectors outgrow
// a cluster.  (All of it in one launch would need p exchanged between the blocks.)
// Cell by cell the operations are those of the four kernels; the FP64 partial sums
// are added in another fixed order.
#pragma once

#include "cg8.cuh"
#include "coarse.cuh"

namespace flub {

constexpr int kCgSmallMaxCells = 65536;
constexpr int kCgSmallMaxBlocks = 16;

struct CgSmallArgs {
    Dims D;
    MgState *st;
    float *x, *p, *r;
    const float *z;
    const uint8_t *code;
    const uint32_t *items;
    const uint16_t *sw;
    double *hist;
    cudaGraphConditionalHandle h;
    int set_cond;
};

__device__ __forceinline__ void remote_store64(uint32_t a, double v) {
    asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(a), "d"(v) : "memory");
}

// Sum over the cluster, in every thread; slot: one entry per block, not used by
// another sum of the launch.
__device__ __forceinline__ double cluster_sum(double v, double *slot, double *out) {
    const double b = block_sum_red(v);
    const unsigned lane = threadIdx.x & 31, blocks = gridDim.x;
    if (threadIdx.x < 32) {
        const double mine = __shfl_sync(0xffffffffu, b, 0);
        if (lane < blocks) remote_store64(remote_addr(slot + blockIdx.x, lane), mine);
    }
    cluster_barrier();
    if (threadIdx.x < 32) {
        const double t = warp_sum(lane < blocks ? slot[lane] : 0.0);
        if (threadIdx.x == 0) *out = t;
    }
    __syncthreads();
    return *out;
}

// The groups of a thread: those with fluid (the others hold 0 in z, p and A p).
template <int G>
struct CgGroups {
    int g[G];
    bool in[G];
};

template <int G>
__device__ __forceinline__ CgGroups<G> cg_groups(const CgSmallArgs &A, int ng) {
    CgGroups<G> o;
#pragma unroll
    for (int q = 0; q < G; q++) {
        o.g[q] = ((int)blockIdx.x * G + q) * kRedThreads + (int)threadIdx.x;
        o.in[q] = o.g[q] < ng && group_has_fluid(load_codes8(A.code + (o.g[q] << 3)));
    }
    return o;
}

// z.r -> beta; x += alpha p; p = z + beta p; it += 1.
template <int G>
__global__ void __launch_bounds__(kRedThreads, 1) k_cg_small_dir(const CgSmallArgs A, unsigned long long *kc) {
    __shared__ double slots[kCgSmallMaxBlocks], sum, bcast;
    pdl_open();
    cluster_barrier();  // every block runs before another stores into its shared memory
    const CgGroups<G> w = cg_groups<G>(A, (int)(A.D.n() >> 3));
    float z[G][8], r[G][8], p[G][8], x[G][8];
#pragma unroll
    for (int q = 0; q < G; q++) {
        if (!w.in[q]) continue;
        const size_t c = (size_t)w.g[q] << 3;
        St<float>::ld8_wide(A.r + c, r[q]);
        St<float>::ld8_wide(A.p + c, p[q]);
        St<float>::ld8_wide(A.x + c, x[q]);
    }
    MgState *st = A.st;
    const float alpha = (float)st->alpha;
    const double zr_old = st->zr_old, eps = st->eps;
    const int it = st->it;
    pdl_wait(kc);
    double s = 0.0;
#pragma unroll
    for (int q = 0; q < G; q++) {
        if (!w.in[q]) continue;
        St<float>::ld8_wide(A.z + ((size_t)w.g[q] << 3), z[q]);
        s += dot8_ff(z[q], r[q]);
    }
    const double zr = cluster_sum(s, slots, &sum);
    if (threadIdx.x == 0) bcast = zr / (zr_old + eps);
    __syncthreads();
    const double beta = bcast;
    const float b = (float)beta;
#pragma unroll
    for (int q = 0; q < G; q++) {
        if (!w.in[q]) continue;
        const size_t c = (size_t)w.g[q] << 3;
#pragma unroll
        for (int m = 0; m < 8; m++) {
            x[q][m] = __fmaf_rn(alpha, p[q][m], x[q][m]);
            p[q][m] = __fmaf_rn(b, p[q][m], z[q][m]);
        }
        St<float>::st8_wide(A.x + c, x[q]);
        St<float>::st8_wide(A.p + c, p[q]);
    }
    if ((blockIdx.x | threadIdx.x) == 0) {
        st->beta = beta;
        st->zr_old = zr;
        st->it = it + 1;
        if (!isfinite(beta)) st->status = FLUB_ERR_BREAKDOWN;
    }
}

// A p; p.Ap -> alpha; r -= alpha A p; r.r, convergence test and loop condition.
template <int G>
__global__ void __launch_bounds__(kRedThreads, 1) k_cg_small_res(const CgSmallArgs A, unsigned long long *kc) {
    __shared__ double slots[2][kCgSmallMaxBlocks], sum[2], bcast;
    pdl_open();
    cluster_barrier();  // every block runs before another stores into its shared memory
    const Dims D = A.D;
    const int ng = (int)(D.n() >> 3);
    const CgGroups<G> w = cg_groups<G>(A, ng);
    MgState *st = A.st;
    const int skip = st->skip_r;
    const double eps = st->eps, tol = st->tol;
    float r[G][8], a[G][8];
    uint32_t e[G], o[G];
    double s = 0.0, off = 0.0;  // off: r.r off the fluid, of a residual that was not masked
#pragma unroll
    for (int q = 0; q < G; q++) {
        if (w.g[q] >= ng || (skip && !w.in[q])) continue;
        St<float>::ld8_wide(A.r + ((size_t)w.g[q] << 3), r[q]);
        if (!w.in[q]) off += dot8_ff(r[q], r[q]);
        e[q] = __ldg(A.items + w.g[q]);
        o[q] = __ldg(A.items + ng + w.g[q]);
    }
    pdl_wait(kc);
    const bool lead = (blockIdx.x | threadIdx.x) == 0;
    const int it = st->it;
    const double zr = st->zr_old;
    // the same in every thread of the cluster
    if (it >= st->max_iters || st->converged || st->status) {
        if (lead) publish_cond(st, 0, A.h, A.set_cond);
        return;
    }
    const int sj = D.nz, si = D.ny * D.nz;
#pragma unroll
    for (int q = 0; q < G; q++) {
        if (!w.in[q]) continue;
        int i, j, kg;
        group_ijk(w.g[q], D, i, j, kg);
        const float *c = A.p + ((size_t)w.g[q] << 3);
        float v[8], n[4][8], km[8], kp[8];
        St<float>::ld8_wide(c, v);
        St<float>::ld8_wide(i + 1 < D.nx ? c + si : c, n[0]);
        St<float>::ld8_wide(i > 0 ? c - si : c, n[1]);
        St<float>::ld8_wide(j + 1 < D.ny ? c + sj : c, n[2]);
        St<float>::ld8_wide(j > 0 ? c - sj : c, n[3]);
        const float xm = kg > 0 ? c[-1] : v[0], xp = 8 * kg + 8 < D.nz ? c[8] : v[7];
#pragma unroll
        for (int m = 0; m < 8; m++) {
            km[m] = m > 0 ? v[m > 0 ? m - 1 : 0] : xm;
            kp[m] = m < 7 ? v[m < 7 ? m + 1 : 7] : xp;
        }
        if ((e[q] | o[q]) & kItemSolid) {
            const uint4 wd = __ldg(reinterpret_cast<const uint4 *>(A.sw + ((size_t)w.g[q] << 3)));
#pragma unroll
            for (int m = 0; m < 8; m++) {
                const uint32_t ns = sw_ns(word_at(wd, m));
                if (!(ns & 4u)) n[0][m] = v[m];
                if (!(ns & 16u)) n[1][m] = v[m];
                if (!(ns & 64u)) n[2][m] = v[m];
                if (!(ns & 256u)) n[3][m] = v[m];
                if (!(ns & 1024u)) kp[m] = v[m];
                if (!(ns & 4096u)) km[m] = v[m];
            }
        }
        const uint32_t ia = (i + j) & 1 ? o[q] : e[q], ib = (i + j) & 1 ? e[q] : o[q];  // k = 2 m, 2 m + 1
#pragma unroll
        for (int m = 0; m < 8; m++) {
            float lz = __fadd_rn(0.0f, __fadd_rn(__fsub_rn(n[0][m], v[m]), __fsub_rn(n[1][m], v[m])));
            lz = __fadd_rn(lz, __fadd_rn(__fsub_rn(n[2][m], v[m]), __fsub_rn(n[3][m], v[m])));
            lz = __fadd_rn(lz, __fadd_rn(__fsub_rn(kp[m], v[m]), __fsub_rn(km[m], v[m])));
            a[q][m] = (((m & 1) ? ib : ia) >> (4 * (m >> 1))) & 7u ? lz : 0.0f;
        }
        s += dot8_ff(v, a[q]);
    }
    const double pap = cluster_sum(s, slots[0], &sum[0]);
    if (threadIdx.x == 0) bcast = zr / (pap + eps);
    __syncthreads();
    const double alpha = bcast;
    if (lead) {
        st->pap = pap;
        st->alpha = alpha;
    }
    if (!isfinite(alpha)) {
        if (lead) {
            st->status = FLUB_ERR_BREAKDOWN;
            publish_cond(st, 0, A.h, A.set_cond);
        }
        return;
    }
    const float al = (float)alpha;
    s = off;
#pragma unroll
    for (int q = 0; q < G; q++) {
        if (!w.in[q]) continue;
#pragma unroll
        for (int m = 0; m < 8; m++) r[q][m] = __fmaf_rn(-al, a[q][m], r[q][m]);
        St<float>::st8_wide(A.r + ((size_t)w.g[q] << 3), r[q]);
        s += dot8_ff(r[q], r[q]);
    }
    const double rtr = cluster_sum(s, slots[1], &sum[1]);
    if (lead) {
        st->rtr = rtr;
        if (it < kHistory) A.hist[it] = rtr;
        const bool bad = !isfinite(rtr);
        if (bad) st->status = FLUB_ERR_BREAKDOWN;
        const int conv = rtr < tol;
        st->converged = conv;
        publish_cond(st, (!conv && !bad) ? 1 : 0, A.h, A.set_cond);
    }
}

}  // namespace flub
