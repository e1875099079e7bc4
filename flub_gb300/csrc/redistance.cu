// Level-set redistance by fast sweeping (redistance.py), used by flub's
// particle level set (particles.py:255, :267-270).
//
// FP32 in the reference's operation order through explicit round-to-nearest
// intrinsics; x ** 2.0 is x * x, sqrt is the correctly rounded square root;
// the min and max of two values are a < b ? a : b and a > b ? a : b.
#include "common.cuh"

namespace flub {

__device__ __forceinline__ float rd_min(float a, float b) { return a < b ? a : b; }
__device__ __forceinline__ float rd_max(float a, float b) { return a > b ? a : b; }

// utils/util.py:403-412 fraction_of_fluid.
__device__ __forceinline__ float rd_frac(float p1, float p2) {
    if (p1 < 0.0f && p2 < 0.0f) return 1.0f;
    if (p1 >= 0.0f && p2 >= 0.0f) return 0.0f;
    return __fsub_rn(1.0f, __fdiv_rn(fmaxf(p1, p2), fabsf(__fsub_rn(p1, p2))));
}

// redistance.py:66-119 _init_distance, out of place: every cell reads the
// values from before the launch (the reference rewrites phi in place inside
// one launch, where a cell may read a neighbour already rewritten).
// Neighbours outside the grid read 0.5 h; the neighbour test keeps the
// reference's precedence, (!boundary && left) || right || ... .
// kSplit: the row is written with its even k first (rd_row below).
// Grid: row_grid(nx, ny, nz).
template <bool kSplit>
__global__ void __launch_bounds__(kRowThreads) k_redistance_init(const float *__restrict__ phi, float *__restrict__ out,
                                                                int nx, int ny, int nz, float h, int set_boundary) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x, j = blockIdx.y, i = blockIdx.z;
    if (k >= nz) return;
    const int64_t c = ((int64_t)i * ny + j) * nz + k, sj = nz, si = (int64_t)ny * nz;
    const float hb = __fmul_rn(0.5f, h);
    const float pl = i > 0 ? __ldg(phi + c - si) : hb, pr = i < nx - 1 ? __ldg(phi + c + si) : hb;
    const float pb = j > 0 ? __ldg(phi + c - sj) : hb, pt = j < ny - 1 ? __ldg(phi + c + sj) : hb;
    const float pf = k > 0 ? __ldg(phi + c - 1) : hb, pn = k < nz - 1 ? __ldg(phi + c + 1) : hb;
    const float pc = __ldg(phi + c);
    const bool bnd = i == 0 || i == nx - 1 || j == 0 || j == ny - 1 || k == 0 || k == nz - 1;
    float v = pc;
    if (bnd && !set_boundary) {
        v = pc;
    } else if (pc > 0.0f) {
        if ((!bnd && pl < 0.0f) || pr < 0.0f || pb < 0.0f || pt < 0.0f || pf < 0.0f || pn < 0.0f) {
            float m = __fsub_rn(1.0f, rd_frac(pc, pl));
            m = rd_min(m, __fsub_rn(1.0f, rd_frac(pc, pr)));
            m = rd_min(m, __fsub_rn(1.0f, rd_frac(pc, pb)));
            m = rd_min(m, __fsub_rn(1.0f, rd_frac(pc, pt)));
            m = rd_min(m, __fsub_rn(1.0f, rd_frac(pc, pf)));
            m = rd_min(m, __fsub_rn(1.0f, rd_frac(pc, pn)));
            v = __fmul_rn(h, m);
        } else {
            v = 2.0f;
        }
    } else if (pc < 0.0f) {
        if ((!bnd && pl > 0.0f) || pr > 0.0f || pb > 0.0f || pt > 0.0f || pf > 0.0f || pn > 0.0f) {
            float m = rd_frac(pc, pl);
            m = rd_min(m, rd_frac(pc, pr));
            m = rd_min(m, rd_frac(pc, pb));
            m = rd_min(m, rd_frac(pc, pt));
            m = rd_min(m, rd_frac(pc, pf));
            m = rd_min(m, rd_frac(pc, pn));
            v = __fmul_rn(-h, m);
        } else {
            v = -2.0f;
        }
    }
    out[kSplit ? c - k + ((k & 1) ? ((nz + 1) >> 1) : 0) + (k >> 1) : c] = v;
}

// redistance.py:7-55 update of a cell off the boundary with |pc| > h from its
// neighbours (x, y, z: the one against the sweep's increment, then the one
// along it): the upwind-sorted values and the 1-, 2- or 3-neighbour Eikonal
// solution, kept where smaller than |pc|.
__device__ __forceinline__ float rd_update(float pc, float phii, float phiii, float phij, float phijj, float phik,
                                           float phikk, float h) {
    float sgn = 1.0f;
    if (phii < 0.0f) {
        phii = -rd_max(phii, phiii);
        phij = -rd_max(phij, phijj);
        phik = -rd_max(phik, phikk);
        sgn = -1.0f;
    } else {
        phii = rd_min(phii, phiii);
        phij = rd_min(phij, phijj);
        phik = rd_min(phik, phikk);
    }
    const float phi0 = rd_min(rd_min(phii, phij), phik);
    const float phi2 = rd_max(rd_max(phii, phij), phik);
    // Where no neighbour has a distance yet (all three at the 2 of the
    // initialisation) no solution below 2 exists: phi1 is exactly 2, the sums 4 and
    // 6 are exact, each square root is at least 0, and 6 times the rounded 1/3 rounds
    // to 2.  (A larger phi2, a boundary value that was kept, could round phi1 below
    // phi0.)  Most warps far from the interface leave here.
    if (phi0 >= 2.0f && phi2 <= 2.0f && fabsf(pc) <= 2.0f && h >= 0.0f) return __fmul_rn(sgn, fabsf(pc));
    const float phi1 = __fsub_rn(__fsub_rn(__fadd_rn(__fadd_rn(phii, phij), phik), phi0), phi2);
    float d = __fadd_rn(phi0, h);
    if (d > phi1) {
        const float e = __fsub_rn(phi0, phi1);
        d = __fmul_rn(0.5f, __fadd_rn(__fadd_rn(phi0, phi1),
                                      __fsqrt_rn(__fsub_rn(__fmul_rn(__fmul_rn(2.0f, h), h), __fmul_rn(e, e)))));
        if (d > phi2) {
            const float s = __fadd_rn(__fadd_rn(phi0, phi1), phi2);
            const float sq = __fadd_rn(__fadd_rn(__fmul_rn(phi0, phi0), __fmul_rn(phi1, phi1)), __fmul_rn(phi2, phi2));
            const float term = __fsub_rn(__fmul_rn(s, s), __fmul_rn(3.0f, __fsub_rn(sq, __fmul_rn(h, h))));
            d = __fmul_rn(1.0f / 3.0f, __fadd_rn(s, __fsqrt_rn(rd_max(0.0f, term))));
        }
    }
    return __fmul_rn(sgn, rd_min(d, fabsf(pc)));
}

// redistance.py:58-63 _sweep: the cells of one parity (colour), off the
// boundary with |phi| > h.  A cell reads only its six neighbours, all of the
// other parity, so the cells of one launch are independent.  Thread t of row
// (i, j) owns k = 2 t + ((colour + i + j) & 1).
// Grid: row_grid(nx, ny, ceil(nz / 2)).
__global__ void __launch_bounds__(kRowThreads) k_redistance_sweep(float *phi, int nx, int ny, int nz, int incx, int incy,
                                                                 int incz, int colour, float h) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x, j = blockIdx.y, i = blockIdx.z;
    const int k = 2 * t + ((colour + i + j) & 1);
    if (k >= nz) return;
    if (i == 0 || i == nx - 1 || j == 0 || j == ny - 1 || k == 0 || k == nz - 1) return;
    const int64_t c = ((int64_t)i * ny + j) * nz + k, sj = nz, si = (int64_t)ny * nz;
    const float pc = phi[c];
    if (!(fabsf(pc) > h)) return;
    const int64_t dx = incx * si, dy = incy * sj, dz = incz;
    phi[c] = rd_update(pc, __ldg(phi + c - dx), __ldg(phi + c + dx), __ldg(phi + c - dy), __ldg(phi + c + dy),
                       __ldg(phi + c - dz), __ldg(phi + c + dz), h);
}

// The same inside flub_redistance, whose array keeps each row's even k first,
// then its odd ones: the cells of one colour in a row are then consecutive, as
// are all their neighbours (the i and j neighbours, of the other colour, have
// the same k and so the same place in their rows; the k neighbours are in the
// row's other part).  In natural order every load of a warp took two lines and
// used half of each.  A lane owns kRdCells cells, 32 apart, with their loads
// in flight together; loads need no alignment, so any nz does.
// Block: kRdRows rows j of 32 lanes.  Grid: (ceil(nz / 2 / (32 kRdCells)),
// ceil(ny / kRdRows), nx).
// Measured at 256 x 64 x 256: 14.2 us a launch in natural order with one cell
// a thread (and every cell far from the interface taking both square roots),
// see flub_redistance for the whole.
constexpr int kRdCells = 4, kRdRows = 4;

__global__ void __launch_bounds__(32 * kRdRows) k_redistance_sweep_rows(float *phi, int nx, int ny, int nz, int incx,
                                                                      int incy, int incz, int colour, float h) {
    // launched with programmatic dependent launch: the next sweep's blocks come
    // up while this one drains, and wait here for its results
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const int i = blockIdx.z, j = blockIdx.y * kRdRows + threadIdx.y;
    if (i == 0 || i == nx - 1 || j == 0 || j >= ny - 1) return;
    const int q = (colour + i + j) & 1, he = (nz + 1) >> 1;  // the cells have k = 2 t + q
    const int64_t row = ((int64_t)i * ny + j) * nz;
    float *own = phi + row + (q ? he : 0);
    const float *oth = phi + row + (q ? 0 : he) + (q - 1);  // oth[t]: k - 1, oth[t + 1]: k + 1
    const int64_t dx = (int64_t)incx * ny * nz, dy = (int64_t)incy * nz;
    const int t0 = blockIdx.x * 32 * kRdCells + threadIdx.x;
    float pc[kRdCells], xm[kRdCells], xp[kRdCells], ym[kRdCells], yp[kRdCells], zm[kRdCells], zp[kRdCells];
#pragma unroll
    for (int u = 0; u < kRdCells; u++) {
        const int t = t0 + 32 * u, k = 2 * t + q;
        pc[u] = 0.0f;
        if (k < 1 || k >= nz - 1) continue;
        // not the read-only path: the sweep in front of this one may have been
        // writing these cells while this block was already resident
        pc[u] = own[t];
        xm[u] = own[t - dx];
        xp[u] = own[t + dx];
        ym[u] = own[t - dy];
        yp[u] = own[t + dy];
        zm[u] = oth[t + (incz < 0 ? 1 : 0)];
        zp[u] = oth[t + (incz < 0 ? 0 : 1)];
    }
#pragma unroll
    for (int u = 0; u < kRdCells; u++) {
        const int t = t0 + 32 * u, k = 2 * t + q;
        if (k < 1 || k >= nz - 1 || !(fabsf(pc[u]) > h)) continue;
        own[t] = rd_update(pc[u], xm[u], xp[u], ym[u], yp[u], zm[u], zp[u], h);
    }
}

// Rows back in natural order, in place: one warp a row, through shared memory
// (nz floats a row).  Grid: ceil(rows / kRdRows).
constexpr int kRdMaxRow = 2048;  // longer rows stay in natural order throughout
__global__ void __launch_bounds__(32 * kRdRows) k_redistance_natural(float *phi, int64_t rows, int nz) {
    extern __shared__ float rd_row[];
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const int64_t r = (int64_t)blockIdx.x * kRdRows + threadIdx.y;
    if (r >= rows) return;
    float *row = phi + r * nz, *s = rd_row + threadIdx.y * nz;
    const int he = (nz + 1) >> 1;
    for (int e = threadIdx.x; e < nz; e += 32) s[e] = row[e];
    __syncwarp();
    for (int k = threadIdx.x; k < nz; k += 32) row[k] = s[((k & 1) ? he : 0) + (k >> 1)];
}

// redistance.py:128-136: the eight sweep directions of one round.
constexpr int kSweepDirs[8][3] = {{1, 1, -1}, {-1, 1, -1}, {-1, -1, -1}, {1, -1, -1},
                                  {1, 1, 1},  {-1, 1, 1},  {-1, -1, 1},  {1, -1, 1}};

// The parity of the cells the reference's launch _sweep(..., odd) updates:
// its thread (a, b, c) with (a + b + c) % 2 == odd writes the cell mirrored on
// every axis with a negative increment, which flips the parity by n - 1 on
// that axis.
static inline int sweep_colour(int nx, int ny, int nz, int incx, int incy, int incz, int odd) {
    int c = odd;
    if (incx < 0) c += nx - 1;
    if (incy < 0) c += ny - 1;
    if (incz < 0) c += nz - 1;
    return c & 1;
}

static int launch_sweep(float *phi, int nx, int ny, int nz, int incx, int incy, int incz, int odd, float h,
                        cudaStream_t s) {
    const int colour = sweep_colour(nx, ny, nz, incx, incy, incz, odd);
    k_redistance_sweep<<<row_grid(nx, ny, (nz + 1) / 2), kRowThreads, 0, s>>>(phi, nx, ny, nz, incx, incy, incz,
                                                                             colour, h);
    FLUB_CHECK_LAUNCH();
    return FLUB_OK;
}

static inline bool rd_shape_ok(int nx, int ny, int nz) {
    return nx > 0 && ny > 0 && nz > 0 && nx < 65536 && ny < 65536;
}

}  // namespace flub

using namespace flub;

extern "C" {

int flub_redistance_init(const float *phi, float *out, int nx, int ny, int nz, float h, int set_boundary,
                         void *stream) {
    FLUB_REQUIRE(phi && out, "flub_redistance_init: NULL argument");
    FLUB_REQUIRE(phi != out, "flub_redistance_init: out must not alias phi");
    FLUB_REQUIRE(rd_shape_ok(nx, ny, nz), "flub_redistance_init: bad shape %dx%dx%d", nx, ny, nz);
    k_redistance_init<false><<<row_grid(nx, ny, nz), kRowThreads, 0, as_stream(stream)>>>(phi, out, nx, ny, nz, h,
                                                                                 set_boundary);
    FLUB_CHECK_LAUNCH();
    return FLUB_OK;
}

int flub_redistance_sweep(float *phi, int nx, int ny, int nz, int incx, int incy, int incz, int odd, float h,
                          void *stream) {
    FLUB_REQUIRE(phi, "flub_redistance_sweep: NULL argument");
    FLUB_REQUIRE(rd_shape_ok(nx, ny, nz), "flub_redistance_sweep: bad shape %dx%dx%d", nx, ny, nz);
    FLUB_REQUIRE((incx == 1 || incx == -1) && (incy == 1 || incy == -1) && (incz == 1 || incz == -1),
                 "flub_redistance_sweep: increments must be +1 or -1");
    FLUB_REQUIRE(odd == 0 || odd == 1, "flub_redistance_sweep: odd must be 0 or 1");
    return launch_sweep(phi, nx, ny, nz, incx, incy, incz, odd, h, as_stream(stream));
}

int flub_redistance(const float *phi, float *phi_out, int nx, int ny, int nz, float h, int set_boundary, int n_rounds,
                    void *stream) {
    FLUB_REQUIRE(phi && phi_out, "flub_redistance: NULL argument");
    FLUB_REQUIRE(phi != phi_out, "flub_redistance: phi_out must not alias phi");
    FLUB_REQUIRE(rd_shape_ok(nx, ny, nz), "flub_redistance: bad shape %dx%dx%d", nx, ny, nz);
    FLUB_REQUIRE(n_rounds >= 0, "flub_redistance: n_rounds must be >= 0");
    cudaStream_t s = as_stream(stream);
    if (n_rounds == 0 || nz > kRdMaxRow) {
        k_redistance_init<false><<<row_grid(nx, ny, nz), kRowThreads, 0, s>>>(phi, phi_out, nx, ny, nz, h, set_boundary);
        FLUB_CHECK_LAUNCH();
    } else {
        k_redistance_init<true><<<row_grid(nx, ny, nz), kRowThreads, 0, s>>>(phi, phi_out, nx, ny, nz, h, set_boundary);
        FLUB_CHECK_LAUNCH();
    }
    const dim3 grid((unsigned)(((nz + 1) / 2 + 32 * kRdCells - 1) / (32 * kRdCells)),
                    (unsigned)((ny + kRdRows - 1) / kRdRows), (unsigned)nx),
        block(32, kRdRows);
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.stream = s;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    for (int r = 0; r < n_rounds; r++)
        for (int d = 0; d < 8; d++)
            for (int odd = 0; odd < 2; odd++) {
                const int ix = kSweepDirs[d][0], iy = kSweepDirs[d][1], iz = kSweepDirs[d][2];
                if (nz > kRdMaxRow) {
                    const int st = launch_sweep(phi_out, nx, ny, nz, ix, iy, iz, odd, h, s);
                    if (st != FLUB_OK) return st;
                    continue;
                }
                FLUB_CHECK_CUDA(cudaLaunchKernelEx(&cfg, k_redistance_sweep_rows, phi_out, nx, ny, nz, ix, iy, iz,
                                                   sweep_colour(nx, ny, nz, ix, iy, iz, odd), h));
                count_launches(1);
            }
    if (n_rounds > 0 && nz <= kRdMaxRow) {
        const int64_t rows = (int64_t)nx * ny;
        cfg.gridDim = dim3((unsigned)((rows + kRdRows - 1) / kRdRows));
        cfg.dynamicSmemBytes = sizeof(float) * kRdRows * nz;
        FLUB_CHECK_CUDA(cudaLaunchKernelEx(&cfg, k_redistance_natural, phi_out, rows, nz));
        count_launches(1);
    }
    return FLUB_OK;
}

}  // extern "C"
