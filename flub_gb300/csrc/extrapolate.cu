// Velocity extrapolation after the projection (water_3d.py:70-73 extrapolate,
// the step that follows project() in water_3d.step, :102).
//
// Face flags ("unknown", int32 per face, the reference's MACGridInt):
// 1 = to be extrapolated, 0 = known, -1 = extrapolated in the current pass.
#include "common.cuh"

namespace flub {

// utils/util.py:423-437 set_unknown over the cell grid: face (i, j, k) of
// every axis gets 1 where phi >= 0, else 0 (i < nx, j < ny, k < nz; the last
// face layer of each array is left as it was).  Grid: row_grid(nx, ny, nz).
__global__ void __launch_bounds__(kRowThreads) k_set_unknown(const float *__restrict__ phi, int32_t *__restrict__ tu,
                                                            int32_t *__restrict__ tv, int32_t *__restrict__ tw, int nx,
                                                            int ny, int nz) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x, j = blockIdx.y, i = blockIdx.z;
    if (k >= nz) return;
    const int32_t v = phi[((int64_t)i * ny + j) * nz + k] >= 0.0f ? 1 : 0;
    tu[((int64_t)i * ny + j) * nz + k] = v;
    tv[((int64_t)i * (ny + 1) + j) * nz + k] = v;
    tw[((int64_t)i * ny + j) * (nz + 1) + k] = v;
}

// extrapolate.py:8-30 extrapolate_3d on one face array q (fx, fy, fz): a face
// with flag 1 takes the mean of its in-bounds 3x3x3 neighbours (itself
// included) whose flag is 0, summed in (ii, jj, kk) order, kk fastest, FP32;
// with none it becomes 0.  kMark: set the flag of an extrapolated face to -1
// (the reference's kernel); otherwise leave it 1, which is the state its
// flush_1_3d (-1 -> 1) restores right after -- only flag-0 faces are ever
// read, so the two give the same values.
//
// One block owns a tile of kTi x kTj x kTk faces and stages the tile plus a
// one-face halo in shared memory (flags as bytes: 0 known, 1 to extrapolate,
// 2 any other flag or outside the array); each of its 256 threads then
// updates kTi faces along i.
// Known faces are never written during a pass and only known faces are read,
// so staging before other blocks write cannot change a result.
constexpr int kTi = 4, kTj = 8, kTk = 32;
constexpr int kHi = kTi + 2, kHj = kTj + 2, kHk = kTk + 2;

template <bool kMark>
__global__ void __launch_bounds__(kTj * kTk) k_extrapolate_tile(float *__restrict__ q, int32_t *__restrict__ unk,
                                                               int fx, int fy, int fz) {
    __shared__ float sv[kHi * kHj * kHk];
    __shared__ uint8_t sk[kHi * kHj * kHk];
    __shared__ int any_known;
    const int i0 = blockIdx.z * kTi, j0 = blockIdx.y * kTj, k0 = blockIdx.x * kTk;
    const int tid = threadIdx.y * kTk + threadIdx.x;
    if (tid == 0) any_known = 0;
    __syncthreads();
    int known = 0;
    for (int e = tid; e < kHi * kHj * kHk; e += kTj * kTk) {
        const int hk = e % kHk, hj = (e / kHk) % kHj, hi = e / (kHk * kHj);
        const int a = i0 + hi - 1, b = j0 + hj - 1, c = k0 + hk - 1;
        uint8_t kn = 2;
        float v = 0.0f;
        if (a >= 0 && a < fx && b >= 0 && b < fy && c >= 0 && c < fz) {
            const int64_t g = ((int64_t)a * fy + b) * fz + c;
            const int32_t fl = __ldg(unk + g);
            if (fl == 0) {
                kn = 0;
                v = __ldg(q + g);
                known = 1;
            } else if (fl == 1) {
                kn = 1;
            }
        }
        sk[e] = kn;
        sv[e] = v;
    }
    if (known) any_known = 1;
    __syncthreads();
    const int k = k0 + threadIdx.x, j = j0 + threadIdx.y;
    if (k >= fz || j >= fy) return;
    const bool none = any_known == 0;  // no known face in the tile and its halo: every unknown face becomes 0
#pragma unroll
    for (int ti = 0; ti < kTi; ti++) {
        const int i = i0 + ti;
        if (i >= fx) break;
        const int64_t f = ((int64_t)i * fy + j) * fz + k;
        const int hc = ((ti + 1) * kHj + threadIdx.y + 1) * kHk + threadIdx.x + 1;
        if (sk[hc] != 1) continue;  // known, or a flag other than 1: not touched, as in the reference
        if (none) {
            q[f] = 0.0f;
            continue;
        }
        int n = 0;
        float s = 0.0f;
#pragma unroll
        for (int ii = -1; ii <= 1; ii++)
#pragma unroll
            for (int jj = -1; jj <= 1; jj++)
#pragma unroll
                for (int kk = -1; kk <= 1; kk++) {
                    const int h = hc + (ii * kHj + jj) * kHk + kk;
                    if (sk[h] != 0) continue;
                    n++;
                    s = __fadd_rn(s, sv[h]);
                }
        if (n > 0) {
            q[f] = __fdiv_rn(s, (float)n);
            if (kMark) unk[f] = -1;
        } else {
            q[f] = 0.0f;
        }
    }
}

// set_unknown and one extrapolation pass of the three face arrays in one
// kernel, from the level set.  Inside the cell grid all three axes share the
// flag phi >= 0 of set_unknown, so one staging of phi serves them; only the
// last face layer of each array (i == nx of u, j == ny of v, k == nz of w)
// takes its flag from the caller's arrays, patched in by the tiles that reach
// it.
//
// A block owns kPi x kPj x kPk faces.  "Known" and "to extrapolate" are one
// bit per face (a ballot per 32 faces along k, with a one-face halo of known
// bits); a thread per word finds the faces that border a known one, and only
// those load face values.  The other unknown faces are written as 0 from the
// bits alone.
constexpr int kPi = 8, kPj = 8, kPk = 128, kPWords = kPk / 32;
constexpr int kPRows = (kPi + 2) * (kPj + 2);
constexpr int kPThreads = kPi * kPj * kPWords;  // one word each in the second step
constexpr int64_t kFusedCells = 1 << 22;        // above: see flub_extrapolate

struct ExtrapArgs {
    float *q[3];
    int32_t *t[3];
    const float *phi;
    int nx, ny, nz;
};

struct ExtrapTile {
    // of each row: words 1 .. kPWords cover the tile's k range; word 0 holds
    // the face below it in bit 31, word kPWords + 1 the face above it in bit 0
    uint32_t known[kPRows][kPWords + 2], todo[kPRows][kPWords + 2];
    uint32_t near[kPi * kPj][kPWords];  // a known face in the 3x3x3 block around
};

// Row (ra, rb) of the halo: the known and to-extrapolate bits of its faces,
// from state(k) = bit 0 known, bit 1 to extrapolate.  One warp.
template <typename F>
__device__ __forceinline__ void extrap_row(ExtrapTile &T, int row, int lane, F state) {
    unsigned st[kPWords];
#pragma unroll
    for (int w = 0; w < kPWords; w++) st[w] = state(32 * w + lane);
    const unsigned edge = lane < 2 ? state(lane ? kPk : -1) : 0u;
#pragma unroll
    for (int w = 0; w < kPWords; w++) {
        const uint32_t kn = __ballot_sync(0xffffffffu, st[w] & 1u), td = __ballot_sync(0xffffffffu, st[w] & 2u);
        if (lane == 0) {
            T.known[row][w + 1] = kn;
            T.todo[row][w + 1] = td;
        }
    }
    if (lane == 0) T.known[row][0] = (edge & 1u) << 31;
    if (lane == 1) T.known[row][kPWords + 1] = edge & 1u;
}

// The last face layer of axis d from the caller's flags (set), or without a
// face again for the next axis (!set).
__device__ __forceinline__ void extrap_patch(ExtrapTile &T, const ExtrapArgs &A, int d, int i0, int j0, int k0,
                                             bool set) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int fy = A.ny + (d == 1), fz = A.nz + (d == 2);
    auto flag = [&](int a, int b, int c) -> unsigned {
        const int32_t fl = __ldg(A.t[d] + ((int64_t)a * fy + b) * fz + c);
        return fl == 0 ? 1u : (fl == 1 ? 2u : 0u);
    };
    if (d < 2) {
        for (int row = warp; row < kPRows; row += kPThreads / 32) {
            const int a = i0 - 1 + row / (kPj + 2), b = j0 - 1 + row % (kPj + 2);
            if ((d == 0 ? a != A.nx : b != A.ny)) continue;
            const bool in = set && (d == 0 ? b >= 0 && b < A.ny : a >= 0 && a < A.nx);
            extrap_row(T, row, lane, [&](int x) -> unsigned {
                const int c = k0 + x;
                return in && c >= 0 && c < A.nz ? flag(a, b, c) : 0u;
            });
        }
        return;
    }
    const int pos = A.nz - k0 + 32;  // bit pos & 31 of word pos / 32 of every row
    if (pos < 31 || pos > kPk + 32) return;
    for (int row = threadIdx.x; row < kPRows; row += kPThreads) {
        const int a = i0 - 1 + row / (kPj + 2), b = j0 - 1 + row % (kPj + 2);
        const unsigned st = set && a >= 0 && a < A.nx && b >= 0 && b < A.ny ? flag(a, b, A.nz) : 0u;
        const uint32_t bit = 1u << (pos & 31);
        uint32_t &kn = T.known[row][pos >> 5], &td = T.todo[row][pos >> 5];
        kn = (st & 1u) ? kn | bit : kn & ~bit;
        td = (st & 2u) ? td | bit : td & ~bit;
    }
}

// One word per thread: the faces of tile row threadIdx.x / kPWords with a
// known face among their 3x3x3 neighbours.
__device__ __forceinline__ void extrap_near(ExtrapTile &T) {
    const int w = threadIdx.x % kPWords, o = threadIdx.x / kPWords;
    const int rc = (o / kPj + 1) * (kPj + 2) + o % kPj + 1;
    uint32_t lo = 0u, mid = 0u, hi = 0u;
#pragma unroll
    for (int m = 0; m < 9; m++) {
        const uint32_t *r = T.known[rc + (m / 3 - 1) * (kPj + 2) + m % 3 - 1] + w;
        lo |= r[0];
        mid |= r[1];
        hi |= r[2];
    }
    T.near[o][w] = mid | (mid << 1) | (lo >> 31) | (mid >> 1) | (hi << 31);
}

__global__ void __launch_bounds__(kPThreads) k_extrapolate_phi(const ExtrapArgs A) {
    __shared__ ExtrapTile T;
    const int i0 = blockIdx.z * kPi, j0 = blockIdx.y * kPj, k0 = blockIdx.x * kPk;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int row = warp; row < kPRows; row += kPThreads / 32) {
        const int a = i0 - 1 + row / (kPj + 2), b = j0 - 1 + row % (kPj + 2);
        const bool in = a >= 0 && a < A.nx && b >= 0 && b < A.ny;
        const float *pr = A.phi + ((int64_t)(in ? a : 0) * A.ny + (in ? b : 0)) * A.nz;
        extrap_row(T, row, lane, [&](int x) -> unsigned {
            const int c = k0 + x;
            return in && c >= 0 && c < A.nz ? (__ldg(pr + c) >= 0.0f ? 2u : 1u) : 0u;
        });
    }
    __syncthreads();
    extrap_near(T);
    __syncthreads();
    bool patched = false;
    for (int d = 0; d < 3; d++) {
        const bool last = d == 0 ? i0 + kPi >= A.nx : (d == 1 ? j0 + kPj >= A.ny : k0 + kPk >= A.nz);
        if (patched || last) {
            __syncthreads();
            if (patched) extrap_patch(T, A, d - 1, i0, j0, k0, false);
            if (patched && last) __syncthreads();
            if (last) extrap_patch(T, A, d, i0, j0, k0, true);
            __syncthreads();
            extrap_near(T);
            __syncthreads();
            patched = last;
        }
        const int fx = A.nx + (d == 0), fy = A.ny + (d == 1), fz = A.nz + (d == 2);
        // (indexed by d the parameters went through local memory)
        float *q = d == 0 ? A.q[0] : (d == 1 ? A.q[1] : A.q[2]);
        int32_t *t = d == 0 ? A.t[0] : (d == 1 ? A.t[1] : A.t[2]);
        for (int o = warp; o < kPi * kPj; o += kPThreads / 32) {
            const int i = i0 + o / kPj, j = j0 + o % kPj;
            if (i >= fx || j >= fy) continue;
            const int rc = (o / kPj + 1) * (kPj + 2) + o % kPj + 1;
            const int64_t f = ((int64_t)i * fy + j) * fz + k0 + lane;
            const bool flags = i < A.nx && j < A.ny;
#pragma unroll
            for (int w = 0; w < kPWords; w++) {
                const int k = k0 + 32 * w + lane;
                const uint32_t td = T.todo[rc][w + 1], nr = T.near[o][w];
                const bool mine = (td >> lane) & 1u;
                if (flags && k < A.nz) t[f + 32 * w] = mine ? 1 : 0;  // set_unknown
                if (mine && !((nr >> lane) & 1u)) q[f + 32 * w] = 0.0f;
                if ((td & nr) == 0u) continue;
                if (!((td & nr) >> lane & 1u)) continue;
                int n = 0;
                float s = 0.0f;
                // nine loads at a time in flight, summed in (ii, jj, kk) order; a face that is
                // not known adds +0, which leaves the sum (never -0) as it is
#pragma unroll 1
                for (int ii = -1; ii <= 1; ii++) {
                    float v[9];
                    unsigned have = 0u;
#pragma unroll
                    for (int jj = -1; jj <= 1; jj++) {
                        const uint32_t *r = T.known[rc + ii * (kPj + 2) + jj] + w;
                        const unsigned b3 =  // the row's faces k - 1, k, k + 1
                            __funnelshift_r(__funnelshift_l(r[0], r[1], 1), __funnelshift_l(r[1], r[2], 1), lane) & 7u;
                        const float *qr = q + f + 32 * w + ((int64_t)ii * fy + jj) * fz;
                        have |= b3 << (3 * (jj + 1));
#pragma unroll
                        for (int kk = 0; kk < 3; kk++) v[3 * (jj + 1) + kk] = (b3 & (1u << kk)) ? qr[kk - 1] : 0.0f;
                    }
                    n += __popc(have);
#pragma unroll
                    for (int m = 0; m < 9; m++) s = __fadd_rn(s, v[m]);
                }
                q[f + 32 * w] = __fdiv_rn(s, (float)n);
            }
        }
    }
}

static inline dim3 tile_grid(int fx, int fy, int fz) {
    return dim3((unsigned)((fz + kTk - 1) / kTk), (unsigned)((fy + kTj - 1) / kTj), (unsigned)((fx + kTi - 1) / kTi));
}

// extrapolate.py:32-36 flush_1_3d.
__global__ void __launch_bounds__(256) k_flush_unknown(int32_t *__restrict__ unk, int64_t n) {
    for (int64_t c = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; c < n; c += (int64_t)gridDim.x * blockDim.x)
        if (unk[c] == -1) unk[c] = 1;
}

}  // namespace flub

using namespace flub;

extern "C" {

int flub_set_unknown(const float *phi, int32_t *tu, int32_t *tv, int32_t *tw, int nx, int ny, int nz, void *stream) {
    FLUB_REQUIRE(phi && tu && tv && tw, "flub_set_unknown: NULL argument");
    FLUB_REQUIRE(nx > 0 && ny > 0 && nz > 0 && nx < 65536 && ny < 65536, "flub_set_unknown: bad shape");
    k_set_unknown<<<row_grid(nx, ny, nz), kRowThreads, 0, as_stream(stream)>>>(phi, tu, tv, tw, nx, ny, nz);
    FLUB_CHECK_LAUNCH();
    return FLUB_OK;
}

int flub_extrapolate_axis(float *q, int32_t *unk, int nx, int ny, int nz, int d, void *stream) {
    FLUB_REQUIRE(q && unk, "flub_extrapolate_axis: NULL argument");
    FLUB_REQUIRE(d >= 1 && d <= 3, "flub_extrapolate_axis: d=%d must be 1, 2 or 3", d);
    FLUB_REQUIRE(nx > 0 && ny > 0 && nz > 0 && nx < 65535 && ny < 65535, "flub_extrapolate_axis: bad shape");
    FLUB_REQUIRE(nx + 1 < 4 * 65535, "flub_extrapolate_axis: nx too large");
    const int fx = nx + (d == 1), fy = ny + (d == 2), fz = nz + (d == 3);
    k_extrapolate_tile<true><<<tile_grid(fx, fy, fz), dim3(kTk, kTj), 0, as_stream(stream)>>>(q, unk, fx, fy, fz);
    FLUB_CHECK_LAUNCH();
    return FLUB_OK;
}

int flub_flush_unknown(int32_t *unk, int64_t n, void *stream) {
    FLUB_REQUIRE(unk && n >= 0, "flub_flush_unknown: bad arguments");
    if (n == 0) return FLUB_OK;
    k_flush_unknown<<<blocks_for(n, 256), 256, 0, as_stream(stream)>>>(unk, n);
    FLUB_CHECK_LAUNCH();
    return FLUB_OK;
}

int flub_extrapolate(float *u, float *v, float *w, int32_t *tu, int32_t *tv, int32_t *tw, const float *phi, int nx,
                     int ny, int nz, int n_passes, void *stream) {
    FLUB_REQUIRE(u && v && w && tu && tv && tw, "flub_extrapolate: NULL argument");
    FLUB_REQUIRE(nx > 0 && ny > 0 && nz > 0 && nx < 65535 && ny < 65535, "flub_extrapolate: bad shape");
    FLUB_REQUIRE(n_passes >= 0, "flub_extrapolate: n_passes must be >= 0");
    cudaStream_t s = as_stream(stream);
    // A pass leaves the flags as they were (the flush turns its -1 back into
    // 1), never writes a known face and reads no other, so every further pass
    // writes the values the first one wrote: one pass gives the result of
    // n_passes >= 1 for any input.
    //
    // The fused kernel reads the level set once and touches few faces away from the
    // interface, but near it loads every neighbour from the caches, with few blocks on
    // a small grid; the tiles have them in shared memory.  Set-up and tiles against
    // fused, a dam / white noise (an interface everywhere): 64^3 38 / 40 us and 64 / 72,
    // 128 x 96 x 128 64 / 87 and 97 / 147, 256 x 64 x 256 116 / 178 and 108 / 233,
    // 172^3 150 / 228 and 110 / 232, 256^3 383 / 619 and 199 / 628.
    if (phi && n_passes > 0 && (int64_t)nx * ny * nz > kFusedCells) {
        ExtrapArgs A{{u, v, w}, {tu, tv, tw}, phi, nx, ny, nz};
        k_extrapolate_phi<<<dim3((unsigned)(nz / kPk + 1), (unsigned)(ny / kPj + 1), (unsigned)(nx / kPi + 1)),
                            kPThreads, 0, s>>>(A);
        FLUB_CHECK_LAUNCH();
        return FLUB_OK;
    }
    if (phi) {
        k_set_unknown<<<row_grid(nx, ny, nz), kRowThreads, 0, s>>>(phi, tu, tv, tw, nx, ny, nz);
        FLUB_CHECK_LAUNCH();
    }
    if (n_passes > 0) {
        k_extrapolate_tile<false><<<tile_grid(nx + 1, ny, nz), dim3(kTk, kTj), 0, s>>>(u, tu, nx + 1, ny, nz);
        FLUB_CHECK_LAUNCH();
        k_extrapolate_tile<false><<<tile_grid(nx, ny + 1, nz), dim3(kTk, kTj), 0, s>>>(v, tv, nx, ny + 1, nz);
        FLUB_CHECK_LAUNCH();
        k_extrapolate_tile<false><<<tile_grid(nx, ny, nz + 1), dim3(kTk, kTj), 0, s>>>(w, tw, nx, ny, nz + 1);
        FLUB_CHECK_LAUNCH();
    }
    return FLUB_OK;
}

}  // extern "C"
