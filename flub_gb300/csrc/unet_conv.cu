// 3x3x3 convolution (stride 1, zero padding 1) as a tcgen05 implicit GEMM.
//
// Layout: activations channels-last [B][X][Y][Z][C] in BF16, weights
// [27][Cout][Cin] BF16 (tap = (dx+1)*9 + (dy+1)*3 + (dz+1)), FP32 accumulation.
// One CTA computes 128 consecutive output voxels (a box of nyb rows of nzb
// voxels at fixed b, x) for all Cout channels:
//   D[128 x Cout] (TMEM, FP32) = sum over taps t and sources s of
//                               A_t,s[128 x Cin_s] * W_t,s[Cout x Cin_s]^T
// where A_t,s is the input box shifted by the tap offset, loaded by TMA with
// zero fill outside the volume (= the convolution's zero padding).  A and W
// land in shared memory in the K-major swizzled layout whose swizzle width is
// one row (Cin * 2 bytes: 32, 64 or 128 B) and feed tcgen05.mma directly.
// A second source (the skip connection of a U-Net decoder) is accumulated
// into the same tile, so a concatenation is never materialised.
//
// Roles (128 threads): thread 0 issues TMA loads into a 4-stage ring, warp 1
// issues the MMAs (one per 16 input channels), all four warps run the
// epilogue (TMEM -> registers, bias, ReLU, BF16 store).  Every mbarrier wait
// is bounded; a timeout sets the error word and the CTA still frees its TMEM.
//
// k_conv3d_halo (below) computes the same convolution from input planes
// staged once per CTA; halo_plan chooses between the two kernels per layer.
// The weight gradient has two more, k_conv3d_wgrad_tc from tap tiles and
// k_conv3d_wgrad_halo from staged planes.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cudaTypedefs.h>

#include <mutex>

#include "common.cuh"

namespace flub {

constexpr int kConvThreads = 128;
constexpr int kConvStages = 4;
constexpr int kConvATile = 128 * 64 * 2;  // bytes, Cin <= 64
constexpr int kConvBTile = 64 * 64 * 2;   // bytes, Cout, Cin <= 64
constexpr int kConvStage = kConvATile + kConvBTile;
constexpr int kConvSmem = kConvStages * kConvStage + 1024 /* alignment */ + 256 /* barriers */;
constexpr uint32_t kWaitLimit = 1u << 22;

static __device__ int g_conv_error;

struct ConvGeom {
    int B, NX, NY, NZ;
    int nzb, nyb;
    int cout;
    int cin0, cin1;  // cin1 = 0: one source
    int relu;
    // forward kernel's pipeline stage: activation tile (128 voxels x max cin)
    // then weight tile, rounded to 1 KB so that every tile stays 1 KB aligned
    int a_bytes, stage_bytes;
};

__device__ __forceinline__ uint32_t smem_u32(const void *p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity) {
    for (uint32_t i = 0; i < kWaitLimit; i++) {
        uint32_t ok;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(ok)
            : "r"(bar), "r"(parity)
            : "memory");
        if (ok) return true;
    }
    return false;
}

// tcgen05 shared-memory matrix descriptor, K-major, swizzle width = row bytes.
__device__ __forceinline__ uint64_t sw_desc(uint32_t saddr, int row_bytes) {
    const uint64_t layout = row_bytes == 128 ? 2ull : (row_bytes == 64 ? 4ull : 6ull);  // 128B / 64B / 32B swizzle
    uint64_t d = 0;
    d |= (uint64_t)((saddr & 0x3FFFFu) >> 4);
    d |= (uint64_t)1 << 16;                          // leading byte offset (unused: K fits one swizzle row)
    d |= (uint64_t)((8u * row_bytes) >> 4) << 32;    // stride byte offset: 8 rows
    d |= (uint64_t)1 << 46;                          // descriptor version
    d |= layout << 61;
    return d;
}

// Instruction descriptor: kind::f16, A = B = BF16 K-major, D = FP32, M = 128.
__device__ __forceinline__ uint32_t mma_idesc(int n) {
    return (1u << 4)                       // D format FP32
           | (1u << 7) | (1u << 10)        // A, B format BF16
           | ((uint32_t)(n >> 3) << 17)    // N / 8
           | ((uint32_t)(128 >> 4) << 24); // M / 16
}

__device__ __forceinline__ void tma_load_5d(uint32_t dst, const CUtensorMap *map, int c0, int c1, int c2, int c3,
                                            int c4, uint32_t bar) {
    asm volatile(
        "cp.async.bulk.tensor.5d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5, %6}], "
        "[%7];" ::"r"(dst),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(c4), "r"(bar)
        : "memory");
}

__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap *map, int c0, int c1, uint32_t bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(
            dst),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(c0), "r"(c1), "r"(bar)
        : "memory");
}

__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float v[16]) {
    uint32_t r[16];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, "
        "%15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int q = 0; q < 16; q++) v[q] = __uint_as_float(r[q]);
}

// One lane of a converged warp.  The MMA warps run their loops with all lanes and
// predicate only the instruction: in a branch of one lane the descriptors, which
// the instruction takes from uniform registers, were moved there one by one.
// k_conv3d_tc, 4 x 32^3, 64 + 32 -> 32 channels: 86.7 us -> 72.4; 16^3, 32 -> 64:
// 17 -> 15.  k_conv3d_wgrad_tc, bound by its copies, is as fast as before.
__device__ __forceinline__ uint32_t elect_one() {
    uint32_t lead;
    asm volatile(
        "{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(lead));
    return lead;
}

// The wait of such a warp: no lane goes on, and so no slot is handed back and
// refilled, before every lane has seen the phase; one left behind could find the
// barrier's parity come round again.
__device__ __forceinline__ bool mbar_wait_warp(uint32_t bar, uint32_t parity) {
    return __all_sync(0xffffffffu, mbar_wait(bar, parity) ? 1 : 0) != 0;
}

__device__ __forceinline__ void mma_if(uint32_t lead, uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t acc) {
    asm volatile(
        "{\n\t.reg .pred p, q;\n\tsetp.ne.b32 p, %4, 0;\n\tsetp.ne.b32 q, %5, 0;\n\t"
        "@q tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d),
        "l"(a), "l"(b), "r"(idesc), "r"(acc), "r"(lead));
}

__device__ __forceinline__ void commit_if(uint32_t lead, uint32_t bar) {
    asm volatile(
        "{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %1, 0;\n\t"
        "@q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}" ::"r"(bar),
        "r"(lead)
        : "memory");
}

template <int COUT>
__global__ void __launch_bounds__(kConvThreads, 1)
    k_conv3d_tc(const __grid_constant__ CUtensorMap mx0, const __grid_constant__ CUtensorMap mw0,
                const __grid_constant__ CUtensorMap mx1, const __grid_constant__ CUtensorMap mw1, const ConvGeom g,
                const float *__restrict__ bias, __nv_bfloat16 *__restrict__ y) {
    extern __shared__ unsigned char conv_smem_raw[];
    unsigned char *smem = reinterpret_cast<unsigned char *>(
        (reinterpret_cast<uintptr_t>(conv_smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
    uint64_t *full = reinterpret_cast<uint64_t *>(smem + kConvStages * g.stage_bytes);
    uint64_t *empty = full + kConvStages;
    uint64_t *done = empty + kConvStages;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(done + 1);
    __shared__ int fail;

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    // tile -> (b, x, y0, z0)
    int t = blockIdx.x;
    const int tz = g.NZ / g.nzb, ty = g.NY / g.nyb;
    const int z0 = (t % tz) * g.nzb;
    t /= tz;
    const int y0 = (t % ty) * g.nyb;
    t /= ty;
    const int x = t % g.NX, b = t / g.NX;

    if (threadIdx.x == 0) {
        fail = 0;
        for (int s = 0; s < kConvStages; s++) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&full[s])));
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&empty[s])));
        }
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(done)));
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    constexpr uint32_t kCols = COUT < 32 ? 32 : COUT;
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                     "r"(kCols));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = *tmem_slot;

    const int nsrc = g.cin1 > 0 ? 2 : 1;
    const int T = 27 * nsrc;
    if (threadIdx.x == 0) {
        // producer
        for (int it = 0; it < T; it++) {
            const int s = it % kConvStages, u = it / kConvStages;
            if (u > 0 && !mbar_wait(smem_u32(&empty[s]), (u - 1) & 1)) {
                fail = 1;
                break;
            }
            const int src = it / 27, tap = it % 27;
            const int dx = tap / 9 - 1, dy = (tap / 3) % 3 - 1, dz = tap % 3 - 1;
            const int cin = src ? g.cin1 : g.cin0;
            const uint32_t bytes = (uint32_t)(128 * cin * 2 + COUT * cin * 2);
            const uint32_t fb = smem_u32(&full[s]);
            asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(fb), "r"(bytes) : "memory");
            const uint32_t a = smem_u32(smem + s * g.stage_bytes), w = a + g.a_bytes;
            tma_load_5d(a, src ? &mx1 : &mx0, 0, z0 + dz, y0 + dy, x + dx, b, fb);
            tma_load_2d(w, src ? &mw1 : &mw0, 0, tap * COUT, fb);
        }
    } else if (warp == 1) {
        // MMA issuer
        const uint32_t lead = elect_one(), idesc = mma_idesc(COUT);
        bool ok = true;
        for (int it = 0; it < T && ok; it++) {
            const int s = it % kConvStages, u = it / kConvStages;
            if (!mbar_wait_warp(smem_u32(&full[s]), u & 1)) {
                ok = false;
                fail = 1;
                break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const int cin = (it / 27) ? g.cin1 : g.cin0;
            const uint32_t a = smem_u32(smem + s * g.stage_bytes), w = a + g.a_bytes;
            for (int kk = 0; kk < cin / 16; kk++) {
                const uint64_t ad = sw_desc(a + kk * 32, cin * 2), bd = sw_desc(w + kk * 32, cin * 2);
                const uint32_t acc = (it > 0 || kk > 0) ? 1u : 0u;
                mma_if(lead, tmem, ad, bd, idesc, acc);
            }
            commit_if(lead, smem_u32(&empty[s]));
        }
        commit_if(lead, smem_u32(done));
    }
    __syncwarp();
    // epilogue: row m of the accumulator is TMEM lane m, owned by warp m / 32
    // warp-uniform outcome: tcgen05.ld below is a .sync.aligned warp instruction
    const bool got = __all_sync(0xffffffffu, mbar_wait(smem_u32(done), 0) ? 1 : 0) != 0;
    if (!got) fail = 1;
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const int m = warp * 32 + lane;
    const int yy = y0 + m / g.nzb, zz = z0 + m % g.nzb;
    const int64_t vox = (((int64_t)b * g.NX + x) * g.NY + yy) * g.NZ + zz;
    if (got) {
        float acc[COUT];
#pragma unroll
        for (int c = 0; c < COUT; c += 16) tmem_ld16(tmem + ((uint32_t)(warp * 32) << 16) + c, acc + c);
        __align__(16) __nv_bfloat16 out[COUT];
#pragma unroll
        for (int c = 0; c < COUT; c++) {
            float v = acc[c] + (bias ? __ldg(bias + c) : 0.0f);
            if (g.relu) v = fmaxf(v, 0.0f);
            out[c] = __float2bfloat16_rn(v);
        }
        uint4 *dst = reinterpret_cast<uint4 *>(y + vox * COUT);
#pragma unroll
        for (int q = 0; q < COUT / 8; q++) dst[q] = reinterpret_cast<const uint4 *>(out)[q];
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (fail && threadIdx.x == 0) atomicExch(&g_conv_error, 1);
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kCols));
}

// ---------------------------------------------------------------- halo-plane forward kernel
//
// The same convolution for NZ % 8 == 0 and NY % 16 == 0 when the layer's
// weights fit in shared memory, organised around input planes instead of
// tap-shifted tiles, with no TMA.
//
// A CTA owns a 16 (y) x 8 (z) voxel tile at up to xr consecutive x planes x0 ..;
// GEMM row m is voxel (y0 + m / 8, z0 + m % 8).  Input plane p (x = x0 - 1 + p)
// of every source is staged once, in coalesced 16-byte pieces, as the haloed
// 18 x 10 voxel region, zero outside the volume (the padding), in the
// no-swizzle K-major layout
//     [chunk of 8 channels][y 0..17][z 0..9][8 channels]   (16-byte rows).
// The A operand of the nine taps (dy, dz) is that plane read from start offset
// ((dy + 1) * 10 + dz + 1) * 16 bytes: a core matrix is the 8 z-voxels of one
// y-row (128 contiguous bytes), core matrices adjacent in M are one padded row
// apart (SBO = 160 bytes) and adjacent chunks one chunk region apart (LBO).
//
// An MMA of N = 16 to 64 is bound by the SM reading its A operand (about 44
// cycles for one 128 x 16 BF16 tile), so the three taps along x share it: input
// plane p contributes to the output planes p - 2, p - 1 and p of the CTA, whose
// accumulators lie side by side in TMEM (columns xi * Cout ...), and the weights
// are staged as [dy, dz][chunk][dx = 1, 0, -1][Cout][8 channels], so that one MMA
// of N = 3 Cout serves all three.  A plane is thus finished with after its own
// MMAs, and planes pass through a ring of R buffers, source 0's, then source 1's:
//   - warps 4-7 stage planes with asynchronous copies, R - 1 planes ahead and,
//     before they reuse a buffer, behind done[p - R]; when plane p has landed they
//     publish it to the tensor core (a proxy fence) and arrive on full[p];
//   - one thread of warp 8 issues its MMAs and commits them to done[p];
//   - warps 0-3 write output plane o after done[o + 2].
// Each role's chain of instructions for a plane is as long as its MMAs, so none
// does another's work.
// 4 x 64^3, 32 + 16 -> 16 channels: the tap tiles' 254 us -> 77 us; 16 -> 32
// and 16 -> 16: 105 and 72 us with one MMA a tap and no overlap -> 54 and 38.
constexpr int kHaloZ = 10, kHaloY = 18;
constexpr int kHaloRows = kHaloZ * kHaloY;  // 16-byte rows per chunk (180)
constexpr int kHaloThreads = 2 * kConvThreads + 32;
constexpr int kHaloMaxX = 16;               // output planes per CTA
// opt-in shared memory per block less an allowance for the kernel's static shared variables
constexpr int kHaloSmemMax = 227 * 1024 - 128;
constexpr int kHaloSteps = 2 * (kHaloMaxX + 2);  // planes of both sources
constexpr int kHaloBars = 8 * 2 * kHaloSteps;

struct HaloGeom {
    int B, NX, NY, NZ;
    int xr, ring;           // output planes per CTA, plane buffers
    int cin0, cin1, relu;   // cin1 = 0: one source
    int chunk0, chunk1;     // bytes from one chunk region to the next, per source
    int slot;               // bytes of a plane buffer
    int w0_off, w1_off;     // weights of source 0 and 1 (27 taps each)
    int bar_off;            // mbarriers full[], done[], TMEM slot
    uint32_t tmem_cols;
};

// tcgen05 shared-memory matrix descriptor, K-major without swizzle: core
// matrices of 8 rows x 16 bytes; lbo = bytes between core matrices adjacent
// in K, sbo = bytes between core matrices adjacent in M (or N).
__device__ __forceinline__ uint64_t ns_desc(uint32_t saddr, uint32_t lbo, uint32_t sbo) {
    uint64_t d = 0;
    d |= (uint64_t)((saddr & 0x3FFFFu) >> 4);
    d |= (uint64_t)((lbo >> 4) & 0x3FFFu) << 16;
    d |= (uint64_t)((sbo >> 4) & 0x3FFFu) << 32;
    d |= (uint64_t)1 << 46;  // descriptor version; layout type 0 (no swizzle) in bits 61-63
    return d;
}

// 16 bytes to shared memory, or 16 zero bytes (src is not read then, but is a valid address).
__device__ __forceinline__ void copy16_async(uint32_t dst, const void *src, bool in) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(__cvta_generic_to_global(src)),
                 "r"(in ? 16 : 0)
                 : "memory");
}

// Stages weights [27][COUT][Cin] (Cin = 8 << c8_log2) as
// [dy, dz][chunk][dx = 1, 0, -1][COUT][8].
template <int COUT>
__device__ __forceinline__ void halo_stage_weights(const uint4 *__restrict__ w, uint32_t dst, int c8_log2,
                                                   int tid) {
    const int C8 = 1 << c8_log2;
    const int total = 27 * COUT * C8;
    for (int q = tid; q < total; q += kConvThreads) {
        const int c = q & (C8 - 1);
        const int r = q >> c8_log2;  // tap * COUT + co
        const int tap = r / COUT, co = r - tap * COUT;
        const int row = (2 - tap / 9) * COUT + co;
        copy16_async(dst + ((((tap % 9) << c8_log2) + c) * 3 * COUT + row) * 16, w + q, true);
    }
}

// ITEMS: 16-byte items of a plane per staging thread, chunks x 180 / 128 rounded up.
template <int COUT, int ITEMS>
__global__ void __launch_bounds__(kHaloThreads, COUT == 64 || ITEMS > 6 ? 2 : 3)
    k_conv3d_halo(const __nv_bfloat16 *__restrict__ x0p, const __nv_bfloat16 *__restrict__ w0p,
                  const __nv_bfloat16 *__restrict__ x1p, const __nv_bfloat16 *__restrict__ w1p, const HaloGeom g,
                  const float *__restrict__ bias, __nv_bfloat16 *__restrict__ y) {
    extern __shared__ unsigned char conv_smem_raw[];
    unsigned char *smem = reinterpret_cast<unsigned char *>(
        (reinterpret_cast<uintptr_t>(conv_smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
    uint64_t *full = reinterpret_cast<uint64_t *>(smem + g.bar_off);
    uint64_t *done = full + kHaloSteps;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(done + kHaloSteps);
    __shared__ int fail;

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    int t = blockIdx.x;
    const int tz = g.NZ >> 3, ty = g.NY >> 4, tx = (g.NX + g.xr - 1) / g.xr;
    const int z0 = (t % tz) * 8;
    t /= tz;
    const int y0 = (t % ty) * 16;
    t /= ty;
    const int x0 = (t % tx) * g.xr, b = t / tx;
    const int xr = min(g.xr, g.NX - x0), np = xr + 2;
    const int nsrc = g.cin1 > 0 ? 2 : 1, steps = nsrc * np;  // step i: plane i % np of source i / np
    const int lg0 = g.cin0 == 16 ? 1 : (g.cin0 == 32 ? 2 : 3), lg1 = g.cin1 == 16 ? 1 : (g.cin1 == 32 ? 2 : 3);

    if (threadIdx.x == 0) {
        fail = 0;
        for (int p = 0; p < steps; p++) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(&full[p])), "r"(kConvThreads));
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&done[p])));
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                     "r"(g.tmem_cols));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = *tmem_slot;

    if (warp >= 4 && warp < 8) {
        const int tid = threadIdx.x - kConvThreads;
        // this thread's items of a plane, the same for every plane of a source: where
        // they come from (in 16-byte units of the plane; -1 outside the volume) and
        // where they go
        int from[ITEMS], to[ITEMS];
        auto map = [&](int src) {
            const int lg = src ? lg1 : lg0, chunk = src ? g.chunk1 : g.chunk0, n = kHaloRows << lg;
#pragma unroll
            for (int u = 0; u < ITEMS; u++) {
                const int q = u * kConvThreads + tid;
                from[u] = -1;
                to[u] = -1;
                if (q >= n) continue;
                const int c = q & ((1 << lg) - 1), r = q >> lg, zh = r % kHaloZ, yh = r / kHaloZ;
                const int yy = y0 - 1 + yh, zz = z0 - 1 + zh;
                to[u] = c * chunk + r * 16;
                if ((unsigned)yy < (unsigned)g.NY && (unsigned)zz < (unsigned)g.NZ)
                    from[u] = ((yy * g.NZ + zz) << lg) + c;
            }
        };
        const int64_t plane = (int64_t)g.NY * g.NZ;
        auto stage = [&](int i) {
            const int src = i >= np ? 1 : 0, xx = x0 - 1 + i - src * np;
            if (i == 0 || i == np) map(src);
            const bool in = (unsigned)xx < (unsigned)g.NX;
            const int64_t at = in ? ((int64_t)b * g.NX + xx) * plane : 0;
            const uint4 *sp = reinterpret_cast<const uint4 *>(src ? x1p : x0p) + (at << (src ? lg1 : lg0));
            const uint32_t dst = smem_u32(smem) + (uint32_t)((i % g.ring) * g.slot);
#pragma unroll
            for (int u = 0; u < ITEMS; u++) {
                const bool any = in && from[u] >= 0;
                if (to[u] >= 0) copy16_async(dst + (uint32_t)to[u], sp + (any ? from[u] : 0), any);
            }
        };
        const int ahead = g.ring - 1;
        for (int p = 0; p < ahead; p++) {
            if (p == 0) {
                halo_stage_weights<COUT>(reinterpret_cast<const uint4 *>(w0p), smem_u32(smem + g.w0_off), lg0, tid);
                if (nsrc > 1)
                    halo_stage_weights<COUT>(reinterpret_cast<const uint4 *>(w1p), smem_u32(smem + g.w1_off), lg1, tid);
            }
            if (p < steps) stage(p);
            asm volatile("cp.async.commit_group;" ::: "memory");
        }
        for (int p = 0; p < steps; p++) {
            // step p has landed when at most the ahead - 1 groups after its own are in flight
            if (ahead == 3) asm volatile("cp.async.wait_group 2;" ::: "memory");
            else asm volatile("cp.async.wait_group 1;" ::: "memory");
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(&full[p])) : "memory");
            if (p + ahead < steps) {
                if (p >= 1 && !mbar_wait(smem_u32(&done[p - 1]), 0)) {
                    fail = 1;
                    break;
                }
                stage(p + ahead);
            }
            asm volatile("cp.async.commit_group;" ::: "memory");
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
    } else if (warp < 4) {
        // output plane o, complete with the last source's input plane o + 2: row m of its accumulator is TMEM lane m
        const int m = threadIdx.x;
        float bs[COUT <= 32 ? COUT : 1];
        if (COUT <= 32)
#pragma unroll
            for (int c = 0; c < (COUT <= 32 ? COUT : 1); c++) bs[c] = bias ? __ldg(bias + c) : 0.0f;
        __nv_bfloat16 *yo = y + ((((int64_t)b * g.NX + x0) * g.NY + y0 + (m >> 3)) * g.NZ + z0 + (m & 7)) * COUT;
        for (int o = 0; o < xr; o++, yo += (int64_t)g.NY * g.NZ * COUT) {
            // warp-uniform outcome: tcgen05.ld is a .sync.aligned warp instruction
            if (!__all_sync(0xffffffffu, mbar_wait(smem_u32(&done[steps - np + o + 2]), 0) ? 1 : 0)) {
                fail = 1;
                break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            float acc[COUT];
#pragma unroll
            for (int c = 0; c < COUT; c += 16)
                tmem_ld16(tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)(o * COUT + c), acc + c);
            __align__(16) __nv_bfloat16 out[COUT];
#pragma unroll
            for (int c = 0; c < COUT; c++) {
                float v = acc[c] + (COUT <= 32 ? bs[COUT <= 32 ? c : 0] : (bias ? __ldg(bias + c) : 0.0f));
                if (g.relu) v = fmaxf(v, 0.0f);
                out[c] = __float2bfloat16_rn(v);
            }
            uint4 *dst = reinterpret_cast<uint4 *>(yo);
#pragma unroll
            for (int q = 0; q < COUT / 8; q++) dst[q] = reinterpret_cast<const uint4 *>(out)[q];
        }
    } else {
        const uint32_t lead = elect_one();
        // MMA issuer: per step 9 x (Cin / 16) MMAs of N = 3 Cout, then one commit.  For
        // an output their order is source, dx, (dy, dz), channels, as in the tap-tile
        // kernel, so the two round alike.
        for (int i = 0; i < steps; i++) {
            if (!mbar_wait_warp(smem_u32(&full[i]), 0)) {
                fail = 1;
                break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const int src = i >= np ? 1 : 0, p = i - src * np;
            const uint32_t slot = smem_u32(smem) + (uint32_t)((i % g.ring) * g.slot);
            const int lo = max(0, p - 2), hi = min(p, xr - 1);  // the output planes it contributes to
            const uint32_t d = tmem + (uint32_t)(lo * COUT), idesc = mma_idesc((hi - lo + 1) * COUT);
            const uint32_t wrow = (uint32_t)((lo - (p - 2)) * COUT * 16);
            const int lg = src ? lg1 : lg0, ksteps = 1 << (lg - 1);
            const uint32_t chunk = (uint32_t)(src ? g.chunk1 : g.chunk0);
            const uint64_t a0 = ns_desc(slot, chunk, kHaloZ * 16);
            uint64_t bd = ns_desc(smem_u32(smem + (src ? g.w1_off : g.w0_off)) + wrow, 3 * COUT * 16, 128);
            const uint64_t astep = (uint64_t)((2 * chunk) >> 4);  // in 16-byte units, as the address field
#pragma unroll
            for (int sft = 0; sft < 9; sft++) {
                uint64_t ad = a0 + (uint64_t)((sft / 3) * kHaloZ + sft % 3);
                for (int kk = 0; kk < ksteps; kk++, ad += astep, bd += (uint64_t)(2 * 3 * COUT)) {
                    if (sft == 0 && src == 0 && kk == 0 && p < xr) {
                        // the planes begun before, then the new one from zero
                        if (hi > lo) mma_if(lead, d, ad, bd, mma_idesc((hi - lo) * COUT), 1u);
                        mma_if(lead, tmem + (uint32_t)(p * COUT), ad, bd + (uint64_t)((hi - lo) * COUT),
                               mma_idesc(COUT), 0u);
                    } else {
                        mma_if(lead, d, ad, bd, idesc, 1u);
                    }
                }
            }
            commit_if(lead, smem_u32(&done[i]));
        }
    }
    __syncwarp();
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (fail && threadIdx.x == 0) atomicExch(&g_conv_error, 1);
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(g.tmem_cols));
}

// ---------------------------------------------------------------- weight gradient
//
//   dW[tap][co][ci] = sum over voxels v of X[v + off(tap)][ci] * dY[v][co]
// as a tcgen05 GEMM with the voxels as K:
//   D[m = (slot, ci)][co] += A[m][v] * B[co][v]
// A holds G = 128 / Cin tap-shifted input tiles side by side (a "tap group":
// M = 128 rows = G taps x Cin channels), B the output-gradient tile.  Both are
// the channels-last tiles TMA already writes for the forward pass, read as
// MN-major operands: the channel dimension is contiguous, one swizzle atom
// wide, and the tap tiles of a group are consecutive atoms along M (leading
// byte offset = one tile).  A persistent CTA walks its share of the
// 128-voxel tiles, keeps one FP32 accumulator per tap group in TMEM for its
// whole life, and adds it to dW with one atomic per entry at the end.
// Groups that do not fit in TMEM (512 columns) are split over blockIdx.y.

constexpr int kWgStages = 4;
constexpr int kWgA = 32768;  // G tap tiles of 128 voxels x Cin BF16
constexpr int kWgB = 16384;  // dY tile, 128 voxels x Cout <= 64
constexpr int kWgStage = kWgA + kWgB;
constexpr int kWgSmem = kWgStages * kWgStage + 1024 + 256;
constexpr uint32_t kDoneWaitLimit = 1u << 26;

// MN-major shared-memory descriptor: swizzle width = one row (the channel
// extent), lbo = stride between atoms along M/N, sbo = 8 rows along K.
__device__ __forceinline__ uint64_t sw_desc_mn(uint32_t saddr, int row_bytes, uint32_t lbo) {
    const uint64_t layout = row_bytes == 128 ? 2ull : (row_bytes == 64 ? 4ull : 6ull);
    uint64_t d = 0;
    d |= (uint64_t)((saddr & 0x3FFFFu) >> 4);
    d |= (uint64_t)((lbo >> 4) & 0x3FFFu) << 16;
    d |= (uint64_t)(((8u * row_bytes) >> 4) & 0x3FFFu) << 32;
    d |= (uint64_t)1 << 46;
    d |= layout << 61;
    return d;
}

__device__ __forceinline__ bool mbar_wait_long(uint32_t bar, uint32_t parity) {
    for (uint32_t i = 0; i < kDoneWaitLimit; i++) {
        uint32_t ok;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(ok)
            : "r"(bar), "r"(parity)
            : "memory");
        if (ok) return true;
    }
    return false;
}

template <int CIN, int COUT>
__global__ void __launch_bounds__(kConvThreads, 1)
    k_conv3d_wgrad_tc(const __grid_constant__ CUtensorMap mx, const __grid_constant__ CUtensorMap mdy, const ConvGeom g,
                      int groups_per_slice, int tmem_cols, float *__restrict__ dw) {
    constexpr int G = 128 / CIN;                 // taps per group
    constexpr int NG = (27 + G - 1) / G;         // groups
    constexpr int TILE_A = 128 * CIN * 2;        // one tap tile
    constexpr int TILE_B = 128 * COUT * 2;
    extern __shared__ unsigned char conv_smem_raw[];
    unsigned char *smem = reinterpret_cast<unsigned char *>(
        (reinterpret_cast<uintptr_t>(conv_smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
    uint64_t *full = reinterpret_cast<uint64_t *>(smem + kWgStages * kWgStage);
    uint64_t *empty = full + kWgStages;
    uint64_t *done = empty + kWgStages;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(done + 1);
    __shared__ int fail;

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int tz = g.NZ / g.nzb, ty = g.NY / g.nyb;
    const int ntiles = g.B * g.NX * ty * tz;
    const int my_tiles = blockIdx.x < (unsigned)ntiles ? (ntiles - 1 - (int)blockIdx.x) / (int)gridDim.x + 1 : 0;
    const int gbeg = blockIdx.y * groups_per_slice;
    const int gend = min(NG, gbeg + groups_per_slice);
    const int ng = gend - gbeg;
    const int T = my_tiles * ng;

    if (threadIdx.x == 0) {
        fail = 0;
        for (int s = 0; s < kWgStages; s++) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&full[s])));
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&empty[s])));
        }
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(done)));
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                     "r"(tmem_cols));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = *tmem_slot;

    if (threadIdx.x == 0) {
        for (int it = 0; it < T; it++) {
            const int s = it % kWgStages, u = it / kWgStages;
            if (u > 0 && !mbar_wait(smem_u32(&empty[s]), (u - 1) & 1)) {
                fail = 1;
                break;
            }
            int t = (int)blockIdx.x + (it / ng) * (int)gridDim.x;
            const int grp = gbeg + it % ng;
            const int z0 = (t % tz) * g.nzb;
            t /= tz;
            const int y0 = (t % ty) * g.nyb;
            t /= ty;
            const int x = t % g.NX, b = t / g.NX;
            const int taps = min(G, 27 - grp * G);
            const uint32_t bytes = (uint32_t)(taps * TILE_A + TILE_B);
            const uint32_t fb = smem_u32(&full[s]);
            asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(fb), "r"(bytes) : "memory");
            const uint32_t a = smem_u32(smem + s * kWgStage);
            for (int q = 0; q < taps; q++) {
                const int tap = grp * G + q;
                const int dx = tap / 9 - 1, dy = (tap / 3) % 3 - 1, dz = tap % 3 - 1;
                tma_load_5d(a + q * TILE_A, &mx, 0, z0 + dz, y0 + dy, x + dx, b, fb);
            }
            tma_load_5d(a + kWgA, &mdy, 0, z0, y0, x, b, fb);
        }
    } else if (warp == 1) {
        const uint32_t lead = elect_one();
        const uint32_t idesc = mma_idesc(COUT) | (1u << 15) | (1u << 16);  // A and B MN-major
        for (int it = 0; it < T; it++) {
            const int s = it % kWgStages, u = it / kWgStages;
            if (!mbar_wait_warp(smem_u32(&full[s]), u & 1)) {
                fail = 1;
                break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const int j = it % ng;
            const uint32_t a = smem_u32(smem + s * kWgStage), bb = a + kWgA;
#pragma unroll
            for (int kk = 0; kk < 8; kk++) {  // 16 voxel rows per MMA
                const uint64_t ad = sw_desc_mn(a + kk * 16 * CIN * 2, CIN * 2, TILE_A);
                const uint64_t bd = sw_desc_mn(bb + kk * 16 * COUT * 2, COUT * 2, TILE_B);
                const uint32_t acc = (it >= ng || kk > 0) ? 1u : 0u;
                mma_if(lead, tmem + (uint32_t)(j * COUT), ad, bd, idesc, acc);
            }
            commit_if(lead, smem_u32(&empty[s]));
        }
        commit_if(lead, smem_u32(done));
    }
    __syncwarp();
    const bool got = __all_sync(0xffffffffu, mbar_wait_long(smem_u32(done), 0) ? 1 : 0) != 0;
    if (!got) fail = 1;
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    __syncthreads();  // every thread sees a failure of the producer or the MMA issuer
    if (got && !fail && my_tiles > 0) {
        const int m = warp * 32 + lane;
        const int slot = m / CIN, ci = m % CIN;
        for (int j = 0; j < ng; j++) {
            const int tap = (gbeg + j) * G + slot;
#pragma unroll
            for (int c = 0; c < COUT; c += 16) {
                float v[16];
                tmem_ld16(tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)(j * COUT + c), v);
                if (tap < 27) {
#pragma unroll
                    for (int e = 0; e < 16; e++) atomicAdd(&dw[((int64_t)tap * COUT + c + e) * CIN + ci], v[e]);
                }
            }
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (fail && threadIdx.x == 0) atomicExch(&g_conv_error, 1);
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(tmem_cols));
}

// ---------------------------------------------------------------- halo-plane weight gradient
//
// The same sums for NZ % 8 == 0, NY % 16 == 0, Cin <= 32 and Cout <= 32 from
// haloed input planes staged once, as k_conv3d_halo stages them, instead of 27
// tap-shifted tiles (216 KB of shared memory filled per 128 voxels and 32
// channels: the copies bound k_conv3d_wgrad_tc).
//
// A segment is a 16 (y) x 8 (z) voxel tile at NQ consecutive x planes x0 ..: the
// NQ tiles of dY and the NQ + 2 haloed planes of X, x = x0 - 1 .., side by side in
// shared memory, so that one MMA of M = 128 rows (plane, ci) and N = NQ Cout
// columns (q, co) multiplies 128 / Cin planes with all NQ tiles: of these
// products those with dx = plane - 1 - q in -1 .. 1 are kept, 3 of 4 with Cin = 32
// and NQ = 2, and the others cost nothing that the A operand's reads do not.  Both
// operands are MN-major without swizzle: a core matrix is 8 channels x 8 voxels of
// a z row (128 contiguous bytes), the next along M or N one chunk region on (SBO),
// the next along K one row of voxels on (LBO; padded for X).  The nine shifts (dy,
// dz) are start offsets into the planes, each with its own accumulator in TMEM for
// the CTA's whole life (S of them; blockIdx.y takes the next S).  At the end the
// CTA sums its NQ parts of every tap in shared memory and adds them to dW with one
// atomic per entry.
// Warps 0-7 stage segments through a ring with asynchronous copies, one thread of
// warp 8 issues the MMAs.  4 x 64^3: Cin 32, Cout 16 232 -> 76 us, Cin 16
// 156 -> 61 us; an MMA here takes about 45 cycles, 32 of them the A operand.
constexpr int kWhStagers = 256;
constexpr int kWhThreads = kWhStagers + 32;
constexpr int kWhMaxRing = 4;

template <int CIN, int COUT>
struct WhShape {
    static constexpr int NQ = CIN == 16 ? 3 : 2;               // dY planes of a segment
    static constexpr int S = COUT == 16 ? 9 : 5;               // shifts per CTA: S * NQ * COUT <= 512 columns
    static constexpr int CHUNK = kHaloRows * 16 + (CIN == 32 ? 32 : 0);
    static constexpr int PLANE = CIN / 8 * CHUNK;
    static constexpr int DCHUNK = 128 * 16 + (COUT == 32 ? 32 : 64);
    static constexpr int DPLANE = COUT / 8 * DCHUNK;
    static constexpr int XBYTES = (NQ + 2) * PLANE;
    static constexpr int SEG = (XBYTES + NQ * DPLANE + 127) / 128 * 128;
    // rows beyond the segment's planes are read and never used: room for them after the last buffer
    static constexpr int OVER = 128 / CIN * PLANE > SEG ? 128 / CIN * PLANE - SEG : 0;
    static constexpr int RING = (kHaloSmemMax - 1024 - 256 - OVER) / SEG < kWhMaxRing
                                    ? (kHaloSmemMax - 1024 - 256 - OVER) / SEG : kWhMaxRing;
    static constexpr int BARS = (RING * SEG + OVER + 15) / 16 * 16;
    static constexpr int SMEM = BARS + 128 + 1024;
    static_assert(27 * CIN * COUT * 4 <= RING * SEG, "the sums reuse the ring");
    static_assert(S * NQ * COUT <= 512 && RING >= 2, "");
};

template <int CIN, int COUT>
__global__ void __launch_bounds__(kWhThreads, 1)
    k_conv3d_wgrad_halo(const __nv_bfloat16 *__restrict__ xp, const __nv_bfloat16 *__restrict__ dyp, int B, int NX,
                        int NY, int NZ, float *__restrict__ dw) {
    using W = WhShape<CIN, COUT>;
    constexpr int NQ = W::NQ, C8 = CIN / 8, D8 = COUT / 8;
    extern __shared__ unsigned char conv_smem_raw[];
    unsigned char *smem = reinterpret_cast<unsigned char *>(
        (reinterpret_cast<uintptr_t>(conv_smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
    uint64_t *full = reinterpret_cast<uint64_t *>(smem + W::BARS);
    uint64_t *empty = full + kWhMaxRing;
    uint64_t *done = empty + kWhMaxRing;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(done + 1);
    __shared__ int fail;

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int tz = NZ >> 3, ty = NY >> 4, tx = (NX + NQ - 1) / NQ;
    const int nseg = B * tx * ty * tz;
    const int mine = blockIdx.x < (unsigned)nseg ? (nseg - 1 - (int)blockIdx.x) / (int)gridDim.x + 1 : 0;
    const int s0 = blockIdx.y * W::S, ns = min(9 - s0, W::S);
    // segment i of this CTA
    auto where = [&](int i, int &b, int &x0, int &y0, int &z0) {
        int t = (int)blockIdx.x + i * (int)gridDim.x;
        z0 = (t % tz) * 8;
        t /= tz;
        y0 = (t % ty) * 16;
        t /= ty;
        x0 = (t % tx) * NQ;
        b = t / tx;
    };
    if (threadIdx.x == 0) {
        fail = 0;
        for (int r = 0; r < W::RING; r++) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(&full[r])), "r"(kWhStagers));
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&empty[r])));
        }
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(done)));
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(smem_u32(tmem_slot)));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = *tmem_slot;

    if (warp < 8) {
        constexpr int IX = (kHaloRows * C8 + kWhStagers - 1) / kWhStagers;  // items of an X plane per thread
        constexpr int ID = 128 * D8 / kWhStagers > 0 ? 128 * D8 / kWhStagers : 1;
        const uint4 *gx = reinterpret_cast<const uint4 *>(xp), *gd = reinterpret_cast<const uint4 *>(dyp);
        const int64_t plane = (int64_t)NY * NZ;
        const uint32_t base = smem_u32(smem);
        auto stage = [&](int i) {
            int b, x0, y0, z0;
            where(i, b, x0, y0, z0);
            const int nq = min(NQ, NX - x0);
            const uint32_t buf = base + (uint32_t)((i % W::RING) * W::SEG);
#pragma unroll
            for (int u = 0; u < IX; u++) {
                const int q = u * kWhStagers + threadIdx.x;
                if (q >= kHaloRows * C8) break;
                const int c = q % C8, r = q / C8, zh = r % kHaloZ, yh = r / kHaloZ;
                const int yy = y0 - 1 + yh, zz = z0 - 1 + zh;
                const bool in = (unsigned)yy < (unsigned)NY && (unsigned)zz < (unsigned)NZ;
                const int from = in ? (yy * NZ + zz) * C8 + c : 0;
                const uint32_t to = buf + (uint32_t)(c * W::CHUNK + r * 16);
#pragma unroll
                for (int pl = 0; pl < NQ + 2; pl++) {
                    const int xx = x0 - 1 + pl;
                    if (pl >= nq + 2) break;
                    const bool ok = in && (unsigned)xx < (unsigned)NX;
                    copy16_async(to + (uint32_t)(pl * W::PLANE), gx + (ok ? ((int64_t)b * NX + xx) * plane * C8 + from : 0),
                                 ok);
                }
            }
#pragma unroll
            for (int u = 0; u < ID; u++) {
                const int q = u * kWhStagers + threadIdx.x;
                if (q >= 128 * D8) break;
                const int c = q % D8, v = q / D8;
                const int from = ((y0 + (v >> 3)) * NZ + z0 + (v & 7)) * D8 + c;
                const uint32_t to = buf + (uint32_t)(W::XBYTES + c * W::DCHUNK + v * 16);
#pragma unroll
                for (int t = 0; t < NQ; t++) {
                    if (t >= nq) break;
                    copy16_async(to + (uint32_t)(t * W::DPLANE),
                                 gd + ((int64_t)b * NX + x0 + t) * plane * D8 + from, true);
                }
            }
        };
        constexpr int ahead = W::RING - 1;
        for (int i = 0; i < ahead; i++) {
            if (i < mine) stage(i);
            asm volatile("cp.async.commit_group;" ::: "memory");
        }
        for (int i = 0; i < mine; i++) {
            // segment i has landed when at most the ahead - 1 groups after its own are in flight
            asm volatile("cp.async.wait_group %0;" ::"n"(ahead - 1) : "memory");
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(&full[i % W::RING])) : "memory");
            const int n = i + ahead;
            if (n < mine) {
                // its buffer was segment n - RING's
                if (n >= W::RING &&
                    !mbar_wait(smem_u32(&empty[n % W::RING]), (uint32_t)((n / W::RING - 1) & 1))) {
                    fail = 1;
                    break;
                }
                stage(n);
            }
            asm volatile("cp.async.commit_group;" ::: "memory");
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
    } else {
        const uint32_t lead = elect_one();
        const uint32_t mn = (1u << 15) | (1u << 16);  // A and B MN-major
        int init = 0;                                  // dY planes whose accumulators hold something
        for (int i = 0; i < mine; i++) {
            if (!mbar_wait_warp(smem_u32(&full[i % W::RING]), (uint32_t)((i / W::RING) & 1))) {
                fail = 1;
                break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            int b, x0, y0, z0;
            where(i, b, x0, y0, z0);
            const int nq = min(NQ, NX - x0);
            const uint32_t buf = smem_u32(smem) + (uint32_t)((i % W::RING) * W::SEG);
            const uint64_t a0 = ns_desc(buf, kHaloZ * 16, W::CHUNK), b0 = ns_desc(buf + W::XBYTES, 128, W::DCHUNK);
            auto mma = [&](uint32_t d, uint64_t aa, uint64_t bb, int n, uint32_t acc) {
                mma_if(lead, d, aa, bb, mma_idesc(n) | mn, acc);
            };
            // shifts inside: successive MMAs add to different accumulators
            for (int kk = 0; kk < 8; kk++) {  // two rows of 8 voxels per MMA
                const uint64_t ak = a0 + (uint64_t)(kk * 2 * kHaloZ), bd = b0 + (uint64_t)(kk * 16);
#pragma unroll
                for (int sl = 0; sl < W::S; sl++) {
                    if (sl >= ns) break;
                    const int sft = s0 + sl;
                    const uint32_t d = tmem + (uint32_t)(sl * NQ * COUT);
                    const uint64_t ad = ak + (uint64_t)((sft / 3) * kHaloZ + sft % 3);
                    if (kk == 0 && nq > init) {
                        if (init > 0) mma(d, ad, bd, init * COUT, 1u);
                        mma(d + (uint32_t)(init * COUT), ad, bd + (uint64_t)(init * (W::DPLANE >> 4)), (nq - init) * COUT,
                            0u);
                    } else {
                        mma(d, ad, bd, nq * COUT, 1u);
                    }
                }
            }
            init = max(init, nq);
            commit_if(lead, smem_u32(&empty[i % W::RING]));
        }
        commit_if(lead, smem_u32(done));
    }
    __syncwarp();
    const bool got = __all_sync(0xffffffffu, mbar_wait_long(smem_u32(done), 0) ? 1 : 0) != 0;
    if (!got) fail = 1;
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    __syncthreads();  // every thread sees a failure; nothing reads the ring any more
    if (!fail && mine > 0) {
        // the dY planes that this CTA had at all
        int init = 0;
        for (int i = 0; i < mine && init < NQ; i++) {
            int b, x0, y0, z0;
            where(i, b, x0, y0, z0);
            init = max(init, min(NQ, NX - x0));
        }
        constexpr int entries = 27 * COUT * CIN;
        float *sum = reinterpret_cast<float *>(smem);
        for (int q = threadIdx.x; q < entries; q += kWhThreads) sum[q] = 0.0f;
        __syncthreads();
        for (int t = 0; t < init; t++) {
            if (warp < 4) {
                const int m = threadIdx.x, ci = m % CIN, dx = m / CIN - 1 - t;
                const bool use = dx >= -1 && dx <= 1;
                if (__any_sync(0xffffffffu, use))
                    for (int sl = 0; sl < ns; sl++)
#pragma unroll
                        for (int c = 0; c < COUT; c += 16) {
                            float v[16];
                            tmem_ld16(tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)((sl * NQ + t) * COUT + c), v);
                            if (use) {
                                float *at = sum + (((dx + 1) * 9 + s0 + sl) * COUT + c) * CIN + ci;
#pragma unroll
                                for (int e = 0; e < 16; e++) at[e * CIN] += v[e];
                            }
                        }
            }
            __syncthreads();  // the next plane's parts go to the same taps from other threads
        }
        for (int q = threadIdx.x; q < entries; q += kWhThreads) {
            const int sft = (q / (COUT * CIN)) % 9;
            if (sft >= s0 && sft < s0 + ns) atomicAdd(dw + q, sum[q]);
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (fail && threadIdx.x == 0) atomicExch(&g_conv_error, 1);
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem));
}

// ---------------------------------------------------------------- host side

static PFN_cuTensorMapEncodeTiled_v12000 g_encode = nullptr;
static std::mutex g_encode_mutex;

static int get_encode() {
    std::lock_guard<std::mutex> lock(g_encode_mutex);
    if (g_encode) return FLUB_OK;
    void *fn = nullptr;
    cudaDriverEntryPointQueryResult q;
    cudaError_t e = cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &fn, 12000, cudaEnableDefault, &q);
    if (e != cudaSuccess || q != cudaDriverEntryPointSuccess || !fn) {
        set_last_error("cuTensorMapEncodeTiled not available: %s", cudaGetErrorString(e));
        cudaGetLastError();
        return FLUB_ERR_CUDA;
    }
    g_encode = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(fn);
    return FLUB_OK;
}

static CUtensorMapSwizzle swizzle_for(int row_bytes) {
    return row_bytes == 128 ? CU_TENSOR_MAP_SWIZZLE_128B
                            : (row_bytes == 64 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_32B);
}

// Activation map: dims (C, Z, Y, X, B), box (C, nzb, nyb, 1, 1).
static int make_act_map(CUtensorMap *m, const void *x, int C, const ConvGeom &g) {
    const cuuint64_t dims[5] = {(cuuint64_t)C, (cuuint64_t)g.NZ, (cuuint64_t)g.NY, (cuuint64_t)g.NX, (cuuint64_t)g.B};
    const cuuint64_t es = 2;
    const cuuint64_t strides[4] = {C * es, (cuuint64_t)g.NZ * C * es, (cuuint64_t)g.NY * g.NZ * C * es,
                                   (cuuint64_t)g.NX * g.NY * g.NZ * C * es};
    const cuuint32_t box[5] = {(cuuint32_t)C, (cuuint32_t)g.nzb, (cuuint32_t)g.nyb, 1, 1};
    const cuuint32_t estr[5] = {1, 1, 1, 1, 1};
    CUresult r = g_encode(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 5, const_cast<void *>(x), dims, strides, box, estr,
                          CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle_for(C * 2), CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                          CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) {
        set_last_error("cuTensorMapEncodeTiled(activations, C=%d) failed: %d", C, (int)r);
        return FLUB_ERR_CUDA;
    }
    return FLUB_OK;
}

// Weight map: [27 * Cout rows][Cin], box (Cin, Cout).
static int make_w_map(CUtensorMap *m, const void *w, int cin, int cout) {
    const cuuint64_t dims[2] = {(cuuint64_t)cin, (cuuint64_t)27 * cout};
    const cuuint64_t strides[1] = {(cuuint64_t)cin * 2};
    const cuuint32_t box[2] = {(cuuint32_t)cin, (cuuint32_t)cout};
    const cuuint32_t estr[2] = {1, 1};
    CUresult r = g_encode(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void *>(w), dims, strides, box, estr,
                          CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle_for(cin * 2), CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                          CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) {
        set_last_error("cuTensorMapEncodeTiled(weights, Cin=%d, Cout=%d) failed: %d", cin, cout, (int)r);
        return FLUB_ERR_CUDA;
    }
    return FLUB_OK;
}

template <int COUT>
static int launch_conv(const CUtensorMap &mx0, const CUtensorMap &mw0, const CUtensorMap &mx1, const CUtensorMap &mw1,
                       const ConvGeom &g, const float *bias, __nv_bfloat16 *y, cudaStream_t s) {
    static bool attr_set = false;
    if (!attr_set) {
        FLUB_CHECK_CUDA(cudaFuncSetAttribute(k_conv3d_tc<COUT>, cudaFuncAttributeMaxDynamicSharedMemorySize, kConvSmem));
        attr_set = true;
    }
    const unsigned tiles = (unsigned)((int64_t)g.B * g.NX * (g.NY / g.nyb) * (g.NZ / g.nzb));
    // shared memory sized for this layer's channels: the 16- and 32-channel
    // layers fit several CTAs per SM, whose pipelines then overlap
    const size_t smem = (size_t)kConvStages * g.stage_bytes + 1024 + 256;
    k_conv3d_tc<COUT><<<tiles, kConvThreads, smem, s>>>(mx0, mw0, mx1, mw1, g, bias, y);
    FLUB_CHECK_LAUNCH();
    return FLUB_OK;
}

static bool aligned16(const void *p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

static inline int align_up(int v, int a) { return (v + a - 1) / a * a; }

// Shared-memory layout of k_conv3d_halo; returns the dynamic shared memory size
// (including the 1 KB alignment slack).
static size_t halo_layout(HaloGeom &h, int cout) {
    // chunk regions start at different 16-byte columns of the banks, so that the
    // lanes that stage one voxel's chunks do not collide
    auto chunk = [](int cin) { return kHaloRows * 16 + (cin == 32 ? 32 : (cin == 64 ? 16 : 0)); };
    h.chunk0 = chunk(h.cin0);
    h.chunk1 = chunk(h.cin1);
    const int plane0 = (h.cin0 >> 3) * h.chunk0, plane1 = (h.cin1 >> 3) * h.chunk1;
    h.slot = align_up(plane0 > plane1 ? plane0 : plane1, 128);
    h.w0_off = h.ring * h.slot;
    h.w1_off = h.w0_off + 27 * cout * h.cin0 * 2;
    h.bar_off = align_up(h.w1_off + 27 * cout * h.cin1 * 2, 16);
    uint32_t cols = 32;
    while (cols < (uint32_t)(h.xr * cout)) cols <<= 1;
    h.tmem_cols = cols;
    return (size_t)h.bar_off + kHaloBars + 16 /* TMEM slot */ + 1024;
}

static bool halo_enabled() {
    const char *e = getenv("FLUB_CONV_HALO");
    return !(e && e[0] == '0');
}

// FLUB_CONV_XR=n forces n planes per CTA (1 to 16, at most NX) where it fits.
static int forced_xr() {
    const char *e = getenv("FLUB_CONV_XR");
    return e ? atoi(e) : 0;
}

// Chooses the planes per CTA and the ring of k_conv3d_halo; returns 0 when the
// layer goes to k_conv3d_tc instead: its weights do not fit beside the planes,
// or k_conv3d_tc takes its shape and there are fewer tiles than SMs (16^3),
// where the staging is not hidden and the tap-tile kernel measured faster.
// The CTAs on an SM share its tensor core, and each has its xr + 2 planes and
// about one more for its start; one that has no other beside it waits for its
// loads in half of that again.  So the shortest is the least CTAs per SM x
// (xr + 3), half as much again without overlap.
static size_t halo_plan(HaloGeom &h, int cout) {
    if (h.NZ % 8 || h.NY % 16) return 0;
    const int64_t tiles = (int64_t)h.B * (h.NY / 16) * (h.NZ / 8);
    // before anything else what rules the layer out: this runs on every call
    h.xr = 1;
    h.ring = 3;
    if (halo_layout(h, cout) > (size_t)kHaloSmemMax || !halo_enabled()) return 0;
    const int forced = forced_xr(), fx = forced < h.NX ? forced : h.NX;
    const int nzb = h.NZ < 128 ? h.NZ : 128;
    const bool tap_ok = 128 % nzb == 0 && h.NZ % nzb == 0 && h.NY % (128 / nzb) == 0;
    if (!fx && tap_ok && tiles * h.NX < kNumSMs) return 0;
    h.ring = 4;
    size_t smem = halo_layout(h, cout);  // of any xr
    if (smem > (size_t)kHaloSmemMax) {
        h.ring = 3;
        smem = halo_layout(h, cout);
    }
    const int fit = (int)((size_t)(228 * 1024) / (smem + 1024));
    const int regs = cout == 64 || h.cin0 == 64 || h.cin1 == 64 ? 2 : 3;  // as the kernel's launch bounds
    int best = 0;
    int64_t best_cost = 0;
    const int top = 256 / cout < kHaloMaxX ? 256 / cout : kHaloMaxX;
    for (int xr = top < h.NX ? top : h.NX; xr >= 1; xr--) {
        if (fx && xr != fx) continue;
        int cols = 32;
        while (cols < xr * cout) cols <<= 1;
        int occ = fit < regs ? fit : regs;
        occ = occ < 512 / cols ? occ : 512 / cols;
        const int64_t ctas = tiles * ((h.NX + xr - 1) / xr), per_sm = (ctas + kNumSMs - 1) / kNumSMs;
        const int64_t cost = per_sm * (xr + 3) * (occ == 1 || per_sm == 1 ? 3 : 2);
        if (!best || cost < best_cost) {
            best = xr;
            best_cost = cost;
        }
    }
    if (!best) return 0;
    h.xr = best;
    return halo_layout(h, cout);
}

template <int COUT, int ITEMS>
static int launch_halo(const void *x0, const void *w0, const void *x1, const void *w1, const HaloGeom &h, size_t smem,
                       const float *bias, __nv_bfloat16 *y, cudaStream_t s) {
    static size_t attr_smem = 0;  // largest dynamic shared memory enabled so far
    if (smem > attr_smem) {
        FLUB_CHECK_CUDA(
            cudaFuncSetAttribute(k_conv3d_halo<COUT, ITEMS>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        attr_smem = smem;
    }
    const unsigned ctas = (unsigned)((int64_t)h.B * ((h.NX + h.xr - 1) / h.xr) * (h.NY / 16) * (h.NZ / 8));
    k_conv3d_halo<COUT, ITEMS><<<ctas, kHaloThreads, smem, s>>>(
        static_cast<const __nv_bfloat16 *>(x0), static_cast<const __nv_bfloat16 *>(w0),
        static_cast<const __nv_bfloat16 *>(x1 ? x1 : x0), static_cast<const __nv_bfloat16 *>(w1 ? w1 : w0), h, bias,
        y);
    FLUB_CHECK_LAUNCH();
    return FLUB_OK;
}

template <int COUT>
static int launch_halo_items(const void *x0, const void *w0, const void *x1, const void *w1, const HaloGeom &h,
                             size_t smem, const float *bias, __nv_bfloat16 *y, cudaStream_t s) {
    const int cin = h.cin0 > h.cin1 ? h.cin0 : h.cin1;
    if (cin == 16) return launch_halo<COUT, 3>(x0, w0, x1, w1, h, smem, bias, y, s);
    if (cin == 32) return launch_halo<COUT, 6>(x0, w0, x1, w1, h, smem, bias, y, s);
    return launch_halo<COUT, 12>(x0, w0, x1, w1, h, smem, bias, y, s);
}

}  // namespace flub

using namespace flub;

extern "C" int flub_conv3d_bf16(const void *x0, int cin0, const void *w0, const void *x1, int cin1, const void *w1,
                                const float *bias, void *y, int cout, int B, int NX, int NY, int NZ, int relu,
                                void *stream) {
    auto okc = [](int c) { return c == 16 || c == 32 || c == 64; };
    FLUB_REQUIRE(x0 && w0 && y, "flub_conv3d_bf16: NULL argument");
    FLUB_REQUIRE(okc(cin0) && okc(cout) && (x1 == nullptr ? cin1 == 0 : (okc(cin1) && w1 != nullptr)),
                 "flub_conv3d_bf16: channels must be 16, 32 or 64 (cin0=%d cin1=%d cout=%d)", cin0, cin1, cout);
    FLUB_REQUIRE(B > 0 && NX > 0 && NY > 0 && NZ > 0, "flub_conv3d_bf16: bad shape");
    FLUB_REQUIRE(aligned16(x0) && aligned16(w0) && aligned16(y) && (!x1 || (aligned16(x1) && aligned16(w1))),
                 "flub_conv3d_bf16: pointers must be 16-byte aligned");
    int st = get_encode();
    if (st) return st;
    {
        HaloGeom h;
        memset(&h, 0, sizeof(h));
        h.B = B; h.NX = NX; h.NY = NY; h.NZ = NZ;
        h.cin0 = cin0;
        h.cin1 = x1 ? cin1 : 0;
        h.relu = relu ? 1 : 0;
        const size_t smem = halo_plan(h, cout);
        if (smem) {
            cudaStream_t s = as_stream(stream);
            __nv_bfloat16 *yo = static_cast<__nv_bfloat16 *>(y);
            switch (cout) {
            case 16: return launch_halo_items<16>(x0, w0, x1, w1, h, smem, bias, yo, s);
            case 32: return launch_halo_items<32>(x0, w0, x1, w1, h, smem, bias, yo, s);
            default: return launch_halo_items<64>(x0, w0, x1, w1, h, smem, bias, yo, s);
            }
        }
    }
    ConvGeom g;
    g.B = B; g.NX = NX; g.NY = NY; g.NZ = NZ;
    g.nzb = NZ < 128 ? NZ : 128;
    FLUB_REQUIRE(128 % g.nzb == 0 && NZ % g.nzb == 0, "flub_conv3d_bf16: NZ=%d must divide 128 or be a multiple of 128",
                 NZ);
    g.nyb = 128 / g.nzb;
    FLUB_REQUIRE(NY % g.nyb == 0, "flub_conv3d_bf16: NY=%d must be a multiple of %d", NY, g.nyb);
    g.cout = cout;
    g.cin0 = cin0;
    g.cin1 = x1 ? cin1 : 0;
    g.relu = relu ? 1 : 0;
    {
        const int cmax = g.cin1 > g.cin0 ? g.cin1 : g.cin0;
        g.a_bytes = 128 * cmax * 2;
        g.stage_bytes = (g.a_bytes + cout * cmax * 2 + 1023) & ~1023;
    }
    CUtensorMap mx0, mw0, mx1, mw1;
    if ((st = make_act_map(&mx0, x0, cin0, g)) || (st = make_w_map(&mw0, w0, cin0, cout))) return st;
    if (x1) {
        if ((st = make_act_map(&mx1, x1, cin1, g)) || (st = make_w_map(&mw1, w1, cin1, cout))) return st;
    } else {
        mx1 = mx0;
        mw1 = mw0;
    }
    cudaStream_t s = as_stream(stream);
    __nv_bfloat16 *yo = static_cast<__nv_bfloat16 *>(y);
    switch (cout) {
    case 16: return launch_conv<16>(mx0, mw0, mx1, mw1, g, bias, yo, s);
    case 32: return launch_conv<32>(mx0, mw0, mx1, mw1, g, bias, yo, s);
    default: return launch_conv<64>(mx0, mw0, mx1, mw1, g, bias, yo, s);
    }
}

namespace flub {
int launch_bias_grad(const void *dy, int cout, int64_t nvox, float *db, cudaStream_t s);

template <int CIN, int COUT>
static int launch_wgrad(const CUtensorMap &mx, const CUtensorMap &mdy, const ConvGeom &g, float *dw, cudaStream_t s) {
    static bool attr_set = false;
    if (!attr_set) {
        FLUB_CHECK_CUDA(
            cudaFuncSetAttribute(k_conv3d_wgrad_tc<CIN, COUT>, cudaFuncAttributeMaxDynamicSharedMemorySize, kWgSmem));
        attr_set = true;
    }
    constexpr int G = 128 / CIN, NG = (27 + G - 1) / G;
    const int per = NG * COUT <= 512 ? NG : 512 / COUT;
    const int slices = (NG + per - 1) / per;
    int cols = 32;
    while (cols < per * COUT) cols <<= 1;
    int dev = 0, sms = kNumSMs;
    FLUB_CHECK_CUDA(cudaGetDevice(&dev));
    FLUB_CHECK_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    const int64_t ntiles = (int64_t)g.B * g.NX * (g.NY / g.nyb) * (g.NZ / g.nzb);
    const unsigned gx = (unsigned)(ntiles < sms ? ntiles : sms);
    k_conv3d_wgrad_tc<CIN, COUT><<<dim3(gx, slices), kConvThreads, kWgSmem, s>>>(mx, mdy, g, per, cols, dw);
    FLUB_CHECK_LAUNCH();
    return FLUB_OK;
}

// k_conv3d_wgrad_halo where it takes the shape and its channels.
template <int CIN, int COUT>
static int launch_wgrad_halo(const void *x, const void *dy, int B, int NX, int NY, int NZ, float *dw, cudaStream_t s) {
    using W = WhShape<CIN, COUT>;
    static bool attr_set = false;
    if (!attr_set) {
        FLUB_CHECK_CUDA(
            cudaFuncSetAttribute(k_conv3d_wgrad_halo<CIN, COUT>, cudaFuncAttributeMaxDynamicSharedMemorySize, W::SMEM));
        attr_set = true;
    }
    const int64_t nseg = (int64_t)B * ((NX + W::NQ - 1) / W::NQ) * (NY / 16) * (NZ / 8);
    const int slices = (9 + W::S - 1) / W::S, sms = kNumSMs / slices;
    const unsigned gx = (unsigned)(nseg < sms ? nseg : sms);
    k_conv3d_wgrad_halo<CIN, COUT><<<dim3(gx, slices), kWhThreads, W::SMEM, s>>>(
        static_cast<const __nv_bfloat16 *>(x), static_cast<const __nv_bfloat16 *>(dy), B, NX, NY, NZ, dw);
    FLUB_CHECK_LAUNCH();
    return FLUB_OK;
}
}  // namespace flub

extern "C" int flub_conv3d_wgrad(const void *x, int cin, const void *dy, int cout, float *dw, float *db, int B, int NX,
                                 int NY, int NZ, void *stream) {
    auto okc = [](int c) { return c == 16 || c == 32 || c == 64; };
    FLUB_REQUIRE(x && dy && dw, "flub_conv3d_wgrad: NULL argument");
    FLUB_REQUIRE(okc(cin) && okc(cout), "flub_conv3d_wgrad: channels must be 16, 32 or 64 (cin=%d cout=%d)", cin, cout);
    FLUB_REQUIRE(B > 0 && NX > 0 && NY > 0 && NZ > 0, "flub_conv3d_wgrad: bad shape");
    FLUB_REQUIRE(aligned16(x) && aligned16(dy), "flub_conv3d_wgrad: pointers must be 16-byte aligned");
    ConvGeom g;
    g.B = B; g.NX = NX; g.NY = NY; g.NZ = NZ;
    g.a_bytes = g.stage_bytes = 0;  // the forward kernel's stage layout; unused here
    g.nzb = NZ < 128 ? NZ : 128;
    FLUB_REQUIRE(128 % g.nzb == 0 && NZ % g.nzb == 0, "flub_conv3d_wgrad: NZ=%d must divide 128 or be a multiple of 128",
                 NZ);
    g.nyb = 128 / g.nzb;
    FLUB_REQUIRE(NY % g.nyb == 0, "flub_conv3d_wgrad: NY=%d must be a multiple of %d", NY, g.nyb);
    g.cout = cout;
    g.cin0 = cin;
    g.cin1 = 0;
    g.relu = 0;
    cudaStream_t s = as_stream(stream);
    // from two waves of tiles: below, at 32^3, the sums at the end weigh more than
    // the tap tiles' copies (1 x 32^3, 16 -> 32: 19 us against 15; 4 x: 27 and 29).
    // FLUB_CONV_XR forces the halo kernel wherever it fits.
    if (cin <= 32 && cout <= 32 && NZ % 8 == 0 && NY % 16 == 0 && halo_enabled() &&
        (forced_xr() || (int64_t)B * NX * (NY / 16) * (NZ / 8) >= 4 * kNumSMs)) {
        int st = FLUB_OK;
#define FLUB_WGH(CI, CO) \
    if (cin == CI && cout == CO) st = launch_wgrad_halo<CI, CO>(x, dy, B, NX, NY, NZ, dw, s);
        FLUB_WGH(16, 16) FLUB_WGH(16, 32) FLUB_WGH(32, 16) FLUB_WGH(32, 32)
#undef FLUB_WGH
        if (st) return st;
        if (db) return launch_bias_grad(dy, cout, (int64_t)B * NX * NY * NZ, db, s);
        return FLUB_OK;
    }
    int st = get_encode();
    if (st) return st;
    CUtensorMap mx, mdy;
    if ((st = make_act_map(&mx, x, cin, g)) || (st = make_act_map(&mdy, dy, cout, g))) return st;
#define FLUB_WG(CI, CO) \
    if (cin == CI && cout == CO) st = launch_wgrad<CI, CO>(mx, mdy, g, dw, s);
    FLUB_WG(16, 16) FLUB_WG(16, 32) FLUB_WG(16, 64)
    FLUB_WG(32, 16) FLUB_WG(32, 32) FLUB_WG(32, 64)
    FLUB_WG(64, 16) FLUB_WG(64, 32) FLUB_WG(64, 64)
#undef FLUB_WG
    if (st) return st;
    if (db) return launch_bias_grad(dy, cout, (int64_t)B * NX * NY * NZ, db, s);
    return FLUB_OK;
}

extern "C" int flub_conv_error(int *out, int reset) {
    FLUB_REQUIRE(out, "flub_conv_error: NULL argument");
    FLUB_CHECK_CUDA(cudaMemcpyFromSymbol(out, g_conv_error, sizeof(int)));
    if (reset) {
        const int z = 0;
        FLUB_CHECK_CUDA(cudaMemcpyToSymbol(g_conv_error, &z, sizeof(int)));
    }
    return FLUB_OK;
}
