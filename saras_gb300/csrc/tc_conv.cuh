// tc_conv.cuh -- 3x3x3 convolution as an implicit GEMM on the 5th-generation
// tensor cores (tcgen05), BF16 operands, FP32 accumulation in tensor memory.
//
// GEMM view (channels-last activations X[z][y][x][C]):
//   out[m][n] = sum_k A[m][k] * B[n][k],   m = output voxel, n = output channel,
//   k = (tap, input channel), 27 taps, input channels in chunks of 16.
// One CTA (4 warps) owns 128 consecutive positions (M = 128) of lines of W voxels with
// one empty position before each, and all N output channels.  A stage is one (dz, dy) of
// the taps: the 130 positions that the tile's three dx taps read, all input channels,
// each once (cp.async; zero at the empty positions and outside the domain), and the
// three taps' packed weights.  Shared memory holds a plane of 16-byte rows per 8
// channels, a row a position: the canonical K-major layout without swizzle with
// M-adjacent core matrices (8 rows, 128 bytes) 128 B apart and K-adjacent ones a plane
// apart, so a tap's A tile is the stage's rows from dx on, and its 128 rows are three
// overlapping views of one copy: 25 us for 16 -> 16 channels on 65^3 voxels, 87 for 48 ->
// 16, where gathering each tap's tile by itself, three times the loads, took 40 and 121.
// The descriptors are formed once (forming two in the loop cost the issuing thread 98 to
// 175 clocks an MMA, 47 with sums; the SM takes one in 39).  The nine stages go round a ring of four (two when
// they are too large for that): a stage's 3 x chunks tcgen05.mma (K = 16), in the taps'
// order, overlap the loads of the next ones; tcgen05.commit arrives on a per-stage
// mbarrier that releases the stage for reuse.  The accumulator (128 lanes x N FP32
// columns) is read back with tcgen05.ld: warp w reads lanes 32w..32w+31, i.e. thread t
// of the CTA reads the N channels of position t, matching channels-last storage.
//
// Every mbarrier wait is bounded; on timeout the kernel raises an error flag,
// drains its own cp.async groups, frees its tensor memory and returns.
#pragma once

#include <cuda_bf16.h>
#include <cstdint>

#include "tma.cuh"

namespace saras {

__device__ __forceinline__ void cp_async16(uint32_t dst, const void *src, int src_bytes) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(dst), "l"(src), "r"(src_bytes) : "memory");
}
// The same through L1: neighbouring taps read the same lines.
__device__ __forceinline__ void cp_async16_l1(uint32_t dst, const void *src, int src_bytes) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 16, %2;\n" ::"r"(dst), "l"(src), "r"(src_bytes) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory"); }

__device__ __forceinline__ void tmem_alloc(uint32_t *slot, uint32_t ncols) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(su32(slot)), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tmem_relinquish() { asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory"); }
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(taddr), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory"); }

__device__ __forceinline__ void tc_mma_bf16(uint32_t dtmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(dtmem),
        "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}
__device__ __forceinline__ void tc_commit(uint64_t *m) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(su32(m)) : "memory");
}
// 32 lanes x 16 consecutive 32-bit columns per warp.
__device__ __forceinline__ void tc_ld16(uint32_t taddr, float (&v)[16]) {
    uint32_t r[16];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];\n"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]),
          "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr)
        : "memory");
    asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
#pragma unroll
    for (int q = 0; q < 16; ++q) v[q] = __uint_as_float(r[q]);
}

// Shared-memory matrix descriptor: start address, leading / stride byte
// offsets (all >> 4), descriptor version 1, no swizzle.
__device__ __forceinline__ uint64_t smem_desc(uint32_t saddr, uint32_t lbo, uint32_t sbo) {
    uint64_t d = 0;
    d |= (uint64_t)((saddr >> 4) & 0x3FFFu);
    d |= (uint64_t)((lbo >> 4) & 0x3FFFu) << 16;
    d |= (uint64_t)((sbo >> 4) & 0x3FFFu) << 32;
    d |= (uint64_t)1 << 46;
    return d;
}
// Instruction descriptor of kind::f16: FP32 accumulator, BF16 A and B, both
// K-major, N >> 3 at bit 17, M >> 4 at bit 24.
__host__ __device__ constexpr uint32_t idesc_bf16(int M, int N) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}

struct ConvArgs {
    const __nv_bfloat16 *in0, *in1;   // channels-last inputs (concatenated along C)
    int c0, c1;                       // their channel counts (multiples of 16; c1 may be 0)
    const __nv_bfloat16 *wpk;         // packed weights, one N x 16 tile per K step
    const float *bias;                // N, or null
    __nv_bfloat16 *out0, *out1;       // BF16 outputs: channels [0, split) and [split, N)
    int split;
    float *out32;                     // FP32 output of channel 0 only (final layer), or null
    const __nv_bfloat16 *mask0, *mask1;  // zero the output where the mask is <= 0 (ReLU backward)
    int relu;
    int D, H, W;
    int nvox;
    int *err;
};

constexpr int kConvRows = 130, kConvPlane = 136 * 16;   // rows of a stage; bytes of an 8-channel plane
__host__ __device__ constexpr int conv_stage_bytes(int N, int nch) { return 2 * nch * kConvPlane + 3 * nch * N * 32; }
template <int N>
__host__ __device__ constexpr uint32_t conv_tmem_cols() { return N <= 32 ? 32u : N <= 64 ? 64u : 128u; }

// Faces a voxel lies on (x low, x high, y low, y high, z low, z high; bit 6: no
// voxel), and the faces a tap's neighbour would cross: the neighbour exists when the
// two sets share no bit.
__device__ __forceinline__ int conv_faces(int x, int y, int z, int W, int H, int D) {
    return (x == 0) | (x == W - 1) << 1 | (y == 0) << 2 | (y == H - 1) << 3 | (z == 0) << 4 | (z == D - 1) << 5;
}
__device__ __forceinline__ int conv_crosses(int tap) {
    const int dz = tap / 9 - 1, dy = (tap / 3) % 3 - 1, dx = tap % 3 - 1;
    return 64 | (dx < 0) | (dx > 0) << 1 | (dy < 0) << 2 | (dy > 0) << 3 | (dz < 0) << 4 | (dz > 0) << 5;
}

template <int N, int STAGES>
__global__ void __launch_bounds__(128) k_conv3d_tc(ConvArgs a) {
    static_assert(N % 16 == 0 && N >= 16 && N <= 128, "N");
    extern __shared__ __align__(128) uint8_t smem[];
    __shared__ int2 rows[kConvRows];   // a row's voxel and its y, z faces (64: an empty position)
    __shared__ __align__(8) uint64_t mbar[STAGES];
    __shared__ uint32_t tslot;
    const int tid = threadIdx.x, warp = tid >> 5;
    const int nch0 = a.c0 >> 4, nch = (a.c0 + a.c1) >> 4, G = 2 * nch;
    const int SA = G * kConvPlane, SB = SA + 3 * nch * N * 32;
    constexpr uint32_t NCOLS = conv_tmem_cols<N>();
    constexpr uint32_t IDESC = idesc_bf16(128, N);

    if (warp == 0) { tmem_alloc(&tslot, NCOLS); tmem_relinquish(); }
    if (tid == 0) {
        for (int s = 0; s < STAGES; ++s) mbar_init(&mbar[s], 1);
        fence_mbar_init();
    }
    for (int row = tid; row < kConvRows; row += 128) {
        const int u = (int)blockIdx.x * 128 - 1 + row;
        int vox = -1, face = 64;
        if (u >= 0) {
            const int line = u / (a.W + 1), x = u - line * (a.W + 1) - 1, y = line % a.H, z = line / a.H;
            if (x >= 0 && z < a.D) {
                vox = line * a.W + x;
                face = conv_faces(1, y, z, 3, a.H, a.D);
            }
        }
        rows[row] = make_int2(vox, face);
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t taddr = tslot;
    const int v = rows[tid + 1].x;   // this thread's output voxel
    const bool valid = v >= 0;

    // a thread loads one 8-channel group of every (128 / G)-th row, a row's groups by neighbours
    const int per = 128 / G, row0 = tid / G, g = tid - row0 * G;
    const bool second = g >= 2 * nch0;
    const int cs = second ? a.c1 : a.c0;
    const __nv_bfloat16 *const src0 = second ? a.in1 + (g - 2 * nch0) * 8 : a.in0 + g * 8;
    // one chunk (G = 2): the thread's rows, tid / 2, + 64 and (four threads) + 128, in registers
    const int2 mine[3] = {rows[tid >> 1], rows[(tid >> 1) + 64], tid < 4 ? rows[128 + (tid >> 1)] : make_int2(0, 64)};
    auto load_step = [&](int s, int st) {
        const uint32_t base = su32(smem + st * SB), dst = base + g * kConvPlane;
        const int mask = conv_crosses(3 * s + 1);
        const __nv_bfloat16 *const src = src0 + (long)(((s / 3 - 1) * a.H + s % 3 - 1) * a.W) * cs;
        if (G == 2) {
#pragma unroll
            for (int u = 0; u < 3; ++u) {
                const bool in = (mine[u].y & mask) == 0;
                if (u < 2 || tid < 4) cp_async16_l1(dst + (row0 + 64 * u) * 16, in ? src + (long)mine[u].x * 16 : a.in0, in ? 16 : 0);
            }
        } else if (row0 < per) {
#pragma unroll 4
            for (int row = row0; row < kConvRows; row += per) {
                const int2 t = rows[row];
                const bool in = (t.y & mask) == 0;
                cp_async16_l1(dst + row * 16, in ? src + (long)t.x * cs : a.in0, in ? 16 : 0);
            }
        }
        const uint8_t *wsrc = reinterpret_cast<const uint8_t *>(a.wpk) + (long)s * 3 * nch * N * 32;
        for (int q = tid; q < 3 * nch * N * 2; q += 128) cp_async16(base + SA + q * 16, wsrc + q * 16, 16);
    };
    // stage 0's descriptors; others by adding to the start addresses (16-byte units: no
    // carry leaves the field, shared memory ends below it)
    const uint64_t ad0 = smem_desc(su32(smem), kConvPlane, 128), bd0 = smem_desc(su32(smem) + SA, 128, 256);

    constexpr int nsteps = 9;
    bool ok = true;
#pragma unroll 1
    for (int s = 0; s < STAGES - 1; ++s) {
        load_step(s, s);
        cp_async_commit();
    }
#pragma unroll 1
    for (int s = 0; s < nsteps; ++s) {
        const int st = s % STAGES;
        cp_async_wait<STAGES - 2>();
        fence_async_smem();
        __syncthreads();
        if (tid == 0 && ok) {
            tc_fence_after();
            uint64_t ad = ad0 + (uint32_t)(st * SB) / 16, bd = bd0 + (uint32_t)(st * SB) / 16;
#pragma unroll
            for (int dx = 0; dx < 3; ++dx)
                for (int ch = 0; ch < nch; ++ch, bd += N * 2)
                    tc_mma_bf16(taddr, ad + ch * (2 * kConvPlane / 16) + dx, bd, IDESC, s + dx + ch > 0 ? 1u : 0u);
            tc_commit(&mbar[st]);
        }
        const int ns = s + STAGES - 1;
        if (ns < nsteps) {
            const int nst = ns % STAGES;
            // stage nst was last read by the MMAs of step ns - STAGES (= s - 1)
            if (ns >= STAGES && ok) ok = mbar_wait(&mbar[nst], (uint32_t)(((ns - STAGES) / STAGES) & 1), a.err);
            if (ok) load_step(ns, nst);
        }
        cp_async_commit();
    }
    cp_async_wait<0>();
    // all MMAs done once the last commit has arrived
    if (ok) {
        const int last = nsteps - 1;
        ok = mbar_wait(&mbar[last % STAGES], (uint32_t)((last / STAGES) & 1), a.err);
    }
    __syncthreads();
    tc_fence_after();
    if (ok) {
        const uint32_t tw = taddr + ((uint32_t)(warp * 32) << 16);
        if (a.out32) {
            float vals[16];
            tc_ld16(tw, vals);
            if (valid) a.out32[v] = vals[0] + (a.bias ? a.bias[0] : 0.0f);
        } else {
#pragma unroll
            for (int q = 0; q < N / 16; ++q) {
                float vals[16];
                tc_ld16(tw + q * 16, vals);
                if (valid) {
                    __align__(16) __nv_bfloat16 o[16];
#pragma unroll
                    for (int e = 0; e < 16; ++e) {
                        int n = q * 16 + e;
                        float t = vals[e] + (a.bias ? a.bias[n] : 0.0f);
                        if (a.relu) t = fmaxf(t, 0.0f);
                        o[e] = __float2bfloat16(t);
                    }
                    int n0 = q * 16;
                    __nv_bfloat16 *dst;
                    const __nv_bfloat16 *msk;
                    if (n0 < a.split) { dst = a.out0 + (long)v * a.split + n0; msk = a.mask0 ? a.mask0 + (long)v * a.split + n0 : nullptr; }
                    else { dst = a.out1 + (long)v * (N - a.split) + (n0 - a.split); msk = a.mask1 ? a.mask1 + (long)v * (N - a.split) + (n0 - a.split) : nullptr; }
                    if (msk) {
#pragma unroll
                        for (int e = 0; e < 16; ++e)
                            if (!(__bfloat162float(msk[e]) > 0.0f)) o[e] = __float2bfloat16(0.0f);
                    }
                    uint4 *d4 = reinterpret_cast<uint4 *>(dst);
                    const uint4 *s4 = reinterpret_cast<const uint4 *>(o);
                    d4[0] = s4[0];
                    d4[1] = s4[1];
                }
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0) tmem_dealloc(taddr, NCOLS);
}

// ---- weight gradient on the tensor cores
// dW[n][tap][c] = sum_v dY[v][n] X[v + off(tap)][c] as GEMMs
//   D[m][n] = sum_k A[m][k] B[n][k],  n = output channel, k = position (the lines of
//   voxels with an empty position before each, as in the forward pass).
// A CTA takes 16 input channels and a chunk of positions for all taps.  A stage holds,
// for kDwK positions, nine copies of X, one a (dz, dy) of the taps, shifted by it (zero
// outside the domain and at empty positions), as 18 planes of 16-byte rows (8 channels of
// a position), and dY as N / 8 planes.  Both operands are MN-major, which is the order
// the channels-last tensors already have: a core matrix is 8 consecutive rows of a plane,
// K-adjacent ones 128 B apart (the leading byte offset), M- or N-adjacent ones a plane
// apart (the stride byte offset).  The planes are the M dimension, m = plane * 8 +
// channel, so the dx taps are the same planes from one row on: one accumulator a dx and
// M tile (16 planes; the second, of 64 rows, holds planes 16, 17 and rows that nothing reads).  Each
// copy serves three taps: 43 us for 16 -> 16 channels on 65^3 voxels, 90 for 48 -> 16,
// where a gather a tap took 52 and 129.  The accumulators are added to the FP32 dW with atomics; the CTAs
// of the first input channels also add their chunk's sum of dY to db.
struct DwArgs {
    const __nv_bfloat16 *in0, *in1;   // X, channels-last, concatenated along C
    int c0, c1;
    const __nv_bfloat16 *dy;          // dY, channels-last, N channels
    float *dw;                        // [N][27][c0 + c1]
    float *db;                        // [N], or null
    int D, H, W, nvox;
    int chunk;                        // positions a CTA reduces (a multiple of kDwK)
    int *err;
};

constexpr int kDwStages = 4, kDwK = 64;
constexpr int kDwPlaneA = (kDwK + 4) * 16, kDwPlaneB = kDwK * 16;   // bytes of a plane (66 rows are read of A's)
constexpr int kDwPlanes = 18;
template <int N>
__host__ __device__ constexpr int dw_stage_bytes() { return kDwPlanes * kDwPlaneA + N / 8 * kDwPlaneB; }
// (the second M tile's unused rows lie up to 6 planes past the last stage's A)
template <int N>
__host__ __device__ constexpr int dw_smem_bytes() { return kDwStages * dw_stage_bytes<N>() + 6 * kDwPlaneA; }
// dx taps of a CTA: all three where their accumulators (two M tiles each) fit the tensor memory
template <int N>
__host__ __device__ constexpr int dw_taps() { return 6 * N <= 512 ? 3 : 1; }
template <int N>
__host__ __device__ constexpr uint32_t dw_tmem_cols() {
    constexpr int c = 2 * N * dw_taps<N>();
    return c <= 32 ? 32u : c <= 64 ? 64u : c <= 128 ? 128u : c <= 256 ? 256u : 512u;
}

// Grid: chunks of positions, groups of 16 input channels, 3 / dw_taps dx taps.
template <int N>
__global__ void __launch_bounds__(128) k_conv_dw_tc(DwArgs a) {
    static_assert(N % 16 == 0 && N >= 16 && N <= 128, "N");
    extern __shared__ __align__(128) uint8_t smem[];
    __shared__ float sdb[N];
    __shared__ __align__(8) uint64_t mbar[kDwStages];
    __shared__ uint32_t tslot;
    constexpr int SB = dw_stage_bytes<N>(), SA = kDwPlanes * kDwPlaneA, KS = kDwK / 16, TAPS = dw_taps<N>();
    const int tid = threadIdx.x, warp = tid >> 5;
    constexpr uint32_t NCOLS = dw_tmem_cols<N>();
    constexpr uint32_t MN = (1u << 15) | (1u << 16), IDESC[2] = {idesc_bf16(128, N) | MN, idesc_bf16(64, N) | MN};   // A and B MN-major
    const int cin = a.c0 + a.c1, c = blockIdx.y * 16, dx0 = blockIdx.z;
    const long u0 = (long)blockIdx.x * a.chunk;
    const long u1 = min(u0 + (long)a.chunk, (long)a.D * a.H * (a.W + 1));
    const int nsteps = u1 > u0 ? (int)((u1 - u0 + kDwK - 1) / kDwK) : 0;

    if (warp == 0) { tmem_alloc(&tslot, NCOLS); tmem_relinquish(); }
    if (tid == 0) {
        for (int s = 0; s < kDwStages; ++s) mbar_init(&mbar[s], 1);
        fence_mbar_init();
    }
    if (tid < N) sdb[tid] = 0.0f;
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t taddr = tslot;

    const __nv_bfloat16 *const src = c < a.c0 ? a.in0 + c : a.in1 + (c - a.c0);
    const int cs = c < a.c0 ? a.c0 : a.c1;
    // Row q of a stage's planes is position u0 + kDwK step - 1 + q of X (A reads rows 0 ..
    // kDwK + 1), dY's row q position u0 + kDwK step + q.  Two neighbouring threads load row
    // tid / 2 of all nine copies, 8 channels each; the first 36 threads also rows 64 and 65.
    struct Pos {
        long u;
        int x, y, z;   // x = -1: an empty position
    };
    auto pos_at = [&](long u) {
        Pos p;
        p.u = u;
        const long w = max(u, 0L), line = w / (a.W + 1);
        p.x = u < 0 ? -1 : (int)(w - line * (a.W + 1)) - 1;
        p.y = (int)(line % a.H);
        p.z = (int)(line / a.H);
        return p;
    };
    const int ax = kDwK % (a.W + 1), ay = (kDwK / (a.W + 1)) % a.H, az = kDwK / ((a.W + 1) * a.H);   // a stage's advance
    auto advance = [&](Pos &p) {
        p.u += kDwK;
        if (p.u - kDwK < 0) { p = pos_at(p.u); return; }
        p.x += ax;
        if (p.x >= a.W) { p.x -= a.W + 1; ++p.y; }
        p.y += ay;
        if (p.y >= a.H) { p.y -= a.H; ++p.z; }
        p.z += az;
    };
    const int half = tid & 1, row = tid >> 1;
    Pos p = pos_at(u0 - 1 + row), e = pos_at(u0 - 1 + kDwK + ((tid >> 1) & 1)), d = pos_at(u0 + row);
    const int soy = a.W * cs, soz = a.H * soy;
    auto face_of = [&](const Pos &q) { return q.x < 0 || q.z >= a.D ? 64 : conv_faces(1, q.y, q.z, 3, a.H, a.D); };
    auto voxel = [&](const Pos &q) { return ((long)q.z * a.H + q.y) * a.W + q.x; };
    auto load_x = [&](const __nv_bfloat16 *x, int face, int seg, uint32_t dst) {
        const bool in = (face & conv_crosses(3 * seg + 1)) == 0;
        cp_async16_l1(dst, in ? x + (seg / 3 - 1) * (long)soz + (seg % 3 - 1) * (long)soy : src, in ? 16 : 0);
    };
    auto load_step = [&](int st) {   // stages in order
        const uint32_t base = su32(smem + st * SB), dst = base + half * kDwPlaneA + row * 16;
        const __nv_bfloat16 *const x = src + voxel(p) * cs + half * 8;
        const int face = face_of(p);
#pragma unroll
        for (int seg = 0; seg < 9; ++seg) load_x(x, face, seg, dst + 2 * seg * kDwPlaneA);
        if (tid < 36)
            load_x(src + voxel(e) * cs + half * 8, face_of(e), tid >> 2, base + (2 * (tid >> 2) + half) * kDwPlaneA + (kDwK + ((tid >> 1) & 1)) * 16);
        const bool ok = d.x >= 0 && d.u < u1;
        const long w = voxel(d);
#pragma unroll
        for (int g = half; g < N / 8; g += 2) cp_async16(base + SA + g * kDwPlaneB + row * 16, ok ? a.dy + w * N + g * 8 : a.dy, ok ? 16 : 0);
        advance(p);
        advance(e);
        advance(d);
    };

    const uint64_t ad0 = smem_desc(su32(smem) + dx0 * 16, 128, kDwPlaneA), bd0 = smem_desc(su32(smem) + SA, 128, kDwPlaneB);
    bool ok = true;
#pragma unroll 1
    for (int s = 0; s < kDwStages - 1; ++s) {
        if (s < nsteps) load_step(s);
        cp_async_commit();
    }
#pragma unroll 1
    for (int s = 0; s < nsteps; ++s) {
        const int st = s % kDwStages;
        cp_async_wait<kDwStages - 2>();
        fence_async_smem();
        __syncthreads();
        if (tid == 0 && ok) {
            tc_fence_after();
            const uint64_t ad = ad0 + (uint32_t)(st * SB) / 16, bd = bd0 + (uint32_t)(st * SB) / 16;
#pragma unroll
            for (int k = 0; k < KS; ++k)
#pragma unroll
                for (int t = 0; t < TAPS; ++t)
#pragma unroll
                    for (int m = 0; m < 2; ++m)
                        tc_mma_bf16(taddr + (2 * t + m) * N, ad + (m * kDwPlaneA + t + 16 * k), bd + k * 16, IDESC[m], s + k > 0 ? 1u : 0u);
            tc_commit(&mbar[st]);
        }
        const int ns = s + kDwStages - 1;
        if (ns < nsteps) {
            const int nst = ns % kDwStages;
            // stage nst was last read by the MMAs of step ns - kDwStages (= s - 1)
            if (ns >= kDwStages && ok) ok = mbar_wait(&mbar[nst], (uint32_t)(((ns - kDwStages) / kDwStages) & 1), a.err);
            if (ok) load_step(nst);
        }
        cp_async_commit();
    }
    cp_async_wait<0>();
    if (ok && nsteps > 0) {
        const int last = nsteps - 1;
        ok = mbar_wait(&mbar[last % kDwStages], (uint32_t)((last / kDwStages) & 1), a.err);
    }
    __syncthreads();
    tc_fence_after();
    if (ok && nsteps > 0) {
        const uint32_t tw = taddr + ((uint32_t)(warp * 32) << 16);
#pragma unroll
        for (int t = 0; t < TAPS; ++t)
#pragma unroll
            for (int m = 0; m < 2; ++m) {
                if (m == 1 && warp > 0) continue;   // rows 0 .. 15 only
                const int plane = m * 16 + (tid >> 3), tap = 3 * (plane >> 1) + dx0 + t, ci = c + (plane & 1) * 8 + (tid & 7);
#pragma unroll
                for (int q = 0; q < N / 16; ++q) {
                    float vals[16];
                    tc_ld16(tw + (2 * t + m) * N + q * 16, vals);
                    if (plane < kDwPlanes) {
#pragma unroll
                        for (int o = 0; o < 16; ++o) atomicAdd(&a.dw[((long)(q * 16 + o) * 27 + tap) * cin + ci], vals[o]);
                    }
                }
            }
    }
    if (a.db && c == 0 && dx0 == 0) {   // the sum of the chunk's share of dY: a thread 8 channels of every (1024 / N)-th voxel
        const long v0 = (long)blockIdx.x * a.nvox / gridDim.x, v1 = ((long)blockIdx.x + 1) * a.nvox / gridDim.x;
        const int ng = tid % (N / 8), rows = 128 / (N / 8);
        float sum[8] = {};
        if (tid < rows * (N / 8)) {
#pragma unroll 4
            for (long w = v0 + tid / (N / 8); w < v1; w += rows) {
                const uint4 q = *reinterpret_cast<const uint4 *>(a.dy + w * N + ng * 8);
                const __nv_bfloat162 *p = reinterpret_cast<const __nv_bfloat162 *>(&q);
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    sum[2 * e] += __low2float(p[e]);
                    sum[2 * e + 1] += __high2float(p[e]);
                }
            }
#pragma unroll
            for (int e = 0; e < 8; ++e) atomicAdd(&sdb[ng * 8 + e], sum[e]);
        }
        __syncthreads();
        if (tid < N) atomicAdd(&a.db[tid], sdb[tid]);
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0) tmem_dealloc(taddr, NCOLS);
}

}  // namespace saras
