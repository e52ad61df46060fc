// 3x3x3 convolution of the learned warm start on the 5th-generation tensor
// cores: tcgen05.mma (kind::f16, BF16 operands, FP32 accumulator in tensor
// memory), its input staged once per block and read shifted by every tap.
//
// A CTA computes a block of TX x TY x TZ voxels for up to 48 output channels.
// Input planes (16 channels of a (TX+2) x (TY+2) halo at one z, zeros outside
// the volume) stream through a ring of shared-memory stages, each loaded once
// by three warps with 16-byte cp.async.  (TMA boxes would need an inner extent
// of 16 bytes for this layout and then move about 3 bytes a clock.)  A stage holds 16-byte
// rows (8 channels of a voxel) in voxel order, which is the canonical K-major
// layout without swizzle with 8-row groups 128 bytes apart, so the operand of
// a tap is the same rows at another start address: nothing is copied per tap.
// The weights of all taps stay in shared memory, the three dz taps of one
// (dy, dx) side by side: one instruction of N = 3 cout columns adds an input
// plane to the three output planes it belongs to, whose accumulators are
// neighbouring tensor-memory columns.  That reads A nine times per plane
// instead of 27 (with N = 16 an instruction is bound by its 4 KB of A).
// M = 128 rows are a line of voxels (TX = 128), else 128 consecutive positions
// of the staged plane, whose halo columns are computed and not stored.
// Warps: 0 issues instructions, 1-3 load, 4-7 store results.  Before this a CTA
// staged 27 tap-shifted copies of 128 voxels through registers, one
// instruction per pair of barriers: 32 -> 32 channels at 62 x 58 x 31 x 4 took
// 197 us, now 69.
//
// Every wait is bounded; on a timeout the CTA raises the error flag read by
// omb_unet_take_error(), waits (bounded) for its copies and instructions in
// flight, frees its tensor memory and leaves without its output.  The weight
// gradient (k_conv3d_wgrad_tc, below) runs on the same instructions with the
// voxels as the reduction dimension.
#include <cuda_bf16.h>

#include <cmath>

#include "kernels.h"
#include "../../include/omega_b200_unet.h"

namespace omb {

__device__ int g_unet_error = 0;

namespace tc {

constexpr int kM = 128;              // voxels per CTA (UMMA M)
constexpr int kCoreGroup = 256;      // bytes between 8-row groups (SBO)
constexpr int kKHalf = 128;          // bytes between the two K halves (LBO)
constexpr int kWaitTries = 1 << 20;  // bounded mbarrier polling

__device__ __forceinline__ uint32_t smem_u32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

// Shared-memory matrix descriptor: K-major, no swizzle, sm100 (version 1).
__device__ __forceinline__ uint64_t smem_desc(uint32_t addr) {
    uint64_t d = 0;
    d |= (uint64_t)((addr >> 4) & 0x3FFF);
    d |= (uint64_t)((kKHalf >> 4) & 0x3FFF) << 16;
    d |= (uint64_t)((kCoreGroup >> 4) & 0x3FFF) << 32;
    d |= (uint64_t)1 << 46;
    return d;  // base offset 0, LBO mode 0, layout type 0 (no swizzle)
}

// Instruction descriptor: D F32, A/B BF16, both K-major, M = 128, N = n.
__host__ __device__ constexpr uint32_t instr_desc(int n) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(kM >> 4) << 24);
}

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(bar), "r"(count) : "memory");
}

__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity) {
    for (int i = 0; i < kWaitTries; ++i) {
        uint32_t done;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}\n"
            : "=r"(done)
            : "r"(bar), "r"(parity)
            : "memory");
        if (done) return true;
    }
    return false;
}

__device__ __forceinline__ void mma_issue(uint32_t tmem_d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t acc) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n"
        ::"r"(tmem_d), "l"(a), "l"(b), "r"(idesc), "r"(acc)
        : "memory");
}

__device__ __forceinline__ void mma_commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(bar)
                 : "memory");
}

__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float (&v)[16]) {
    uint32_t r[16];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];\n"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
#pragma unroll
    for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
}

}  // namespace tc

// Shape of one convolution launch (conv_plan).
struct ConvPlan {
    int X, Y, Z, B;
    int TX, TY, TZ;      // output voxels of a CTA's block
    int P, S, T;         // staged line length, positions between M tiles, M tiles per plane
    int ntx, nty, ntz;   // blocks per axis
    int tiles;           // blocks in all
    int ring;            // stages
    int plane, stage;    // bytes of one 8-channel half plane (128-byte aligned) and of a stage
    int cols;            // tensor-memory columns to allocate
    int smem;            // dynamic shared memory
};

namespace tc {

// One instruction with descriptors given as their low words (`hi` is the same
// for both operands), issued by the lanes where `on` is set.  The whole warp
// computes the operands: they stay in uniform registers, which the instruction
// reads; a lone thread's would be moved there one by one.
__device__ __forceinline__ void mma_lo(uint32_t tmem_d, uint32_t a_lo, uint32_t b_lo, uint32_t hi, uint32_t idesc,
                                       uint32_t acc, uint32_t on) {
    asm volatile(
        "{\n\t.reg .pred p, e;\n\t.reg .b64 da, db;\n\t"
        "mov.b64 da, {%1, %3};\n\t"
        "mov.b64 db, {%2, %3};\n\t"
        "setp.ne.b32 p, %5, 0;\n\t"
        "setp.ne.b32 e, %6, 0;\n\t"
        "@e tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %4, p;\n\t}\n"
        ::"r"(tmem_d), "r"(a_lo), "r"(b_lo), "r"(hi), "r"(idesc), "r"(acc), "r"(on)
        : "memory");
}

}  // namespace tc

// CO: output channels of a CTA; blockIdx.y picks which of COUT.
template <int CIN, int COUT, int CO, bool RELU, bool MASK>
__global__ void __launch_bounds__(256) k_conv3d_tc(const __grid_constant__ ConvPlan pl,
                                                   const __nv_bfloat16 *__restrict__ in,
                                                   const __nv_bfloat16 *__restrict__ w,
                                                   const float *__restrict__ bias, __nv_bfloat16 *__restrict__ out,
                                                   const __nv_bfloat16 *__restrict__ mask) {
    static_assert(CIN % 16 == 0 && COUT % CO == 0 && CO % 16 == 0 && CO <= 80, "channel counts");
    constexpr int NCH = CIN / 16;             // 16-channel chunks: stages per input plane
    constexpr int WBLOCK = 3 * CO * 32;       // weights of one (chunk, dy, dx): 3 dz taps x CO rows x 16 channels
    constexpr int WBYTES = NCH * 9 * WBLOCK;
    constexpr int kLoaders = 96;
    extern __shared__ __align__(1024) uint8_t smem[];
    __shared__ __align__(8) uint64_t full[4], empty[4], done, drained;
    __shared__ uint32_t tmem_base;
    __shared__ int failed;
    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
    const int co0 = blockIdx.y * CO;
    if (tid == 0) {
        for (int i = 0; i < 4; ++i) {
            tc::mbar_init(tc::smem_u32(&full[i]), kLoaders / 32);
            tc::mbar_init(tc::smem_u32(&empty[i]), 1);
        }
        tc::mbar_init(tc::smem_u32(&done), 1);
        tc::mbar_init(tc::smem_u32(&drained), 128);
        failed = 0;
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(tc::smem_u32(&tmem_base)),
                     "r"(pl.cols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
    }
    // weights: block (chunk, dy, dx), K half, row = (dz = +1, 0, -1) x CO, 8 channels
    for (int i = tid; i < WBYTES / 16; i += 256) {
        const int row = i % (3 * CO), q = i / (3 * CO);
        const int h = q & 1, blk = q >> 1;
        const int t9 = blk % 9, c = blk / 9;
        const int tap = (2 - row / CO) * 9 + t9;
        *reinterpret_cast<uint4 *>(smem + (size_t)i * 16) = __ldg(reinterpret_cast<const uint4 *>(
            w + ((int64_t)tap * COUT + co0 + row % CO) * CIN + c * 16 + h * 8));
    }
    asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    const uint32_t tmem = tmem_base;
    const uint32_t wbase = tc::smem_u32(smem), ring = wbase + WBYTES;
    const int nst = (pl.TZ + 2) * NCH;   // stages per block
    const int mine = (int)blockIdx.x < pl.tiles ? (pl.tiles - 1 - (int)blockIdx.x) / (int)gridDim.x + 1 : 0;
    const int total = mine * nst;

    auto block_origin = [&](int k, int &x0, int &y0, int &z0, int &b) {
        int tile = (int)blockIdx.x + k * (int)gridDim.x;
        x0 = tile % pl.ntx * pl.TX;
        tile /= pl.ntx;
        y0 = tile % pl.nty * pl.TY;
        tile /= pl.nty;
        z0 = tile % pl.ntz * pl.TZ;
        b = tile / pl.ntz;
    };
    auto fail = [&] {
        atomicExch(&g_unet_error, 1);
        *(volatile int *)&failed = 1;
    };

    if (warp >= 1 && warp <= 3) {
        // loaders: stage it + lag is requested before stage `it` is handed over
        const int j = tid - 32;
        const int lag = pl.ring > 2 ? 2 : 1;
        const int items = 2 * pl.P * (pl.TY + 2);
        const uint32_t bar0 = tc::smem_u32(&full[0]);
        auto hand_over = [&](int it) {
            // (cp.async writes through the generic proxy, the tensor core reads through the async one)
            asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
            __syncwarp();
            if (lane == 0)
                asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(bar0 + 8u * (it % pl.ring)) : "memory");
        };
        int x0 = 0, y0 = 0, z0 = 0, b = 0, it = 0;
        bool ok = true;
        for (int k = 0; k < mine && ok; ++k) {
            block_origin(k, x0, y0, z0, b);
            for (int st = 0; st < nst; ++st, ++it) {
                const int slot = it % pl.ring, use = it / pl.ring;
                if (use > 0) ok = tc::mbar_wait(tc::smem_u32(&empty[slot]), (uint32_t)(use - 1) & 1u);
                if (!__all_sync(0xffffffffu, ok)) {
                    ok = false;
                    break;
                }
                const int zi = st / NCH, c = st - zi * NCH, z = z0 + zi - 1;
                const bool zin = z >= 0 && z < pl.Z;
                const uint32_t dst0 = ring + slot * pl.stage;
                const __nv_bfloat16 *plane = in + ((int64_t)b * pl.Z + (zin ? z : 0)) * pl.Y * pl.X * CIN + c * 16;
                // item i: half i & 1 of position i >> 1
                int line = 0, x = j >> 1;
                const int h = j & 1;
                for (int i = j; i < items; i += kLoaders, x += kLoaders / 2) {
                    while (x >= pl.P) {
                        x -= pl.P;
                        ++line;
                    }
                    const int gx = x0 + x - 1, gy = y0 + line - 1;
                    const bool inside = zin && gx >= 0 && gx < pl.X && gy >= 0 && gy < pl.Y;
                    const __nv_bfloat16 *src = inside ? plane + ((int64_t)gy * pl.X + gx) * CIN + h * 8 : in;
                    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(dst0 + h * pl.plane + (i >> 1) * 16),
                                 "l"(src), "r"(inside ? 16 : 0)
                                 : "memory");
                }
                asm volatile("cp.async.commit_group;\n" ::: "memory");
                if (it >= lag) {
                    if (lag == 2)
                        asm volatile("cp.async.wait_group 2;\n" ::: "memory");
                    else
                        asm volatile("cp.async.wait_group 1;\n" ::: "memory");
                    hand_over(it - lag);
                }
            }
        }
        asm volatile("cp.async.wait_all;\n" ::: "memory");
        if (ok)
            for (int i = total > lag ? total - lag : 0; i < total; ++i) hand_over(i);
        else if (lane == 0)
            fail();
    } else if (warp == 0) {
        const uint32_t t0 = __shfl_sync(0xffffffffu, tmem, 0), on = lane == 0;
        // descriptor words: start address and K-half stride below, 8-row stride (128 bytes) and version above
        constexpr uint32_t kHi = (128u >> 4) | (1u << 14);
        const uint32_t a_base = ((ring >> 4) & 0x3FFF) | (uint32_t)(pl.plane >> 4) << 16;
        const uint32_t b_base = ((wbase >> 4) & 0x3FFF) | (uint32_t)(3 * CO) << 16;
        const uint32_t dstep = pl.TZ * CO;
        int it = 0;
        bool ok = true;
        for (int k = 0; k < mine && ok; ++k) {
            // the previous block's sums have been read
            if (k > 0) ok = __all_sync(0xffffffffu, tc::mbar_wait(tc::smem_u32(&drained), (uint32_t)(k - 1) & 1u));
            for (int st = 0; st < nst && ok; ++st, ++it) {
                const int slot = it % pl.ring;
                ok = __all_sync(0xffffffffu, tc::mbar_wait(tc::smem_u32(&full[slot]), (uint32_t)(it / pl.ring) & 1u));
                if (!ok) break;
                asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
                const int zr = st / NCH, c = st - zr * NCH;               // input plane z0 + zr - 1
                const int lo = max(zr - 2, 0), hi = min(zr, pl.TZ - 1);   // output planes it adds to
                const bool opens = c == 0 && zr < pl.TZ;                  // the last of them gets its first sum
                const uint32_t a0 = a_base + (uint32_t)(slot * (pl.stage >> 4));
                const uint32_t b0 = b_base + (uint32_t)(c * 9 * (WBLOCK / 16)), d0 = t0 + lo * CO;
                const uint32_t skip = (uint32_t)((lo - (zr - 2)) * CO);   // weight rows of planes below the block
                if (opens) {
                    // the first tap apart: it overwrites the new plane's sums and adds to the others'
                    const int n = (hi - lo) * CO;
                    for (int t = 0; t < pl.T; ++t) {
                        if (n > 0)
                            tc::mma_lo(d0 + t * dstep, a0 + t * pl.S, b0 + skip, kHi, tc::instr_desc(n), 1u, on);
                        tc::mma_lo(t0 + hi * CO + t * dstep, a0 + t * pl.S, b0 + 2 * CO, kHi, tc::instr_desc(CO), 0u, on);
                    }
                }
                const uint32_t idesc = tc::instr_desc((hi - lo + 1) * CO);
                for (int t9 = opens ? 1 : 0; t9 < 9; ++t9) {
                    uint32_t a = a0 + (uint32_t)(t9 / 3 * pl.P + t9 % 3), d = d0;
                    const uint32_t b = b0 + skip + (uint32_t)(t9 * (WBLOCK / 16));
#pragma unroll 4
                    for (int t = 0; t < pl.T; ++t, a += pl.S, d += dstep) tc::mma_lo(d, a, b, kHi, idesc, 1u, on);
                }
                if (on) tc::mma_commit(tc::smem_u32(&empty[slot]));
            }
            // (on failure too: whoever waits for it is let go once the instructions in flight have ended)
            if (on) {
                if (!ok) fail();
                tc::mma_commit(tc::smem_u32(&done));
            }
            __syncwarp();
        }
    } else if (warp >= 4) {
        const int quarter = warp & 3;   // the tensor-memory lanes this warp can read
        for (int k = 0; k < mine; ++k) {
            const bool ok = tc::mbar_wait(tc::smem_u32(&done), (uint32_t)k & 1u) && !*(volatile int *)&failed;
            if (!__all_sync(0xffffffffu, ok)) {
                if (lane == 0) fail();
                break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
            int x0, y0, z0, b;
            block_origin(k, x0, y0, z0, b);
            for (int t = 0; t < pl.T; ++t) {
                const int pos = t * pl.S + quarter * 32 + lane;
                const int line = pos / pl.P, x = x0 + pos - line * pl.P, y = y0 + line;
                const bool inside = pos - line * pl.P < pl.TX && line < pl.TY && x < pl.X && y < pl.Y;
                for (int zo = 0; zo < pl.TZ && z0 + zo < pl.Z; ++zo) {
                    const int64_t vo = (((int64_t)b * pl.Z + z0 + zo) * pl.Y + y) * pl.X + x;
#pragma unroll
                    for (int c0 = 0; c0 < CO; c0 += 16) {
                        float acc[16];
                        __syncwarp();
                        tc::tmem_ld16(tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)((t * pl.TZ + zo) * CO + c0), acc);
                        if (inside) {
                            __nv_bfloat16 m16[16];
                            if (MASK) {
                                const uint4 *mp = reinterpret_cast<const uint4 *>(mask + vo * COUT + co0 + c0);
                                *reinterpret_cast<uint4 *>(m16) = __ldg(mp);
                                *reinterpret_cast<uint4 *>(m16 + 8) = __ldg(mp + 1);
                            }
                            uint32_t packed[8];
#pragma unroll
                            for (int i = 0; i < 16; i += 2) {
                                float lo = acc[i], hi = acc[i + 1];
                                if (bias) {
                                    lo += __ldg(bias + co0 + c0 + i);
                                    hi += __ldg(bias + co0 + c0 + i + 1);
                                }
                                if (RELU) {
                                    lo = fmaxf(lo, 0.f);
                                    hi = fmaxf(hi, 0.f);
                                }
                                if (MASK) {
                                    if (!(__bfloat162float(m16[i]) > 0.f)) lo = 0.f;
                                    if (!(__bfloat162float(m16[i + 1]) > 0.f)) hi = 0.f;
                                }
                                const __nv_bfloat162 pr = __floats2bfloat162_rn(lo, hi);
                                packed[i / 2] = *reinterpret_cast<const uint32_t *>(&pr);
                            }
                            uint4 *op = reinterpret_cast<uint4 *>(out + vo * COUT + co0 + c0);
                            op[0] = make_uint4(packed[0], packed[1], packed[2], packed[3]);
                            op[1] = make_uint4(packed[4], packed[5], packed[6], packed[7]);
                        }
                    }
                }
            }
            // the next block's instructions overwrite the accumulators
            asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
            asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(tc::smem_u32(&drained)) : "memory");
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    if (warp == 0) {
        asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(pl.cols) : "memory");
    }
}

// ---------------------------------------------------------------------------
// Lines of 65 to 128 voxels.  An instruction of M = 128, K = 16 takes about 128
// clocks whatever its N up to 256 (it reads A at 32 bytes a clock; timed with N =
// 16 to 144), so the taps of an input line should share as few instructions as
// their outputs allow.  A CTA marches along y with 16 output channels: for every
// input line and dx one instruction of N = 144 columns adds to the nine output
// lines of its (dy, dz) neighbourhood.  Their accumulators are neighbouring
// tensor-memory columns: z planes of the block outside, three slots inside, the
// slot of an output line its y modulo 3.  The order of the dy taps within the
// instruction turns with y, so the weights are kept in three orders.  When an
// input line has been added, the output line behind it is complete: it is stored
// and its slot cleared before the next input line.  Two CTAs on an SM hide that
// from the tensor core.  Against the kernel above (N = 3 cout, nine instructions
// per line), 128 x 128 x 64 x 4: 16 -> 16 channels 255 to 149 us, 48 -> 16 705 to
// 515 us, 16 -> 48 365 to 361 us; a training step of the two-level network 8.10 to
// 7.24 ms.
// ---------------------------------------------------------------------------
struct LinePlan {
    int X, Y, Z, B;
    int TX, TZ, YS;       // x voxels, z planes and output lines of a block
    int P;                // staged line length
    int ntx, ntz, nys;    // blocks per axis
    int tiles;
    int ring, plane, stage;   // stages; bytes of an 8-channel half and of a stage
    int cols, smem, occ;
};

template <int CIN, int COUT, bool RELU, bool MASK>
__global__ void __launch_bounds__(256) k_conv3d_lines(const __grid_constant__ LinePlan pl,
                                                      const __nv_bfloat16 *__restrict__ in,
                                                      const __nv_bfloat16 *__restrict__ w,
                                                      const float *__restrict__ bias, __nv_bfloat16 *__restrict__ out,
                                                      const __nv_bfloat16 *__restrict__ mask) {
    constexpr int CO = 16, NCH = CIN / 16;
    constexpr int WBLOCK = 9 * CO * 32;            // weights of one (order, chunk, dx): 9 (dz, dy) x CO rows x 16 channels
    constexpr int WBYTES = 3 * NCH * 3 * WBLOCK;
    constexpr int kLoaders = 96;
    extern __shared__ __align__(1024) uint8_t smem[];
    __shared__ __align__(8) uint64_t full[4], empty[4], done, drained;
    __shared__ uint32_t tmem_base;
    __shared__ int failed;
    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
    const int co0 = blockIdx.y * CO;
    if (tid == 0) {
        for (int i = 0; i < 4; ++i) {
            tc::mbar_init(tc::smem_u32(&full[i]), kLoaders / 32);
            tc::mbar_init(tc::smem_u32(&empty[i]), 1);
        }
        tc::mbar_init(tc::smem_u32(&done), 1);
        tc::mbar_init(tc::smem_u32(&drained), 128);
        failed = 0;
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(tc::smem_u32(&tmem_base)),
                     "r"(pl.cols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
    }
    // weights: order o (input line y = o modulo 3), chunk, dx, K half, row (dz = +1, 0, -1) x slot x CO, 8 channels.
    // Slot s of order o holds the output line yo = s modulo 3 among o - 1, o, o + 1: tap dy = y - yo.
    for (int i = tid; i < WBYTES / 16; i += 256) {
        const int row = i % (9 * CO), q = i / (9 * CO);
        const int h = q & 1, blk = q >> 1;
        const int dx = blk % 3, c = blk / 3 % NCH, o = blk / (3 * NCH);
        const int zb = row / (3 * CO), s = row / CO % 3;
        const int dy = (o - s + 4) % 3 - 1;   // (o - s) modulo 3 in -1, 0, 1
        const int tap = (2 - zb) * 9 + (dy + 1) * 3 + dx;
        *reinterpret_cast<uint4 *>(smem + (size_t)i * 16) = __ldg(reinterpret_cast<const uint4 *>(
            w + ((int64_t)tap * COUT + co0 + row % CO) * CIN + c * 16 + h * 8));
    }
    asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    const uint32_t tmem = tmem_base;
    const uint32_t wbase = tc::smem_u32(smem), ring = wbase + WBYTES;
    const int mine = (int)blockIdx.x < pl.tiles ? (pl.tiles - 1 - (int)blockIdx.x) / (int)gridDim.x + 1 : 0;

    struct Block {
        int x0, y0, z0, b, ny;   // ny output lines
    };
    auto block_at = [&](int k) {
        int tile = (int)blockIdx.x + k * (int)gridDim.x;
        Block q;
        q.x0 = tile % pl.ntx * pl.TX;
        tile /= pl.ntx;
        q.z0 = tile % pl.ntz * pl.TZ;
        tile /= pl.ntz;
        q.y0 = tile % pl.nys * pl.YS;
        q.b = tile / pl.nys;
        q.ny = min(pl.YS, pl.Y - q.y0);
        return q;
    };
    auto fail = [&] {
        atomicExch(&g_unet_error, 1);
        *(volatile int *)&failed = 1;
    };

    if (warp >= 1 && warp <= 3) {
        const int j = tid - 32;
        const int lag = pl.ring > 2 ? 2 : 1;
        const int items = 2 * pl.P * (pl.TZ + 2);
        const uint32_t bar0 = tc::smem_u32(&full[0]);
        auto hand_over = [&](int it) {
            // (cp.async writes through the generic proxy, the tensor core reads through the async one)
            asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
            __syncwarp();
            if (lane == 0)
                asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(bar0 + 8u * (it % pl.ring)) : "memory");
        };
        int it = 0;
        bool ok = true;
        for (int k = 0; k < mine && ok; ++k) {
            const Block q = block_at(k);
            for (int st = 0; st < (q.ny + 2) * NCH; ++st, ++it) {
                const int slot = it % pl.ring, use = it / pl.ring;
                if (use > 0) ok = tc::mbar_wait(tc::smem_u32(&empty[slot]), (uint32_t)(use - 1) & 1u);
                if (!__all_sync(0xffffffffu, ok)) {
                    ok = false;
                    break;
                }
                const int line = st / NCH, c = st - line * NCH, y = q.y0 + line - 1;
                const bool yin = y >= 0 && y < pl.Y;
                const uint32_t dst0 = ring + slot * pl.stage;
                const __nv_bfloat16 *row = in + (((int64_t)q.b * pl.Z) * pl.Y + (yin ? y : 0)) * pl.X * CIN + c * 16;
                const int64_t zstep = (int64_t)pl.Y * pl.X * CIN;
                int zr = 0, x = j >> 1;
                const int h = j & 1;
                for (int i = j; i < items; i += kLoaders, x += kLoaders / 2) {
                    while (x >= pl.P) {
                        x -= pl.P;
                        ++zr;
                    }
                    const int gx = q.x0 + x - 1, gz = q.z0 + zr - 1;
                    const bool inside = yin && gx >= 0 && gx < pl.X && gz >= 0 && gz < pl.Z;
                    const __nv_bfloat16 *src = inside ? row + gz * zstep + (int64_t)gx * CIN + h * 8 : in;
                    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(dst0 + h * pl.plane + (i >> 1) * 16),
                                 "l"(src), "r"(inside ? 16 : 0)
                                 : "memory");
                }
                asm volatile("cp.async.commit_group;\n" ::: "memory");
                if (it >= lag) {
                    if (lag == 2)
                        asm volatile("cp.async.wait_group 2;\n" ::: "memory");
                    else
                        asm volatile("cp.async.wait_group 1;\n" ::: "memory");
                    hand_over(it - lag);
                }
            }
        }
        asm volatile("cp.async.wait_all;\n" ::: "memory");
        if (ok)
            for (int i = it > lag ? it - lag : 0; i < it; ++i) hand_over(i);
        else if (lane == 0)
            fail();
    } else if (warp == 0) {
        const uint32_t t0 = __shfl_sync(0xffffffffu, tmem, 0), on = lane == 0;
        constexpr uint32_t kHi = (128u >> 4) | (1u << 14);
        const uint32_t a_base = ((ring >> 4) & 0x3FFF) | (uint32_t)(pl.plane >> 4) << 16;
        const uint32_t b_base = ((wbase >> 4) & 0x3FFF) | (uint32_t)(9 * CO) << 16;
        int it = 0, step = 0;   // stages; input lines (the epilogue clears the accumulators before the first)
        bool ok = true;
        for (int k = 0; k < mine && ok; ++k) {
            const Block q = block_at(k);
            for (int line = 0; line < q.ny + 2 && ok; ++line, ++step) {
                ok = __all_sync(0xffffffffu, tc::mbar_wait(tc::smem_u32(&drained), (uint32_t)step & 1u));
                asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
                const int order = (q.y0 + line - 1 + 3) % 3;
                for (int c = 0; c < NCH && ok; ++c, ++it) {
                    const int slot = it % pl.ring;
                    ok = __all_sync(0xffffffffu, tc::mbar_wait(tc::smem_u32(&full[slot]), (uint32_t)(it / pl.ring) & 1u));
                    if (!ok) break;
                    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
                    const uint32_t a0 = a_base + (uint32_t)(slot * (pl.stage >> 4));
                    const uint32_t b0 = b_base + (uint32_t)((order * NCH + c) * 3 * (WBLOCK / 16));
                    for (int zr = 0; zr < pl.TZ + 2; ++zr) {   // input plane z0 + zr - 1
                        const int lo = max(zr - 2, 0), hi = min(zr, pl.TZ - 1);
                        const uint32_t d = t0 + (uint32_t)(lo * 3 * CO), a = a0 + (uint32_t)(zr * pl.P);
                        const uint32_t b = b0 + (uint32_t)((lo - (zr - 2)) * 3 * CO);
                        const uint32_t idesc = tc::instr_desc((hi - lo + 1) * 3 * CO);
#pragma unroll
                        for (int dx = 0; dx < 3; ++dx)
                            tc::mma_lo(d, a + dx, b + dx * (WBLOCK / 16), kHi, idesc, 1u, on);
                    }
                    if (on) tc::mma_commit(tc::smem_u32(&empty[slot]));
                }
                // (on failure too: whoever waits for it is let go once the instructions in flight have ended)
                if (on) {
                    if (!ok) fail();
                    tc::mma_commit(tc::smem_u32(&done));
                }
                __syncwarp();
            }
        }
    } else if (warp >= 4) {
        const int quarter = warp & 3;   // the tensor-memory lanes this warp can read
        const uint32_t tq = tmem + ((uint32_t)(quarter * 32) << 16);
        auto clear = [&](uint32_t col) {
            asm volatile(
                "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1};\n" ::"r"(
                    tq + col),
                "r"(0u)
                : "memory");
        };
        auto hand_back = [&] {
            asm volatile("tcgen05.wait::st.sync.aligned;\n" ::: "memory");
            asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
            asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(tc::smem_u32(&drained)) : "memory");
        };
        float bv[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) bv[i] = bias ? __ldg(bias + co0 + i) : 0.f;
        int step = 0;
        bool ok = true;
        for (int k = 0; k < mine && ok; ++k) {
            const Block q = block_at(k);
            const int pos = quarter * 32 + lane, x = q.x0 + pos;
            const bool xin = pos < pl.TX && x < pl.X;
            // before a block every accumulator is cleared
            for (int col = 0; col < pl.TZ * 3; ++col) clear((uint32_t)(col * CO));
            hand_back();
            for (int line = 0; line < q.ny + 2; ++line, ++step) {
                ok = tc::mbar_wait(tc::smem_u32(&done), (uint32_t)step & 1u) && !*(volatile int *)&failed;
                if (!__all_sync(0xffffffffu, ok)) {
                    ok = false;
                    if (lane == 0) fail();
                    break;
                }
                asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
                // the input line y is in: the output line y - 1 is complete
                const int yo = q.y0 + line - 2, slot = (yo + 3) % 3;
                // After a block's last line nothing is cleared here: the next block begins by clearing every
                // accumulator, and after the last block the tensor memory is given back, by when every store
                // to it has been waited for (hand_back does, so no clearing goes without one).
                const bool more = line + 1 < q.ny + 2;
                for (int zo = 0; zo < pl.TZ; ++zo) {
                    const uint32_t col = (uint32_t)((zo * 3 + slot) * CO);
                    if (line >= 2 && q.z0 + zo < pl.Z) {
                        float acc[16];
                        __syncwarp();
                        tc::tmem_ld16(tq + col, acc);
                        if (xin) {
                            const int64_t vo = (((int64_t)q.b * pl.Z + q.z0 + zo) * pl.Y + yo) * pl.X + x;
                            __nv_bfloat16 m16[16];
                            if (MASK) {
                                const uint4 *mp = reinterpret_cast<const uint4 *>(mask + vo * COUT + co0);
                                *reinterpret_cast<uint4 *>(m16) = __ldg(mp);
                                *reinterpret_cast<uint4 *>(m16 + 8) = __ldg(mp + 1);
                            }
                            uint32_t packed[8];
#pragma unroll
                            for (int i = 0; i < 16; i += 2) {
                                float lo = acc[i] + bv[i], hi = acc[i + 1] + bv[i + 1];
                                if (RELU) {
                                    lo = fmaxf(lo, 0.f);
                                    hi = fmaxf(hi, 0.f);
                                }
                                if (MASK) {
                                    if (!(__bfloat162float(m16[i]) > 0.f)) lo = 0.f;
                                    if (!(__bfloat162float(m16[i + 1]) > 0.f)) hi = 0.f;
                                }
                                const __nv_bfloat162 pr = __floats2bfloat162_rn(lo, hi);
                                packed[i / 2] = *reinterpret_cast<const uint32_t *>(&pr);
                            }
                            uint4 *op = reinterpret_cast<uint4 *>(out + vo * COUT + co0);
                            op[0] = make_uint4(packed[0], packed[1], packed[2], packed[3]);
                            op[1] = make_uint4(packed[4], packed[5], packed[6], packed[7]);
                        }
                    }
                    __syncwarp();
                    if (more) clear(col);
                }
                // the next line's instructions add to every slot
                if (more) hand_back();
            }
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    if (warp == 0) {
        asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(pl.cols) : "memory");
    }
}

#define OMB_TC_SHAPES(X) X(16, 16) X(16, 32) X(32, 32) X(32, 64) X(64, 64) X(96, 32) X(48, 16) \
    X(32, 16) X(64, 32) X(32, 96) X(16, 48)

// Dynamic shared memory of a CTA that leaves room for a second one (228 KB per
// SM, 1 KB of it per CTA reserved and 1 KB static).
constexpr int kHalfSmem = 111 * 1024;

// Block shape of a convolution: the least estimated time per output voxel over
// the blocks that fit.  The estimate counts an instruction as 32 clocks for its
// 4 KB of A plus one per 4 columns (timed alone it takes about 128 whatever its
// columns, see k_conv3d_lines: the estimate leans to fewer columns, that is
// planes, than that would; shapes planned with 128 have not been timed); a
// staged 16-byte row costs the loaders about a third; two CTAs on an SM (half
// the shared memory and tensor-memory columns each) hide the epilogue, and a
// last wave that is partly empty counts in full.
static ConvPlan conv_plan(int cin, int co, int groups, int X, int Y, int Z, int B) {
    ConvPlan best{};
    double best_cost = 1e300;
    const int nch = cin / 16, wbytes = nch * 9 * 3 * co * 32;
    for (int occ = 2; occ >= 1; --occ) {
        const int max_cols = occ == 2 ? 256 : 512, max_smem = occ == 2 ? kHalfSmem : 226 * 1024;
        for (int ty = 1; ty <= 32 && (ty <= Y || ty == 1); ++ty)
            for (int tz = 1; tz <= 8 && (tz <= Z || tz == 1); ++tz) {
                ConvPlan p{X, Y, Z, B};
                p.ntx = (X + 127) / 128;
                p.TX = (X + p.ntx - 1) / p.ntx;
                p.TY = ty;
                p.TZ = tz;
                p.P = p.TX + 2;
                p.S = p.TX == 128 ? p.P : 128;
                p.T = p.TX == 128 ? ty : ((ty - 1) * p.P + p.TX + 127) / 128;
                if (p.T * tz * co > max_cols) continue;
                for (p.cols = 32; p.cols < p.T * tz * co;) p.cols *= 2;
                p.plane = ((ty + 2) * p.P * 16 + 127) / 128 * 128;
                p.stage = 2 * p.plane;
                // rows past the plane are read by the last M tile and dropped
                const int over = ((p.T - 1) * p.S + 128 + 2 * p.P + 2) * 16;
                const int pad = over > p.plane ? over - p.plane : 0;
                p.ring = 4;
                while (p.ring > 1 && wbytes + p.ring * p.stage + pad > max_smem) --p.ring;
                if (p.ring < 2) continue;
                p.smem = wbytes + p.ring * p.stage + pad;
                p.nty = (Y + ty - 1) / ty;
                p.ntz = (Z + tz - 1) / tz;
                const int64_t tiles = (int64_t)p.ntx * p.nty * p.ntz * B;
                if (tiles > 0x7fffffff / (10 * nch)) continue;   // (stage counters are 32-bit)
                p.tiles = (int)tiles;
                const double mma = (double)(tz + 2) * nch * 9 * p.T * (32 + co * 0.75 * tz / (tz + 2));
                const double load = 0.35 * (tz + 2) * nch * 2 * (ty + 2) * p.P;
                const double epi = 60.0 * p.T * tz * co / 16;
                const double busy = (mma > load ? mma : load) * (p.ring > 2 ? 1.0 : 1.2);
                const double per = occ == 2 ? (busy > epi ? busy : epi) : busy + epi;
                const double slots = (double)num_sms() * occ;
                const double cost = ceil(tiles * (double)groups / slots) * slots * per / occ;
                if (cost < best_cost * (occ == 2 ? 1.0 : 0.999)) {
                    best_cost = cost;
                    best = p;
                }
            }
    }
    return best;
}

template <int CIN, int COUT, int CO, bool RELU, bool MASK>
static int conv_launch(const ConvPlan &pl, const __nv_bfloat16 *in, const __nv_bfloat16 *w, const float *bias,
                       __nv_bfloat16 *out, const __nv_bfloat16 *mask, cudaStream_t st) {
    auto kernel = k_conv3d_tc<CIN, COUT, CO, RELU, MASK>;
    OMB_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, pl.smem));
    const int occ = pl.smem <= kHalfSmem && pl.cols <= 256 ? 2 : 1;
    const int slots = num_sms() * occ / (COUT / CO);
    const int grid = pl.tiles < slots ? pl.tiles : slots;
    kernel<<<dim3(grid, COUT / CO), 256, pl.smem, st>>>(pl, in, w, bias, out, mask);
    OMB_LAUNCH_CHECK("tcgen05 conv launch");
    return OMB_OK;
}

// Block shape of k_conv3d_lines: the least estimated tensor-core time over what
// fits (three instructions of 128 clocks per input line and chunk, an epilogue of
// about 250 clocks per output line that only a second CTA on the SM hides).
static LinePlan line_plan(int cin, int groups, int X, int Y, int Z, int B) {
    LinePlan best{};
    double best_cost = 1e300;
    const int nch = cin / 16, wbytes = 3 * nch * 3 * 9 * 16 * 32;
    for (int occ = 2; occ >= 1; --occ)
        for (int tz = 1; tz <= 10 && (tz <= Z || tz == 1); ++tz) {
            LinePlan p{X, Y, Z, B};
            p.ntx = (X + 127) / 128;
            p.TX = (X + p.ntx - 1) / p.ntx;
            p.TZ = tz;
            p.P = p.TX + 2;
            p.occ = occ;
            if (tz * 48 > (occ == 2 ? 256 : 512)) continue;
            for (p.cols = 32; p.cols < tz * 48;) p.cols *= 2;
            p.plane = ((tz + 2) * p.P * 16 + 127) / 128 * 128;
            p.stage = 2 * p.plane;
            const int pad = 128 * 16;   // the last line's M = 128 rows read past it
            for (p.ring = 4; p.ring >= 2 && wbytes + p.ring * p.stage + pad > (occ == 2 ? kHalfSmem : 226 * 1024);) --p.ring;
            if (p.ring < 2) continue;
            p.smem = wbytes + p.ring * p.stage + pad;
            p.ntz = (Z + tz - 1) / tz;
            const int slots = num_sms() * occ / groups;
            const int64_t columns = (int64_t)p.ntx * p.ntz * B;
            for (int nys = 1; nys <= Y && nys <= 64; ++nys) {
                p.YS = (Y + nys - 1) / nys;
                p.nys = (Y + p.YS - 1) / p.YS;
                const int64_t tiles = columns * p.nys;
                if (tiles > 0x7fffffff / 4096 || (int64_t)(p.YS + 2) * nch > 0x7fffff) continue;
                p.tiles = (int)tiles;
                const double mma = (double)(p.YS + 2) * nch * (tz + 2) * 3 * 128, epi = (double)(p.YS + 2) * (400 + 250 * tz);
                const double per = occ == 2 ? (2 * mma > mma + epi ? 2 * mma : mma + epi) : mma + epi;
                const double cost = (double)((tiles + slots - 1) / slots) * per;
                if (cost < best_cost) {
                    best_cost = cost;
                    best = p;
                }
            }
        }
    return best;
}

template <int CIN, int COUT, bool RELU, bool MASK>
static int lines_launch(const LinePlan &pl, const __nv_bfloat16 *in, const __nv_bfloat16 *w, const float *bias,
                        __nv_bfloat16 *out, const __nv_bfloat16 *mask, cudaStream_t st) {
    auto kernel = k_conv3d_lines<CIN, COUT, RELU, MASK>;
    OMB_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, pl.smem));
    const int slots = num_sms() * pl.occ / (COUT / 16);
    const int grid = pl.tiles < slots ? pl.tiles : slots;
    kernel<<<dim3(grid, COUT / 16), 256, pl.smem, st>>>(pl, in, w, bias, out, mask);
    OMB_LAUNCH_CHECK("tcgen05 conv launch");
    return OMB_OK;
}

template <int CIN, int COUT>
static int conv_shape(const __nv_bfloat16 *in, const __nv_bfloat16 *w, const float *bias, __nv_bfloat16 *out,
                      const __nv_bfloat16 *mask, int relu, int X, int Y, int Z, int B, cudaStream_t st) {
    // Lines that fill more than half of M, up to 48 channels on either side (the
    // network's full-resolution layers): the kernel that marches along them.
    // Shorter lines would leave most of M empty there, and wider layers' weights
    // do not fit in three orders.
    if constexpr (CIN <= 48 && COUT <= 48) {
        const int ntx = (X + 127) / 128, tx = (X + ntx - 1) / ntx;
        if (tx > 64) {
            static thread_local LinePlan lines[8];
            static thread_local int at = 0;
            const LinePlan *lp = nullptr;
            for (const LinePlan &p : lines)
                if (p.tiles > 0 && p.X == X && p.Y == Y && p.Z == Z && p.B == B) lp = &p;
            if (!lp) {
                lines[at] = line_plan(CIN, COUT / 16, X, Y, Z, B);
                lp = &lines[at];
                at = (at + 1) % 8;
            }
            if (lp->tiles > 0) {
                const LinePlan p = *lp;
                if (mask) return lines_launch<CIN, COUT, false, true>(p, in, w, bias, out, mask, st);
                if (relu) return lines_launch<CIN, COUT, true, false>(p, in, w, bias, out, mask, st);
                return lines_launch<CIN, COUT, false, false>(p, in, w, bias, out, mask, st);
            }
        }
    }
    // output channels of a CTA: all of them up to 48 (their weights and three
    // planes of accumulators must fit), else thirds or halves
    constexpr int CO = COUT <= 48 ? COUT : (COUT % 48 == 0 ? 48 : 32);
    // the plans of the last sizes this thread used (the search takes some
    // microseconds; a plan depends on the sizes alone)
    static thread_local ConvPlan plans[8];
    static thread_local int next = 0;
    const ConvPlan *found = nullptr;
    for (const ConvPlan &p : plans)
        if (p.tiles > 0 && p.X == X && p.Y == Y && p.Z == Z && p.B == B) found = &p;
    if (!found) {
        plans[next] = conv_plan(CIN, CO, COUT / CO, X, Y, Z, B);
        found = &plans[next];
        next = (next + 1) % 8;
    }
    const ConvPlan pl = *found;
    if (pl.tiles == 0) return set_error(OMB_ERR_UNSUPPORTED, "conv volume too large");
    if (mask) return conv_launch<CIN, COUT, CO, false, true>(pl, in, w, bias, out, mask, st);
    if (relu) return conv_launch<CIN, COUT, CO, true, false>(pl, in, w, bias, out, mask, st);
    return conv_launch<CIN, COUT, CO, false, false>(pl, in, w, bias, out, mask, st);
}

int unet_conv_tc(int cin, int cout, const void *in, const void *w, const float *bias, void *out, const void *mask,
                 int relu, int X, int Y, int Z, int B, cudaStream_t st) {
    if (X <= 0 || Y <= 0 || Z <= 0 || B <= 0) return set_error(OMB_ERR_INVALID, "bad conv volume");
    const auto *i = static_cast<const __nv_bfloat16 *>(in), *wt = static_cast<const __nv_bfloat16 *>(w),
               *mk = static_cast<const __nv_bfloat16 *>(mask);
    auto *o = static_cast<__nv_bfloat16 *>(out);
#define X(ci, co) \
    if (cin == ci && cout == co) return conv_shape<ci, co>(i, wt, bias, o, mk, relu, X, Y, Z, B, st);
    OMB_TC_SHAPES(X)
#undef X
    return set_error(OMB_ERR_UNSUPPORTED, "conv shape " + std::to_string(cin) + "->" + std::to_string(cout) +
                                              " is not built");
}

// ---------------------------------------------------------------------------
// Weight gradient on the tensor cores.  dW[tap][co][ci] = sum_v dz[v][co]
// in[v + off(tap)][ci] is a GEMM with the voxels as its K dimension:
// D[m][co] = sum_v A[m][v] B[co][v], the rows m = tap * CIN + ci of all 27
// taps taken 128 at a time (grid.y), B = dz.  A CTA reduces `per_cta`
// voxels (grid.x) in stages of 32 (two K = 16 instructions) and adds its
// 128 x COUT partial sums to dW with FP32 atomics.  Both operands are staged
// MN-major (the transpose bits of the instruction descriptor): 8 consecutive
// rows of A are 8 consecutive channels of one tap-shifted input voxel and 8
// consecutive rows of B 8 output channels of one dz voxel, so every 16-byte
// global load lands as one 16-byte row of a core matrix (8 voxels x 16
// bytes).  Core matrix (row group g, voxel group k) lies at g * 256 + k *
// 128 bytes: a row-group stride of 256 (SBO) and a voxel-group stride of 128
// (LBO), the same address map as the K-major operands of the forward kernel,
// so the MMA reads stay inside each 128-row x 16-voxel sub-tile.
// ---------------------------------------------------------------------------
template <int CIN, int COUT>
__global__ void __launch_bounds__(128) k_conv3d_wgrad_tc(const __nv_bfloat16 *__restrict__ in,
                                                         const __nv_bfloat16 *__restrict__ dz,
                                                         float *__restrict__ dw, int X, int Y, int Z, int64_t nvox,
                                                         int per_cta) {
    static_assert(CIN % 8 == 0 && COUT % 16 == 0 && COUT <= 128, "channel counts");
    constexpr int MROWS = 27 * CIN;
    constexpr int KV = 32;                       // voxels per stage
    constexpr int A_SUB = tc::kM * 16 * 2;       // one K = 16 sub-tile of A (bytes)
    constexpr int B_SUB = COUT * 16 * 2;         // of B
    constexpr int NG = COUT / 8;                 // 8-channel groups of B
    constexpr int TMEM_COLS = COUT <= 32 ? 32 : (COUT <= 64 ? 64 : 128);
    __shared__ __align__(1024) uint8_t sA[2][2 * A_SUB];
    __shared__ __align__(1024) uint8_t sB[2][2 * B_SUB];
    __shared__ __align__(8) uint64_t bars[2];
    __shared__ uint32_t tmem_base;
    __shared__ short4 vc[2][KV];  // (x, y, z, inside) of each staged voxel
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    if (tid == 0) {
        tc::mbar_init(tc::smem_u32(&bars[0]), 1);
        tc::mbar_init(tc::smem_u32(&bars[1]), 1);
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(tc::smem_u32(&tmem_base)),
                     "r"(TMEM_COLS)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    const uint32_t tmem = tmem_base;
    const int m0 = blockIdx.y * tc::kM;
    // this thread's A row group (the same in every stage): tap, first channel and the tap's voxel offset
    const int ga = tid & 15, ma = m0 + ga * 8;
    const bool arow = ma < MROWS;
    const int tapa = arow ? ma / CIN : 0, cia = arow ? ma - tapa * CIN : 0;
    const int ddx = tapa % 3 - 1, ddy = (tapa / 3) % 3 - 1, ddz = tapa / 9 - 1;
    const int64_t doff = ((int64_t)ddz * Y + ddy) * X + ddx;
    const int64_t v_begin = (int64_t)blockIdx.x * per_cta;
    const int64_t v_end = min(v_begin + (int64_t)per_cta, nvox);
    const int nst = (int)((v_end - v_begin + KV - 1) / KV);
    // A and B both MN-major (transpose bits 15 and 16)
    const uint32_t idesc = tc::instr_desc(COUT) | (1u << 15) | (1u << 16);
    // (x, y, z) of voxel v0 + k of a stage, in 32-bit arithmetic (the launch keeps nvox below 2^31)
    auto coords = [&](int st_idx, int buf) {
        if (tid < KV) {
            const int64_t v = v_begin + (int64_t)st_idx * KV + tid;
            short4 c = make_short4(0, 0, 0, 0);
            if (v < v_end) {
                int q = (int)v;
                c.x = (short)(q % X);
                q /= X;
                c.y = (short)(q % Y);
                q /= Y;
                c.z = (short)(q % Z);
                c.w = 1;
            }
            vc[buf][tid] = c;
        }
    };
    int issued = 0;
    bool ok = true;
    if (nst > 0) coords(0, 0);
    for (int ks = 0; ks < nst; ++ks) {
        const int s = ks & 1;
        if (ks >= 2) {
            if (!tc::mbar_wait(tc::smem_u32(&bars[s]), (uint32_t)((ks >> 1) - 1) & 1u)) ok = false;
        }
        if (!__syncthreads_and(ok)) {
            ok = false;
            break;
        }
        if (ks + 1 < nst) coords(ks + 1, s ^ 1);  // read after the next barrier
        const int64_t v0 = v_begin + (int64_t)ks * KV;
        // A: 32 voxels x 16 row groups, 4 per thread (the voxel k = idx / 16, this thread's row group ga); the
        // voxel coordinates come from the table the previous step filled
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int k = (tid >> 4) + 8 * j;
            const short4 c = vc[s][k];
            uint4 val = make_uint4(0, 0, 0, 0);
            if (arow && c.w) {
                const int xs = c.x + ddx, ys = c.y + ddy, zs = c.z + ddz;
                if (xs >= 0 && xs < X && ys >= 0 && ys < Y && zs >= 0 && zs < Z)
                    val = __ldg(reinterpret_cast<const uint4 *>(in + (v0 + k + doff) * CIN + cia));
            }
            const int kk = k & 15;
            *reinterpret_cast<uint4 *>(sA[s] + (k >> 4) * A_SUB + ga * tc::kCoreGroup + (kk >> 3) * tc::kKHalf +
                                       (kk & 7) * 16) = val;
        }
        // B: 32 voxels x NG channel groups
        for (int idx = tid; idx < KV * NG; idx += 128) {
            const int k = idx / NG, g = idx - k * NG;
            const int64_t v = v0 + k;
            uint4 val = make_uint4(0, 0, 0, 0);
            if (v < v_end) val = __ldg(reinterpret_cast<const uint4 *>(dz + v * COUT + g * 8));
            const int kk = k & 15;
            *reinterpret_cast<uint4 *>(sB[s] + (k >> 4) * B_SUB + g * tc::kCoreGroup + (kk >> 3) * tc::kKHalf +
                                       (kk & 7) * 16) = val;
        }
        asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
        __syncthreads();
        if (tid == 0) {
            asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
#pragma unroll
            for (int sub = 0; sub < 2; ++sub)
                tc::mma_issue(tmem, tc::smem_desc(tc::smem_u32(sA[s] + sub * A_SUB)),
                              tc::smem_desc(tc::smem_u32(sB[s] + sub * B_SUB)), idesc, (ks > 0 || sub > 0) ? 1u : 0u);
            tc::mma_commit(tc::smem_u32(&bars[s]));
        }
        issued = ks + 1;
    }
    if (ok && nst > 0) {
        const int last = nst - 1;
        if (!tc::mbar_wait(tc::smem_u32(&bars[last & 1]), (uint32_t)(last >> 1) & 1u)) ok = false;
    }
    if (!ok) {
        if (tid == 0) atomicExch(&g_unet_error, 1);
        if (issued > 0) tc::mbar_wait(tc::smem_u32(&bars[(issued - 1) & 1]), (uint32_t)((issued - 1) >> 1) & 1u);
    }
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    if (ok && nst > 0) {
        // row m of D = TMEM lane m: warp w holds rows 32w..32w+31
        const int m = m0 + warp * 32 + lane;
        const bool mrow = m < MROWS;
        const int tap = mrow ? m / CIN : 0, ci = mrow ? m - tap * CIN : 0;
        float *d = dw + (int64_t)tap * COUT * CIN + ci;
#pragma unroll
        for (int c0 = 0; c0 < COUT; c0 += 16) {
            float acc[16];
            tc::tmem_ld16(tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)c0, acc);
            if (mrow) {
#pragma unroll
                for (int i = 0; i < 16; ++i) atomicAdd(d + (c0 + i) * CIN, acc[i]);
            }
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(TMEM_COLS) : "memory");
}

int unet_conv_wgrad_tc(int cin, int cout, const void *in, const void *dz, float *dw, int X, int Y, int Z, int B,
                       cudaStream_t st) {
    if (X <= 0 || Y <= 0 || Z <= 0 || B <= 0) return set_error(OMB_ERR_INVALID, "bad conv volume");
    const int64_t nvox = (int64_t)X * Y * Z * B;
    const int per_cta = 32 * 256;  // voxels per CTA (a multiple of the 32-voxel stage)
    const int64_t chunks = (nvox + per_cta - 1) / per_cta;
    if (nvox > 2147483647 || X > 32767 || Y > 32767 || Z > 32767)
        return set_error(OMB_ERR_UNSUPPORTED, "wgrad volume too large (2^31 voxels, 32767 per axis)");
    const auto *i = static_cast<const __nv_bfloat16 *>(in), *d = static_cast<const __nv_bfloat16 *>(dz);
#define X(ci, co)                                                                                             \
    if (cin == ci && cout == co) {                                                                            \
        dim3 grid((unsigned)chunks, (unsigned)((27 * ci + tc::kM - 1) / tc::kM));                              \
        k_conv3d_wgrad_tc<ci, co><<<grid, 128, 0, st>>>(i, d, dw, X, Y, Z, nvox, per_cta);                     \
        OMB_LAUNCH_CHECK("tcgen05 wgrad launch");                                                             \
        return OMB_OK;                                                                                        \
    }
    OMB_TC_SHAPES(X)
#undef X
    return set_error(OMB_ERR_UNSUPPORTED, "wgrad shape " + std::to_string(cin) + "->" + std::to_string(cout) +
                                              " is not built");
}

}  // namespace omb

extern "C" {

int omb_unet_conv_tc(int32_t cin, int32_t cout, const void *in, const void *w, const float *bias, void *out,
                     const void *relu_mask, int32_t relu, int32_t X, int32_t Y, int32_t Z, int32_t B, void *stream) {
    if (!in || !w || !out) return omb::set_error(OMB_ERR_INVALID, "NULL buffer passed to omb_unet_conv_tc");
    return omb::unet_conv_tc(cin, cout, in, w, bias, out, relu_mask, relu, X, Y, Z, B, (cudaStream_t)stream);
}

int omb_unet_conv_wgrad_tc(int32_t cin, int32_t cout, const void *in, const void *dz, float *dw, int32_t X,
                           int32_t Y, int32_t Z, int32_t B, void *stream) {
    if (!in || !dz || !dw) return omb::set_error(OMB_ERR_INVALID, "NULL buffer passed to omb_unet_conv_wgrad_tc");
    return omb::unet_conv_wgrad_tc(cin, cout, in, dz, dw, X, Y, Z, B, (cudaStream_t)stream);
}

int omb_unet_take_error(int32_t *out_host) {
    if (!out_host) return omb::set_error(OMB_ERR_INVALID, "output pointer is NULL");
    int v = 0;
    const cudaError_t e = cudaMemcpyFromSymbol(&v, omb::g_unet_error, sizeof(int));
    if (e != cudaSuccess) return omb::cuda_fail(e, "read conv error flag");
    const int zero = 0;
    const cudaError_t e2 = cudaMemcpyToSymbol(omb::g_unet_error, &zero, sizeof(int));
    if (e2 != cudaSuccess) return omb::cuda_fail(e2, "clear conv error flag");
    *out_host = v;
    return OMB_OK;
}

}  // extern "C"
