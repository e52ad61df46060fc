// Kernels of the learned OSEM warm start: a small 3-D U-Net (3x3x3
// convolutions, BF16 weights and activations, FP32 accumulation) trained and
// run on the GPU by these kernels alone.
//
// Layouts: activations are channels-last BF16, [B][Z][Y][X][C] with C a
// multiple of 16; conv weights are BF16 [27][Cout][Cin] (tap-major, input
// channels contiguous), tap = (dz+1)*9 + (dy+1)*3 + (dx+1); biases FP32.
//
// Convolutions are implicit GEMMs on the tensor cores (mma.sync m16n8k16,
// BF16 in, FP32 accumulate):
//   forward  out[v][co] = relu(bias[co] + sum_tap sum_ci in[v+off(tap)][ci] W[tap][co][ci])
//   dgrad    the same kernel on the flipped, transposed weights
//            W'[tap][ci][co] = W[26 - tap][co][ci] (off(26 - tap) = -off(tap)),
//            with the next ReLU's derivative fused as a mask on the output
//   wgrad    dW[tap][co][ci] = sum_v dz[v][co] in[v+off(tap)][ci]: voxels are
//            the GEMM's K; lines of voxels with their halo staged once in shared
//            memory and read transposed and shifted with ldmatrix.trans, partial
//            sums added with FP32 atomics.
#include <cuda_bf16.h>

#include <initializer_list>

#include "kernels.h"
#include "../../include/omega_b200_unet.h"

namespace omb {

using bf16 = __nv_bfloat16;

__device__ __forceinline__ void mma_bf16(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                         uint32_t b0, uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
        "{%0,%1,%2,%3};\n"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

__device__ __forceinline__ uint32_t ld_pair(const bf16 *p) { return __ldg(reinterpret_cast<const unsigned int *>(p)); }

__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
    const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<const uint32_t *>(&v);
}

// ---------------------------------------------------------------------------
// Forward / dgrad convolution.  Block = 4 warps = 64 consecutive voxels along
// x of one (y, z, batch) row; warp = 16 voxels x COUT channels.
// ---------------------------------------------------------------------------
template <int CIN, int COUT, bool RELU, bool MASK>
__global__ void __launch_bounds__(128) k_conv3d(const bf16 *__restrict__ in, const bf16 *__restrict__ w,
                                                const float *__restrict__ bias, bf16 *__restrict__ out,
                                                const bf16 *__restrict__ mask, int X, int Y, int Z) {
    static_assert(CIN % 16 == 0 && COUT % 8 == 0, "channel counts");
    constexpr int NT = COUT / 8;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int g = lane >> 2, t = lane & 3;
    const int y = blockIdx.y;
    const int z = blockIdx.z % Z, b = blockIdx.z / Z;
    const int xbase = blockIdx.x * 64 + warp * 16;
    const int xr0 = xbase + g, xr1 = xbase + g + 8;  // the two A rows of this thread
    const int64_t row_off = (((int64_t)b * Z + z) * Y + y) * X;
    float acc[NT][4];
#pragma unroll
    for (int j = 0; j < NT; ++j) acc[j][0] = acc[j][1] = acc[j][2] = acc[j][3] = 0.f;
    if (xbase < X) {
        for (int tap = 0; tap < 27; ++tap) {
            const int dz = tap / 9 - 1, dy = (tap / 3) % 3 - 1, dx = tap % 3 - 1;
            const int zz = z + dz, yy = y + dy;
            if (zz < 0 || zz >= Z || yy < 0 || yy >= Y) continue;
            const int x0 = xr0 + dx, x1 = xr1 + dx;
            const bool v0 = x0 >= 0 && x0 < X, v1 = x1 >= 0 && x1 < X;
            const int64_t base = (((int64_t)b * Z + zz) * Y + yy) * X;
            const bf16 *p0 = in + (base + (v0 ? x0 : 0)) * CIN + 2 * t;
            const bf16 *p1 = in + (base + (v1 ? x1 : 0)) * CIN + 2 * t;
            const bf16 *wt = w + (int64_t)tap * COUT * CIN + (int64_t)g * CIN + 2 * t;
#pragma unroll
            for (int c = 0; c < CIN; c += 16) {
                const uint32_t a0 = v0 ? ld_pair(p0 + c) : 0u, a1 = v1 ? ld_pair(p1 + c) : 0u;
                const uint32_t a2 = v0 ? ld_pair(p0 + c + 8) : 0u, a3 = v1 ? ld_pair(p1 + c + 8) : 0u;
#pragma unroll
                for (int j = 0; j < NT; ++j) {
                    const bf16 *wj = wt + (int64_t)j * 8 * CIN + c;
                    mma_bf16(acc[j], a0, a1, a2, a3, ld_pair(wj), ld_pair(wj + 8));
                }
            }
        }
    }
    // epilogue: rows g and g+8, channels j*8 + 2t, +1
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const int xr = h ? xr1 : xr0;
        if (xr >= X) continue;
        const int64_t v = row_off + xr;
#pragma unroll
        for (int j = 0; j < NT; ++j) {
            const int co = j * 8 + 2 * t;
            float lo = acc[j][2 * h], hi = acc[j][2 * h + 1];
            if (bias) {
                lo += __ldg(bias + co);
                hi += __ldg(bias + co + 1);
            }
            if (RELU) {
                lo = fmaxf(lo, 0.f);
                hi = fmaxf(hi, 0.f);
            }
            if (MASK) {
                const __nv_bfloat162 m = *reinterpret_cast<const __nv_bfloat162 *>(mask + v * COUT + co);
                if (!(__low2float(m) > 0.f)) lo = 0.f;
                if (!(__high2float(m) > 0.f)) hi = 0.f;
            }
            *reinterpret_cast<uint32_t *>(out + v * COUT + co) = pack_bf16(lo, hi);
        }
    }
}

// ---------------------------------------------------------------------------
// Weight gradient.  A stage is TY lines of dz with a one-voxel halo in x and
// TY + 2 lines of the input plane dz away (blockIdx.y picks dz = -1, 0, 1),
// both as planes of 8 channels with 16-byte rows in voxel order, copied with
// cp.async into a ring of stages; ldmatrix reads any 8 consecutive voxels
// without bank conflicts.  A shift by dx is put on the dz operand and a shift
// by dy on the input, so the 9 taps of a stage need 3 + 3 operand loads per 16
// voxels.  A warp holds the three dx taps of one dy for MTW x NTW tiles of 16
// output x 8 input channels (up to 96 accumulators); MS x NS warps cover the
// channels and KS of them share the voxels.  Bound by the tensor cores'
// m16n8k16 rate with the operand loads beside it; one tap per block of a 27-fold
// grid, as it was before, staged both operands again for each tap
// (training step at 128 x 128 x 64 x 4: 19.1 -> 11.8 ms).  The copies and the operand
// addresses advance without divisions or line loops: at that size 16 -> 16 channels
// 437 to 408 us, 48 -> 16 1106 to 1063, 16 -> 48 998 to 940.
// ---------------------------------------------------------------------------
struct WgradPlan {
    int X, Y, Z, B;
    int TX, TY;            // voxels of a stage (TX a multiple of 16; past the line's end the input is zero)
    int ntx, nty, tiles;   // stages in all
    int ring;              // stages in shared memory
    int in_plane, dz_plane, dz_off, stage;   // bytes
    int flush;             // stages whose sums a warp adds up before they go to dw
    uint32_t inv;          // 65536 / (TX / 16) + 1: s * inv >> 16 is s / (TX / 16) for every group s of a stage
    int smem;
};

__device__ __forceinline__ void ldmatrix_x4_trans(uint32_t (&r)[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];\n"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(addr)
                 : "memory");
}

template <int CIN, int COUT>
struct WgradShape {
    static constexpr int MT = COUT / 16, NT = CIN / 8;
    static constexpr int MTW = MT <= 3 ? MT : 2, NTW = NT <= 2 ? NT : (MTW == 1 && NT == 6 ? 6 : (MTW == 3 ? 2 : 4));
    static constexpr int MS = MT / MTW, NS = NT / NTW;
    static constexpr int kSums = 3 * MTW * NTW * 4;   // accumulators of a thread
    static constexpr int KS = MS * NS >= 4 ? 1 : 4 / (MS * NS);
    static constexpr bool kPairs = kSums <= 72;       // (registers)
    static constexpr int kWarps = 3 * MS * NS * KS, kThreads = 32 * kWarps;
    static_assert(MT % MTW == 0 && NT % NTW == 0 && NTW % 2 == 0 && 3 * MTW * NTW * 4 <= 96, "wgrad tiles");
    static_assert(kThreads % (CIN / 8) == 0 && kThreads % (COUT / 8) == 0, "copy loops");
};

template <int CIN, int COUT>
__global__ void __launch_bounds__(WgradShape<CIN, COUT>::kThreads, 1)
    k_conv3d_wgrad(const __grid_constant__ WgradPlan pl, const bf16 *__restrict__ in, const bf16 *__restrict__ dz,
                   float *__restrict__ dw) {
    using S = WgradShape<CIN, COUT>;
    constexpr int MTW = S::MTW, NTW = S::NTW, CI8 = CIN / 8, CO8 = COUT / 8;
    extern __shared__ __align__(128) uint8_t wsmem[];
    const uint32_t base = (uint32_t)__cvta_generic_to_shared(wsmem);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int dy = warp % 3, part = warp / 3;
    const int ks = part % S::KS, ns = part / S::KS % S::NS, ms = part / S::KS / S::NS;
    const int dzi = (int)blockIdx.y - 1;
    const int P = pl.TX + 2;
    float acc[3][MTW][NTW][4];
    auto clear = [&] {
#pragma unroll
        for (int d = 0; d < 3; ++d)
#pragma unroll
            for (int m = 0; m < MTW; ++m)
#pragma unroll
                for (int n = 0; n < NTW; ++n) acc[d][m][n][0] = acc[d][m][n][1] = acc[d][m][n][2] = acc[d][m][n][3] = 0.f;
    };
    clear();
    const int mine = (int)blockIdx.x < pl.tiles ? (pl.tiles - 1 - (int)blockIdx.x) / (int)gridDim.x + 1 : 0;
    auto copy16 = [](uint32_t dst, const bf16 *src, bool ok) {
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(dst), "l"(src), "r"(ok ? 16 : 0) : "memory");
    };
    // 16-byte rows of one operand: this thread's channels are fixed, and it goes from
    // a row to the one `step` rows on without a division
    struct Rows {
        int c, x, line, dx, dl;
    };
    auto rows = [&](int c8, int pitch) {
        const int step = S::kThreads / c8, x = tid / c8;
        return Rows{tid % c8, x % pitch, x / pitch, step % pitch, step / pitch};
    };
    const Rows ri = rows(CI8, pl.TX), rd = rows(CO8, P);
    auto copy_rows = [&](const Rows &r, uint32_t dst, const bf16 *src, int c8, int pitch, int lines, int x0, int y0, bool zin) {
        // src: channels of the plane's voxel 0; x0, y0: voxel of the stage's row 0
        const int chan = c8 * 8;
        int x = r.x, gy = r.line + y0;
        const bf16 *p = src + ((int64_t)gy * pl.X + x0 + x) * chan + r.c * 8;
        const int64_t inc = ((int64_t)r.dl * pl.X + r.dx) * chan, wrap = (int64_t)(pl.X - pitch) * chan;
        const uint32_t end = dst + (uint32_t)(lines * pitch) * 16u;
        for (dst += (uint32_t)(tid / c8) * 16u; dst < end; dst += (uint32_t)(S::kThreads / c8) * 16u) {
            const bool ok = zin && (unsigned)(x0 + x) < (unsigned)pl.X && (unsigned)gy < (unsigned)pl.Y;
            copy16(dst, ok ? p : src, ok);
            x += r.dx;
            gy += r.dl;
            p += inc;
            if (x >= pitch) {
                x -= pitch;
                ++gy;
                p += wrap;
            }
        }
    };
    // requests stage k of this block's sequence
    auto load = [&](int k) {
        int tile = (int)blockIdx.x + k * (int)gridDim.x;
        const int x0 = tile % pl.ntx * pl.TX;
        tile /= pl.ntx;
        const int y0 = tile % pl.nty * pl.TY;
        tile /= pl.nty;
        const int z = tile % pl.Z, b = tile / pl.Z, zi = z + dzi;
        const uint32_t st = base + (uint32_t)(k % pl.ring) * pl.stage;
        const bool zin = zi >= 0 && zi < pl.Z;
        copy_rows(ri, st + ri.c * pl.in_plane, in + ((int64_t)b * pl.Z + (zin ? zi : 0)) * pl.Y * pl.X * CIN, CI8, pl.TX,
                  pl.TY + 2, x0, y0 - 1, zin);
        copy_rows(rd, st + pl.dz_off + rd.c * pl.dz_plane, dz + ((int64_t)b * pl.Z + z) * pl.Y * pl.X * COUT, CO8, P, pl.TY,
                  x0 - 1, y0, true);
        asm volatile("cp.async.commit_group;\n" ::: "memory");
    };
    auto flush = [&] {
        const int g = lane >> 2, t = lane & 3;
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            float *dt = dw + (int64_t)((dzi + 1) * 9 + dy * 3 + d) * COUT * CIN;
#pragma unroll
            for (int m = 0; m < MTW; ++m)
#pragma unroll
                for (int n = 0; n < NTW; ++n) {
                    const int co = (ms * MTW + m) * 16 + g, ci = (ns * NTW + n) * 8 + 2 * t;
                    atomicAdd(dt + co * CIN + ci, acc[d][m][n][0]);
                    atomicAdd(dt + co * CIN + ci + 1, acc[d][m][n][1]);
                    atomicAdd(dt + (co + 8) * CIN + ci, acc[d][m][n][2]);
                    atomicAdd(dt + (co + 8) * CIN + ci + 1, acc[d][m][n][3]);
                }
        }
    };
    for (int k = 0; k < pl.ring - 1; ++k) {
        if (k < mine)
            load(k);
        else
            asm volatile("cp.async.commit_group;\n" ::: "memory");
    }
    // ldmatrix rows of this lane: matrix mi, row rr
    const int mi = lane >> 3, rr = lane & 7;
    const int total = pl.TX / 16 * pl.TY;
    for (int k = 0; k < mine; ++k) {
        if (pl.ring == 3)
            asm volatile("cp.async.wait_group 1;\n" ::: "memory");
        else
            asm volatile("cp.async.wait_group 0;\n" ::: "memory");
        __syncthreads();   // stage k is here for everybody, and everybody is done with stage k - 1
        const uint32_t st = base + (uint32_t)(k % pl.ring) * pl.stage;
        // input: matrices (voxels 0-7 / 8-15) of two channel planes; dz: two planes for each half of the voxels
        const uint32_t ib = st + (ns * NTW + (mi >> 1)) * pl.in_plane + ((mi & 1) * 8 + rr) * 16;
        const uint32_t db = st + pl.dz_off + (ms * MTW * 2 + (mi & 1)) * pl.dz_plane + ((mi >> 1) * 8 + rr) * 16;
        auto fetch = [&](int s, uint32_t (&bq)[NTW / 2][4], uint32_t (&aq)[3][MTW][4]) {
            const int line = (int)((uint32_t)s * pl.inv >> 16);   // s / (TX / 16)
            const uint32_t ia = ib + (uint32_t)(dy * pl.TX + s * 16) * 16u, da = db + (uint32_t)(s * 16 + line * 2) * 16u;
#pragma unroll
            for (int n = 0; n < NTW / 2; ++n) ldmatrix_x4_trans(bq[n], ia + 2 * n * pl.in_plane);
#pragma unroll
            for (int d = 0; d < 3; ++d)
#pragma unroll
                for (int m = 0; m < MTW; ++m)
                    // tap dx = d - 1 pairs input voxel u with dz voxel u - dx, staged at u - dx + 1
                    ldmatrix_x4_trans(aq[d][m], da + (2 - d) * 16 + 2 * m * pl.dz_plane);
        };
        auto multiply = [&](const uint32_t (&bq)[NTW / 2][4], const uint32_t (&aq)[3][MTW][4]) {
#pragma unroll
            for (int d = 0; d < 3; ++d)
#pragma unroll
                for (int m = 0; m < MTW; ++m)
#pragma unroll
                    for (int n = 0; n < NTW; ++n)
                        mma_bf16(acc[d][m][n], aq[d][m][0], aq[d][m][1], aq[d][m][2], aq[d][m][3], bq[n / 2][(n & 1) * 2],
                                 bq[n / 2][(n & 1) * 2 + 1]);
        };
        uint32_t bq[2][NTW / 2][4], aq[2][3][MTW][4];
        int s = ks;
        // a third of the warps of a scheduler requests the stage after next before its groups,
        // a third between them and a third after them, so that the copies' issue does not stop
        // the tensor cores (with two stages they would come too late); all before their groups,
        // at 128 x 128 x 64 x 4: 16 -> 16 channels 408 us, now 304; 48 -> 16 1063, now 759;
        // 16 -> 48 940, now 662
        const int phase = pl.ring == 3 ? (warp >> 2) % 3 : 0;
#pragma unroll 1
        for (int part = 0;; ++part) {
            if (part == phase) {
                if (k + pl.ring - 1 < mine)
                    load(k + pl.ring - 1);
                else
                    asm volatile("cp.async.commit_group;\n" ::: "memory");
            }
            if (part == 2) break;
            const int stop = part == 0 ? total / 2 : total;
            // two groups of 16 voxels at a time, where the registers allow: the operands of the
            // second are on their way while the first's are multiplied
            if constexpr (S::kPairs)
                for (; s + S::KS < stop; s += 2 * S::KS) {
                    fetch(s, bq[0], aq[0]);
                    fetch(s + S::KS, bq[1], aq[1]);
                    multiply(bq[0], aq[0]);
                    multiply(bq[1], aq[1]);
                }
            for (; s < stop; s += S::KS) {
                fetch(s, bq[0], aq[0]);
                multiply(bq[0], aq[0]);
            }
        }
        // sums of at most about 8192 voxels are added up before they go to memory
        if ((k + 1) % pl.flush == 0 && k + 1 < mine) {
            flush();
            clear();
        }
    }
    if (mine > 0) flush();
}

// Bias gradient: db[co] = sum_v dz[v][co] (FP32 atomics per block).
template <int C>
__global__ void k_bias_grad(const bf16 *__restrict__ dz, float *__restrict__ db, int64_t nvox) {
    __shared__ float part[C];
    for (int c = threadIdx.x; c < C; c += blockDim.x) part[c] = 0.f;
    __syncthreads();
    const int c = threadIdx.x % C;
    const int lanes = blockDim.x / C;
    float s = 0.f;
    for (int64_t v = (int64_t)blockIdx.x * lanes + threadIdx.x / C; v < nvox; v += (int64_t)gridDim.x * lanes)
        s += __bfloat162float(dz[v * C + c]);
    atomicAdd(part + c, s);
    __syncthreads();
    for (int cc = threadIdx.x; cc < C; cc += blockDim.x) atomicAdd(db + cc, part[cc]);
}

// d = d * (a > 0) in place (the derivative of a = relu(z) applied to dL/da).
__global__ void k_relu_mask(bf16 *__restrict__ d, const bf16 *__restrict__ a, int64_t n) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        if (!(__bfloat162float(a[i]) > 0.f)) d[i] = __float2bfloat16(0.f);
}

// W'[tap][ci][co] = W[26 - tap][co][ci]
__global__ void k_flip_weights(const bf16 *__restrict__ w, bf16 *__restrict__ wf, int cin, int cout) {
    const int n = 27 * cin * cout;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const int tap = i / (cin * cout), r = i % (cin * cout);
        const int ci = r / cout, co = r % cout;
        wf[i] = w[(int64_t)(26 - tap) * cout * cin + (int64_t)co * cin + ci];
    }
}

// ---------------------------------------------------------------------------
// Resampling and channel plumbing (channels-last BF16)
// ---------------------------------------------------------------------------

// 2x2x2 average pooling: out [B][Z/2][Y/2][X/2][C].
__global__ void k_avgpool2(const bf16 *__restrict__ in, bf16 *__restrict__ out, int X, int Y, int Z, int C,
                           int64_t nout) {
    const int Xo = X / 2, Yo = Y / 2, Zo = Z / 2;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < nout * C; i += (int64_t)gridDim.x * blockDim.x) {
        const int c = (int)(i % C);
        int64_t v = i / C;
        const int x = (int)(v % Xo);
        v /= Xo;
        const int y = (int)(v % Yo);
        v /= Yo;
        const int z = (int)(v % Zo);
        const int64_t b = v / Zo;
        float s = 0.f;
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            const int xx = 2 * x + (k & 1), yy = 2 * y + ((k >> 1) & 1), zz = 2 * z + (k >> 2);
            s += __bfloat162float(in[((((b * Z) + zz) * Y + yy) * X + xx) * C + c]);
        }
        out[i] = __float2bfloat16(0.125f * s);
    }
}

// Backward of the average pooling, accumulated: din[child] += dout[parent] / 8.
__global__ void k_avgpool2_bwd(const bf16 *__restrict__ dout, bf16 *__restrict__ din, int X, int Y, int Z, int C,
                               int64_t nin) {
    const int Xo = X / 2, Yo = Y / 2, Zo = Z / 2;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < nin * C; i += (int64_t)gridDim.x * blockDim.x) {
        const int c = (int)(i % C);
        int64_t v = i / C;
        const int x = (int)(v % X);
        v /= X;
        const int y = (int)(v % Y);
        v /= Y;
        const int z = (int)(v % Z);
        const int64_t b = v / Z;
        const int64_t p = (((b * Zo + z / 2) * Yo + y / 2) * Xo + x / 2) * C + c;
        din[i] = __float2bfloat16(__bfloat162float(din[i]) + 0.125f * __bfloat162float(dout[p]));
    }
}

// Nearest 2x upsampling of `low` ([B][Z/2][Y/2][X/2][Cl]) written into channels
// [0, Cl) of `cat` ([B][Z][Y][X][Cl + Cs]) and `skip` ([..][Cs]) into [Cl, Cl + Cs).
__global__ void k_up_concat(const bf16 *__restrict__ low, const bf16 *__restrict__ skip, bf16 *__restrict__ cat,
                            int X, int Y, int Z, int Cl, int Cs, int64_t nvox) {
    const int C = Cl + Cs;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < nvox * C; i += (int64_t)gridDim.x * blockDim.x) {
        const int c = (int)(i % C);
        const int64_t v = i / C;
        if (c >= Cl) {
            cat[i] = skip[v * Cs + (c - Cl)];
        } else {
            int64_t q = v;
            const int x = (int)(q % X);
            q /= X;
            const int y = (int)(q % Y);
            q /= Y;
            const int z = (int)(q % Z);
            const int64_t b = q / Z;
            cat[i] = low[(((b * (Z / 2) + z / 2) * (Y / 2) + y / 2) * (X / 2) + x / 2) * Cl + c];
        }
    }
}

// Backward of k_up_concat: dlow[parent] = sum of the 8 children's first Cl
// channels; dskip += the remaining Cs channels (added to the gradient that
// already flows into the skip tensor).
__global__ void k_up_concat_bwd(const bf16 *__restrict__ dcat, bf16 *__restrict__ dlow, bf16 *__restrict__ dskip,
                                int X, int Y, int Z, int Cl, int Cs, int64_t nlow, int64_t nvox) {
    const int C = Cl + Cs;
    const int Xl = X / 2, Yl = Y / 2, Zl = Z / 2;
    const int64_t total_low = nlow * Cl, total_skip = nvox * Cs;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total_low + total_skip;
         i += (int64_t)gridDim.x * blockDim.x) {
        if (i < total_low) {
            const int c = (int)(i % Cl);
            int64_t q = i / Cl;
            const int x = (int)(q % Xl);
            q /= Xl;
            const int y = (int)(q % Yl);
            q /= Yl;
            const int z = (int)(q % Zl);
            const int64_t b = q / Zl;
            float s = 0.f;
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                const int xx = 2 * x + (k & 1), yy = 2 * y + ((k >> 1) & 1), zz = 2 * z + (k >> 2);
                s += __bfloat162float(dcat[((((b * Z) + zz) * Y + yy) * X + xx) * C + c]);
            }
            dlow[i] = __float2bfloat16(s);
        } else {
            const int64_t j = i - total_low;
            const int c = (int)(j % Cs);
            const int64_t v = j / Cs;
            dskip[j] = __float2bfloat16(__bfloat162float(dskip[j]) + __bfloat162float(dcat[v * C + Cl + c]));
        }
    }
}

// ---------------------------------------------------------------------------
// The same with 8 channels (16 bytes) per thread, for channel counts that are
// multiples of 8 on 16-byte aligned tensors (every layer of the network).
// These passes move memory only; one 2-byte element and up to four 64-bit
// divisions per thread kept them at a tenth of its bandwidth
// (training step at 128 x 128 x 64 x 4: 11.8 -> 9.0 ms).
// ---------------------------------------------------------------------------
struct Vox {
    int x, y, z;
    int64_t b;
};
__device__ __forceinline__ Vox voxel_at(int64_t v, int X, int Y, int Z) {
    Vox q;
    if (v <= 0xffffffffll) {   // (a 64-bit division is a long software routine)
        unsigned u = (unsigned)v;
        q.x = (int)(u % (unsigned)X);
        u /= (unsigned)X;
        q.y = (int)(u % (unsigned)Y);
        u /= (unsigned)Y;
        q.z = (int)(u % (unsigned)Z);
        q.b = u / (unsigned)Z;
    } else {
        q.x = (int)(v % X);
        v /= X;
        q.y = (int)(v % Y);
        v /= Y;
        q.z = (int)(v % Z);
        q.b = v / Z;
    }
    return q;
}
__device__ __forceinline__ int64_t vox_index(int64_t b, int z, int y, int x, int Z, int Y, int X) {
    return ((b * Z + z) * Y + y) * X + x;
}
__device__ __forceinline__ void add8(float (&s)[8], uint4 q) {
    const uint32_t w[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const float2 f = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162 *>(&w[i]));
        s[2 * i] += f.x;
        s[2 * i + 1] += f.y;
    }
}
__device__ __forceinline__ uint4 pack8(const float (&s)[8]) {
    return make_uint4(pack_bf16(s[0], s[1]), pack_bf16(s[2], s[3]), pack_bf16(s[4], s[5]), pack_bf16(s[6], s[7]));
}

__global__ void k_avgpool2_v8(const uint4 *__restrict__ in, uint4 *__restrict__ out, int X, int Y, int Z, int C8,
                              int64_t n) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const int64_t v = i <= 0xffffffffll ? (unsigned)i / (unsigned)C8 : i / C8;
        const int c = (int)(i - v * C8);
        const Vox o = voxel_at(v, X / 2, Y / 2, Z / 2);
        float s[8] = {};
#pragma unroll
        for (int k = 0; k < 8; ++k)
            add8(s, __ldg(in + vox_index(o.b, 2 * o.z + (k >> 2), 2 * o.y + ((k >> 1) & 1), 2 * o.x + (k & 1), Z, Y, X) * C8 + c));
#pragma unroll
        for (int k = 0; k < 8; ++k) s[k] *= 0.125f;
        out[i] = pack8(s);
    }
}

// thread = (parent voxel, 8 channels): its gradient read once for the 8 children
__global__ void k_avgpool2_bwd_v8(const uint4 *__restrict__ dout, uint4 *__restrict__ din, int X, int Y, int Z, int C8,
                                  int64_t n) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const int64_t v = i <= 0xffffffffll ? (unsigned)i / (unsigned)C8 : i / C8;
        const int c = (int)(i - v * C8);
        const Vox o = voxel_at(v, X / 2, Y / 2, Z / 2);
        float d[8] = {};
        add8(d, __ldg(dout + i));
#pragma unroll
        for (int k = 0; k < 8; ++k) d[k] *= 0.125f;
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            uint4 *p = din + vox_index(o.b, 2 * o.z + (k >> 2), 2 * o.y + ((k >> 1) & 1), 2 * o.x + (k & 1), Z, Y, X) * C8 + c;
            float s[8] = {};
            add8(s, *p);
#pragma unroll
            for (int j = 0; j < 8; ++j) s[j] += d[j];
            *p = pack8(s);
        }
    }
}

// A block takes whole lines, so that the line's place is found once (the
// divisions of a flat index were most of the kernel), and a thread has
// kUpLoads reads on their way before its first write.  32 + 16 channels at
// 128 x 128 x 64 x 4: 193 us with a flat index and one read at a time, 154 with
// four reads, 106 so (a training step 6288 -> 6186 us).
constexpr int kUpLoads = 4;
__global__ void k_up_concat_v8(const uint4 *__restrict__ low, const uint4 *__restrict__ skip, uint4 *__restrict__ cat,
                               int X, int Y, int Z, int L8, int S8, int64_t lines) {
    const unsigned C8 = L8 + S8, row = X * C8;
    for (int64_t l = blockIdx.x; l < lines; l += gridDim.x) {
        const int y = (int)(l % Y), z = (int)(l / Y % Z);
        const int64_t b = l / Y / Z;
        const uint4 *lp = low + vox_index(b, z / 2, y / 2, 0, Z / 2, Y / 2, X / 2) * L8, *sp = skip + l * X * S8;
        uint4 *op = cat + l * row;
        for (unsigned e0 = threadIdx.x; e0 < row; e0 += kUpLoads * blockDim.x) {
            uint4 r[kUpLoads];
#pragma unroll
            for (int u = 0; u < kUpLoads; ++u) {
                const unsigned e = e0 + u * blockDim.x;
                if (e >= row) continue;
                const unsigned x = e / C8, c = e - x * C8;
                r[u] = __ldg(c < (unsigned)L8 ? lp + (x / 2) * L8 + c : sp + x * S8 + (c - L8));
            }
#pragma unroll
            for (int u = 0; u < kUpLoads; ++u)
                if (e0 + u * blockDim.x < row) op[e0 + u * blockDim.x] = r[u];
        }
    }
}
__global__ void k_up_concat_bwd_v8(const uint4 *__restrict__ dcat, uint4 *__restrict__ dlow, uint4 *__restrict__ dskip,
                                   int X, int Y, int Z, int L8, int S8, int64_t n_low, int64_t n) {
    const int C8 = L8 + S8;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        float s[8] = {};
        if (i < n_low) {
            const int64_t v = i <= 0xffffffffll ? (unsigned)i / (unsigned)L8 : i / L8;
            const int c = (int)(i - v * L8);
            const Vox o = voxel_at(v, X / 2, Y / 2, Z / 2);
#pragma unroll
            for (int k = 0; k < 8; ++k)
                add8(s, __ldg(dcat + vox_index(o.b, 2 * o.z + (k >> 2), 2 * o.y + ((k >> 1) & 1), 2 * o.x + (k & 1), Z, Y, X) *
                                  C8 + c));
            dlow[i] = pack8(s);
        } else {
            const int64_t j = i - n_low;
            const int64_t v = j <= 0xffffffffll ? (unsigned)j / (unsigned)S8 : j / S8;
            const int c = (int)(j - v * S8);
            add8(s, dskip[j]);
            add8(s, __ldg(dcat + v * C8 + L8 + c));
            dskip[j] = pack8(s);
        }
    }
}

__global__ void k_relu_mask_v8(uint4 *__restrict__ d, const uint4 *__restrict__ a, int64_t n) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const uint4 q = __ldg(a + i);
        uint4 r = d[i];
        const uint32_t w[4] = {q.x, q.y, q.z, q.w};
        uint32_t o[4] = {r.x, r.y, r.z, r.w};
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const float2 f = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162 *>(&w[k]));
            o[k] &= (f.x > 0.f ? 0xffffu : 0u) | (f.y > 0.f ? 0xffff0000u : 0u);
        }
        d[i] = make_uint4(o[0], o[1], o[2], o[3]);
    }
}

// Bias gradient, 8 channels per thread: C8 (2, 4 or 8) threads side by side take
// a voxel.  Few large blocks and a tree inside each, because the FP32 additions
// of the blocks' sums are what the rounding of the result comes from.  4.2M x 16,
// 524288 x 32 and 65536 x 64 values: relative error 1.9e-7, 2.0e-7 and 1.4e-7;
// with 592 blocks of 256 threads 3.7e-7, 5.0e-7 and 2.6e-7 (a training step's ten
// launches 174 us, were 151).
constexpr int kBiasThreads = 1024, kBiasLoads = 4;
__global__ void __launch_bounds__(kBiasThreads) k_bias_grad_v8(const uint4 *__restrict__ dz, float *__restrict__ db, int C8,
                                                               int64_t n) {
    __shared__ float part[kBiasThreads / 32][64];
    float s[8] = {};
    const int64_t stride = (int64_t)gridDim.x * kBiasThreads;   // (a multiple of C8: a thread keeps its channels)
    for (int64_t i = (int64_t)blockIdx.x * kBiasThreads + threadIdx.x; i < n; i += kBiasLoads * stride) {
        uint4 q[kBiasLoads];
#pragma unroll
        for (int u = 0; u < kBiasLoads; ++u) q[u] = i + u * stride < n ? __ldg(dz + i + u * stride) : make_uint4(0, 0, 0, 0);
#pragma unroll
        for (int u = 0; u < kBiasLoads; ++u) add8(s, q[u]);
    }
    const int lane = threadIdx.x & 31;
    for (int o = 16; o >= C8; o >>= 1)
#pragma unroll
        for (int k = 0; k < 8; ++k) s[k] += __shfl_xor_sync(0xffffffffu, s[k], o);
    if (lane < C8)
#pragma unroll
        for (int k = 0; k < 8; ++k) part[threadIdx.x >> 5][lane * 8 + k] = s[k];
    __syncthreads();
    const int c = threadIdx.x >> 5;   // warp c adds up channels c and c + 32
    for (int ch = c; ch < 8 * C8; ch += 32) {
        float t = part[lane][ch];
        for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
        if (lane == 0) atomicAdd(db + ch, t);
    }
}

static bool vec8(std::initializer_list<const void *> p, int c) {
    if (c % 8) return false;
    for (const void *q : p)
        if ((uintptr_t)q & 15) return false;
    return true;
}

// ---------------------------------------------------------------------------
// Network input / output

// 16 channels of a voxel; V: 16-byte aligned tensors (the network's are)
template <bool V>
__device__ __forceinline__ void load16(const bf16 *p, float (&f)[16]) {
    if constexpr (!V) {
#pragma unroll
        for (int c = 0; c < 16; ++c) f[c] = __bfloat162float(p[c]);
        return;
    }
    const uint4 *q = reinterpret_cast<const uint4 *>(p);
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const uint4 v = __ldg(q + h);
        const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float2 t = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162 *>(&w[i]));
            f[8 * h + 2 * i] = t.x;
            f[8 * h + 2 * i + 1] = t.y;
        }
    }
}
// ---------------------------------------------------------------------------

// Input tensor [B][Z][Y][X][16] from the Fortran-order FP32 volumes: channel 0
// = osem[b] * scale[b], channel 1 = sens * sens_scale, other channels 0.
// Source volumes have Zs <= Z slices (the rest is zero padding).
__global__ void k_make_input(const float *__restrict__ osem, int64_t osem_stride, const float *__restrict__ sens,
                             const float *__restrict__ scale, float sens_scale, bf16 *__restrict__ out, int X, int Y,
                             int Z, int Zs, int64_t nvox) {
    for (int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; v < nvox; v += (int64_t)gridDim.x * blockDim.x) {
        const Vox at = voxel_at(v, X, Y, Z);
        const int x = at.x, y = at.y, z = at.z;
        const int64_t b = at.b;
        float c0 = 0.f, c1 = 0.f;
        if (z < Zs) {
            const int64_t s = x + (int64_t)X * (y + (int64_t)Y * z);
            c0 = osem[b * osem_stride + s] * scale[b];
            c1 = sens[s] * sens_scale;
        }
        uint4 *o = reinterpret_cast<uint4 *>(out + v * 16);
        o[0] = make_uint4(pack_bf16(c0, c1), 0u, 0u, 0u);
        o[1] = make_uint4(0u, 0u, 0u, 0u);
    }
}

// Head: pred[b][v] = osem_n[b][v] + bias + sum_c w[c] a[v][c] (a: [..][16]),
// written as FP32 in the padded volume order.
template <bool V>
__global__ void k_head_fwd(const bf16 *__restrict__ a, const bf16 *__restrict__ inp, const float *__restrict__ w,
                           const float *__restrict__ bias, float *__restrict__ pred, int64_t nvox) {
    for (int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; v < nvox; v += (int64_t)gridDim.x * blockDim.x) {
        float s = __bfloat162float(inp[v * 16]) + bias[0];
        float f[16];
        load16<V>(a + v * 16, f);
#pragma unroll
        for (int c = 0; c < 16; ++c) s = fmaf(w[c], f[c], s);
        pred[v] = s;
    }
}

// Loss and head backward: r = pred - target on the valid slices (z < Zs),
// loss += sum r^2 / count; d a[v][c] = g w[c] masked by relu(a) > 0, g = 2 r / count;
// dw[c] += g a[v][c]; db += g.
template <bool V>
__global__ void k_head_bwd(const bf16 *__restrict__ a, const float *__restrict__ pred,
                           const float *__restrict__ target, int64_t target_stride, const float *__restrict__ tscale,
                           const float *__restrict__ w, bf16 *__restrict__ da, float *__restrict__ dw,
                           float *__restrict__ db, float *__restrict__ loss, int X, int Y, int Z, int Zs,
                           int64_t nvox, float inv_count) {
    __shared__ float sw[17];
    __shared__ float sl;
    if (threadIdx.x < 17) sw[threadIdx.x] = 0.f;
    if (threadIdx.x == 0) sl = 0.f;
    __syncthreads();
    float lw[16], lb = 0.f, ll = 0.f;
#pragma unroll
    for (int c = 0; c < 16; ++c) lw[c] = 0.f;
    for (int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; v < nvox; v += (int64_t)gridDim.x * blockDim.x) {
        const Vox at = voxel_at(v, X, Y, Z);
        const int x = at.x, y = at.y, z = at.z;
        const int64_t b = at.b;
        float gr = 0.f;
        if (z < Zs) {
            const float tv = target[b * target_stride + x + (int64_t)X * (y + (int64_t)Y * z)] * tscale[b];
            const float r = pred[v] - tv;
            ll = fmaf(r, r, ll);
            gr = 2.f * r * inv_count;
        }
        lb += gr;
        float f[16];
        load16<V>(a + v * 16, f);
        uint32_t o[8];
#pragma unroll
        for (int c = 0; c < 16; c += 2) {
            lw[c] = fmaf(gr, f[c], lw[c]);
            lw[c + 1] = fmaf(gr, f[c + 1], lw[c + 1]);
            o[c / 2] = pack_bf16(f[c] > 0.f ? gr * w[c] : 0.f, f[c + 1] > 0.f ? gr * w[c + 1] : 0.f);
        }
        if constexpr (V) {
            uint4 *dst = reinterpret_cast<uint4 *>(da + v * 16);
            dst[0] = make_uint4(o[0], o[1], o[2], o[3]);
            dst[1] = make_uint4(o[4], o[5], o[6], o[7]);
        } else {
#pragma unroll
            for (int c = 0; c < 8; ++c) reinterpret_cast<uint32_t *>(da + v * 16)[c] = o[c];
        }
    }
    // a warp's sums first: 18 shared-memory atomics per warp instead of per thread
    auto warp_sum = [](float v) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        return v;
    };
#pragma unroll
    for (int c = 0; c < 16; ++c) lw[c] = warp_sum(lw[c]);
    lb = warp_sum(lb);
    ll = warp_sum(ll);
    if ((threadIdx.x & 31) == 0) {
#pragma unroll
        for (int c = 0; c < 16; ++c) atomicAdd(sw + c, lw[c]);
        atomicAdd(sw + 16, lb);
        atomicAdd(&sl, ll * inv_count);
    }
    __syncthreads();
    if (threadIdx.x < 16) atomicAdd(dw + threadIdx.x, sw[threadIdx.x]);
    if (threadIdx.x == 16) atomicAdd(db, sw[16]);
    if (threadIdx.x == 0) atomicAdd(loss, sl);
}

// Network output back to Fortran-order FP32 volumes: out[b][s] = pred / scale[b], clamped >= floor.
__global__ void k_head_out(const float *__restrict__ pred, const float *__restrict__ scale, float *__restrict__ out,
                           int64_t out_stride, float floor_v, int X, int Y, int Z, int Zs, int64_t nvox) {
    for (int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; v < nvox; v += (int64_t)gridDim.x * blockDim.x) {
        const Vox at = voxel_at(v, X, Y, Z);
        const int x = at.x, y = at.y, z = at.z;
        const int64_t b = at.b;
        if (z < Zs) out[b * out_stride + x + (int64_t)X * (y + (int64_t)Y * z)] = fmaxf(pred[v] / scale[b], floor_v);
    }
}

// Adam on FP32 master weights; writes the BF16 copy used by the kernels.
__global__ void k_adam(float *__restrict__ p, float *__restrict__ m, float *__restrict__ v,
                       const float *__restrict__ gr, bf16 *__restrict__ pb, int64_t n, float lr, float b1, float b2,
                       float c1, float c2, float eps) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const float g = gr[i];
        const float mi = b1 * m[i] + (1.f - b1) * g;
        const float vi = b2 * v[i] + (1.f - b2) * g * g;
        m[i] = mi;
        v[i] = vi;
        const float upd = lr * (mi * c1) / (sqrtf(vi * c2) + eps);
        p[i] -= upd;
        if (pb) pb[i] = __float2bfloat16(p[i]);
    }
}

__global__ void k_f32_to_bf16(const float *__restrict__ a, bf16 *__restrict__ b, int64_t n) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        b[i] = __float2bfloat16(a[i]);
}

// ---------------------------------------------------------------------------
// launchers
// ---------------------------------------------------------------------------

#define OMB_CONV_SHAPES(X) X(16, 16) X(16, 32) X(32, 32) X(32, 64) X(64, 64) X(96, 32) X(48, 16) \
    X(32, 16) X(64, 32) X(32, 96) X(16, 48)

int unet_conv(int cin, int cout, const void *in, const void *w, const float *bias, void *out, const void *mask,
              int relu, int X, int Y, int Z, int B, cudaStream_t st) {
    if (X <= 0 || Y <= 0 || Z <= 0 || B <= 0) return set_error(OMB_ERR_INVALID, "bad conv volume");
    if ((int64_t)Z * B > 65535 || Y > 65535) return set_error(OMB_ERR_UNSUPPORTED, "conv volume too large");
    dim3 grid((X + 63) / 64, Y, Z * B);
    const bf16 *i = static_cast<const bf16 *>(in), *wt = static_cast<const bf16 *>(w),
               *mk = static_cast<const bf16 *>(mask);
    bf16 *o = static_cast<bf16 *>(out);
#define X(ci, co)                                                                                   \
    if (cin == ci && cout == co) {                                                                  \
        if (mask)                                                                                   \
            k_conv3d<ci, co, false, true><<<grid, 128, 0, st>>>(i, wt, bias, o, mk, X, Y, Z);       \
        else if (relu)                                                                              \
            k_conv3d<ci, co, true, false><<<grid, 128, 0, st>>>(i, wt, bias, o, mk, X, Y, Z);       \
        else                                                                                        \
            k_conv3d<ci, co, false, false><<<grid, 128, 0, st>>>(i, wt, bias, o, mk, X, Y, Z);      \
        OMB_LAUNCH_CHECK("conv launch");                                                            \
        return OMB_OK;                                                                              \
    }
    OMB_CONV_SHAPES(X)
#undef X
    return set_error(OMB_ERR_UNSUPPORTED, "conv shape " + std::to_string(cin) + "->" + std::to_string(cout) +
                                              " is not built");
}

// The largest stage (at most 8 lines: the input's two halo lines weigh less)
// of which three, or else two, fit an SM's shared memory.
template <int CIN, int COUT>
static int launch_wgrad(const bf16 *in, const bf16 *dz, float *dw, int X, int Y, int Z, int B, cudaStream_t st) {
    using S = WgradShape<CIN, COUT>;
    WgradPlan p{X, Y, Z, B};
    p.ntx = (X + 127) / 128;
    p.TX = ((X + p.ntx - 1) / p.ntx + 15) / 16 * 16;
    // planes start 16 to 64 bytes apart modulo 128, so that the copies of
    // neighbouring channels of a voxel meet different banks
    auto plane = [](int rows, int planes) { return (rows * 16 + 127) / 128 * 128 + (planes <= 2 ? 64 : (planes <= 4 ? 32 : 16)); };
    for (p.ring = 3; p.ring >= 2 && !p.smem; --p.ring) {
        for (p.TY = Y < 8 ? Y : 8; p.TY >= 1; --p.TY) {
            p.in_plane = plane((p.TY + 2) * p.TX, CIN / 8);
            p.dz_plane = plane(p.TY * (p.TX + 2), COUT / 8);
            p.dz_off = (p.in_plane * (CIN / 8) + 127) / 128 * 128;
            p.stage = (p.dz_off + p.dz_plane * (COUT / 8) + 127) / 128 * 128;
            if (p.ring * p.stage <= 226 * 1024) {
                p.smem = p.ring * p.stage;
                break;
            }
        }
        if (p.smem) break;
    }
    p.nty = (Y + p.TY - 1) / p.TY;
    p.inv = 65536u / (p.TX / 16) + 1;   // (at most 64 groups of a stage, 8 of a line: exact)
    const int64_t tiles = (int64_t)p.ntx * p.nty * Z * B;
    if (!p.smem || tiles > 2147483647) return set_error(OMB_ERR_UNSUPPORTED, "wgrad volume too large");
    p.tiles = (int)tiles;
    p.flush = 8192 * S::KS / (p.TX * p.TY) > 1 ? 8192 * S::KS / (p.TX * p.TY) : 1;
    auto kernel = k_conv3d_wgrad<CIN, COUT>;
    OMB_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, p.smem));
    const int blocks = num_sms() / 3 > 0 ? num_sms() / 3 : 1;
    kernel<<<dim3(p.tiles < blocks ? p.tiles : blocks, 3), S::kThreads, p.smem, st>>>(p, in, dz, dw);
    OMB_LAUNCH_CHECK("wgrad launch");
    return OMB_OK;
}

int unet_conv_wgrad(int cin, int cout, const void *in, const void *dz, float *dw, int X, int Y, int Z, int B,
                    cudaStream_t st) {
    if ((int64_t)X * Y * Z * B <= 0) return OMB_OK;
    const bf16 *i = static_cast<const bf16 *>(in), *d = static_cast<const bf16 *>(dz);
#define X(ci, co) \
    if (cin == ci && cout == co) return launch_wgrad<ci, co>(i, d, dw, X, Y, Z, B, st);
    OMB_CONV_SHAPES(X)
#undef X
    return set_error(OMB_ERR_UNSUPPORTED, "wgrad shape is not built");
}

int unet_bias_grad(int c, const void *dz, float *db, int64_t nvox, cudaStream_t st) {
    const bf16 *d = static_cast<const bf16 *>(dz);
    if ((c == 16 || c == 32 || c == 64) && vec8({dz}, c)) {
        const int64_t n = nvox * (c / 8);
        k_bias_grad_v8<<<grid_for(n, 1, kBiasThreads), kBiasThreads, 0, st>>>(static_cast<const uint4 *>(dz), db, c / 8, n);
        OMB_LAUNCH_CHECK("bias gradient launch");
        return OMB_OK;
    }
    const unsigned grid = grid_for(nvox * c / 256 + 1, 4);
    switch (c) {
        case 16: k_bias_grad<16><<<grid, 256, 0, st>>>(d, db, nvox); break;
        case 32: k_bias_grad<32><<<grid, 256, 0, st>>>(d, db, nvox); break;
        case 64: k_bias_grad<64><<<grid, 256, 0, st>>>(d, db, nvox); break;
        default: return set_error(OMB_ERR_UNSUPPORTED, "bias gradient channel count");
    }
    OMB_LAUNCH_CHECK("bias grad launch");
    return OMB_OK;
}

int unet_flip_weights(const void *w, void *wf, int cin, int cout, cudaStream_t st) {
    k_flip_weights<<<grid_for(27 * cin * cout, 2), 256, 0, st>>>(static_cast<const bf16 *>(w), static_cast<bf16 *>(wf),
                                                                 cin, cout);
    OMB_LAUNCH_CHECK("flip launch");
    return OMB_OK;
}

int unet_avgpool(const void *in, void *out, int X, int Y, int Z, int B, int C, int backward, cudaStream_t st) {
    if (X % 2 || Y % 2 || Z % 2) return set_error(OMB_ERR_INVALID, "pooling needs even sizes");
    if (vec8({in, out}, C)) {
        const int64_t n = (int64_t)(X / 2) * (Y / 2) * (Z / 2) * B * (C / 8);
        if (!backward)
            k_avgpool2_v8<<<grid_for(n, 8), 256, 0, st>>>(static_cast<const uint4 *>(in), static_cast<uint4 *>(out), X, Y,
                                                          Z, C / 8, n);
        else
            k_avgpool2_bwd_v8<<<grid_for(n, 8), 256, 0, st>>>(static_cast<const uint4 *>(in), static_cast<uint4 *>(out),
                                                              X, Y, Z, C / 8, n);
    } else if (!backward) {
        const int64_t nout = (int64_t)(X / 2) * (Y / 2) * (Z / 2) * B;
        k_avgpool2<<<grid_for(nout * C, 8), 256, 0, st>>>(static_cast<const bf16 *>(in), static_cast<bf16 *>(out), X,
                                                          Y, Z, C, nout);
    } else {
        const int64_t nin = (int64_t)X * Y * Z * B;
        k_avgpool2_bwd<<<grid_for(nin * C, 8), 256, 0, st>>>(static_cast<const bf16 *>(in), static_cast<bf16 *>(out),
                                                             X, Y, Z, C, nin);
    }
    OMB_LAUNCH_CHECK("pool launch");
    return OMB_OK;
}

int unet_up_concat(const void *low, const void *skip, void *cat, int X, int Y, int Z, int B, int cl, int cs,
                   cudaStream_t st) {
    const int64_t nvox = (int64_t)X * Y * Z * B, lines = (int64_t)Y * Z * B;
    // (a line's 16-byte words are counted in 32 bits)
    if (vec8({low, skip, cat}, cl) && cs % 8 == 0 && X > 0 && lines > 0 && (int64_t)X * ((cl + cs) / 8) < 0x40000000) {
        k_up_concat_v8<<<grid_for(lines, 8, 1), 256, 0, st>>>(static_cast<const uint4 *>(low),
                                                              static_cast<const uint4 *>(skip), static_cast<uint4 *>(cat),
                                                              X, Y, Z, cl / 8, cs / 8, lines);
        OMB_LAUNCH_CHECK("upsample launch");
        return OMB_OK;
    }
    k_up_concat<<<grid_for(nvox * (cl + cs), 8), 256, 0, st>>>(static_cast<const bf16 *>(low),
                                                               static_cast<const bf16 *>(skip), static_cast<bf16 *>(cat),
                                                               X, Y, Z, cl, cs, nvox);
    OMB_LAUNCH_CHECK("upsample launch");
    return OMB_OK;
}

int unet_up_concat_bwd(const void *dcat, void *dlow, void *dskip, int X, int Y, int Z, int B, int cl, int cs,
                       cudaStream_t st) {
    const int64_t nvox = (int64_t)X * Y * Z * B, nlow = nvox / 8;
    if (vec8({dcat, dlow, dskip}, cl) && cs % 8 == 0) {
        const int64_t n_low = nlow * (cl / 8), n = n_low + nvox * (cs / 8);
        k_up_concat_bwd_v8<<<grid_for(n, 8), 256, 0, st>>>(static_cast<const uint4 *>(dcat), static_cast<uint4 *>(dlow),
                                                           static_cast<uint4 *>(dskip), X, Y, Z, cl / 8, cs / 8, n_low, n);
        OMB_LAUNCH_CHECK("upsample backward launch");
        return OMB_OK;
    }
    k_up_concat_bwd<<<grid_for(nlow * cl + nvox * cs, 8), 256, 0, st>>>(
        static_cast<const bf16 *>(dcat), static_cast<bf16 *>(dlow), static_cast<bf16 *>(dskip), X, Y, Z, cl, cs, nlow,
        nvox);
    OMB_LAUNCH_CHECK("upsample backward launch");
    return OMB_OK;
}

int unet_make_input(const float *osem, int64_t osem_stride, const float *sens, const float *scale, float sens_scale,
                    void *out, int X, int Y, int Z, int Zs, int B, cudaStream_t st) {
    const int64_t nvox = (int64_t)X * Y * Z * B;
    k_make_input<<<grid_for(nvox, 8), 256, 0, st>>>(osem, osem_stride, sens, scale, sens_scale,
                                                    static_cast<bf16 *>(out), X, Y, Z, Zs, nvox);
    OMB_LAUNCH_CHECK("input launch");
    return OMB_OK;
}

int unet_head_fwd(const void *a, const void *inp, const float *w, const float *bias, float *pred, int64_t nvox,
                  cudaStream_t st) {
    auto kernel = vec8({a}, 16) ? k_head_fwd<true> : k_head_fwd<false>;
    kernel<<<grid_for(nvox, 8), 256, 0, st>>>(static_cast<const bf16 *>(a), static_cast<const bf16 *>(inp), w, bias, pred,
                                              nvox);
    OMB_LAUNCH_CHECK("head launch");
    return OMB_OK;
}

int unet_head_bwd(const void *a, const float *pred, const float *target, int64_t target_stride, const float *tscale,
                  const float *w, void *da, float *dw, float *db, float *loss, int X, int Y, int Z, int Zs, int B,
                  cudaStream_t st) {
    const int64_t nvox = (int64_t)X * Y * Z * B;
    const float inv = 1.f / (float)((int64_t)X * Y * Zs * B);
    auto kernel = vec8({a, da}, 16) ? k_head_bwd<true> : k_head_bwd<false>;
    kernel<<<grid_for(nvox, 4), 256, 0, st>>>(static_cast<const bf16 *>(a), pred, target, target_stride, tscale, w,
                                              static_cast<bf16 *>(da), dw, db, loss, X, Y, Z, Zs, nvox, inv);
    OMB_LAUNCH_CHECK("head backward launch");
    return OMB_OK;
}

int unet_head_out(const float *pred, const float *scale, float *out, int64_t out_stride, float floor_v, int X, int Y,
                  int Z, int Zs, int B, cudaStream_t st) {
    const int64_t nvox = (int64_t)X * Y * Z * B;
    k_head_out<<<grid_for(nvox, 8), 256, 0, st>>>(pred, scale, out, out_stride, floor_v, X, Y, Z, Zs, nvox);
    OMB_LAUNCH_CHECK("output launch");
    return OMB_OK;
}

int unet_adam(float *p, float *m, float *v, const float *g, void *pb, int64_t n, float lr, float b1, float b2,
              int step, float eps, cudaStream_t st) {
    const float c1 = 1.f / (1.f - powf(b1, (float)step)), c2 = 1.f / (1.f - powf(b2, (float)step));
    k_adam<<<grid_for(n, 4), 256, 0, st>>>(p, m, v, g, static_cast<bf16 *>(pb), n, lr, b1, b2, c1, c2, eps);
    OMB_LAUNCH_CHECK("adam launch");
    return OMB_OK;
}

int unet_relu_mask(void *d, const void *a, int64_t n, cudaStream_t st) {
    if (n % 8 == 0 && vec8({d, a}, 8)) {
        k_relu_mask_v8<<<grid_for(n / 8, 8), 256, 0, st>>>(static_cast<uint4 *>(d), static_cast<const uint4 *>(a), n / 8);
        OMB_LAUNCH_CHECK("relu mask launch");
        return OMB_OK;
    }
    k_relu_mask<<<grid_for(n, 8), 256, 0, st>>>(static_cast<bf16 *>(d), static_cast<const bf16 *>(a), n);
    OMB_LAUNCH_CHECK("relu mask launch");
    return OMB_OK;
}

int unet_to_bf16(const float *a, void *b, int64_t n, cudaStream_t st) {
    k_f32_to_bf16<<<grid_for(n, 4), 256, 0, st>>>(a, static_cast<bf16 *>(b), n);
    OMB_LAUNCH_CHECK("bf16 conversion launch");
    return OMB_OK;
}

}  // namespace omb

// ---------------------------------------------------------------------------
// C-ABI (include/omega_b200_unet.h)
// ---------------------------------------------------------------------------
extern "C" {

int omb_unet_conv(int32_t cin, int32_t cout, const void *in, const void *w, const float *bias, void *out,
                  const void *relu_mask, int32_t relu, int32_t X, int32_t Y, int32_t Z, int32_t B, void *stream) {
    if (!in || !w || !out) return omb::set_error(OMB_ERR_INVALID, "NULL buffer passed to omb_unet_conv");
    return omb::unet_conv(cin, cout, in, w, bias, out, relu_mask, relu, X, Y, Z, B, (cudaStream_t)stream);
}

int omb_unet_conv_wgrad(int32_t cin, int32_t cout, const void *in, const void *dz, float *dw, int32_t X, int32_t Y,
                        int32_t Z, int32_t B, void *stream) {
    if (!in || !dz || !dw) return omb::set_error(OMB_ERR_INVALID, "NULL buffer passed to omb_unet_conv_wgrad");
    return omb::unet_conv_wgrad(cin, cout, in, dz, dw, X, Y, Z, B, (cudaStream_t)stream);
}

int omb_unet_bias_grad(int32_t c, const void *dz, float *db, int64_t nvox, void *stream) {
    if (!dz || !db) return omb::set_error(OMB_ERR_INVALID, "NULL buffer passed to omb_unet_bias_grad");
    return omb::unet_bias_grad(c, dz, db, nvox, (cudaStream_t)stream);
}

int omb_unet_flip_weights(const void *w, void *wf, int32_t cin, int32_t cout, void *stream) {
    if (!w || !wf) return omb::set_error(OMB_ERR_INVALID, "NULL buffer passed to omb_unet_flip_weights");
    return omb::unet_flip_weights(w, wf, cin, cout, (cudaStream_t)stream);
}

int omb_unet_avgpool(const void *in, void *out, int32_t X, int32_t Y, int32_t Z, int32_t B, int32_t C,
                     int32_t backward, void *stream) {
    if (!in || !out) return omb::set_error(OMB_ERR_INVALID, "NULL buffer passed to omb_unet_avgpool");
    return omb::unet_avgpool(in, out, X, Y, Z, B, C, backward, (cudaStream_t)stream);
}

int omb_unet_up_concat(const void *low, const void *skip, void *cat, int32_t X, int32_t Y, int32_t Z, int32_t B,
                       int32_t cl, int32_t cs, void *stream) {
    if (!low || !skip || !cat) return omb::set_error(OMB_ERR_INVALID, "NULL buffer passed to omb_unet_up_concat");
    return omb::unet_up_concat(low, skip, cat, X, Y, Z, B, cl, cs, (cudaStream_t)stream);
}

int omb_unet_up_concat_bwd(const void *dcat, void *dlow, void *dskip, int32_t X, int32_t Y, int32_t Z, int32_t B,
                           int32_t cl, int32_t cs, void *stream) {
    if (!dcat || !dlow || !dskip) return omb::set_error(OMB_ERR_INVALID, "NULL buffer passed to omb_unet_up_concat_bwd");
    return omb::unet_up_concat_bwd(dcat, dlow, dskip, X, Y, Z, B, cl, cs, (cudaStream_t)stream);
}

int omb_unet_relu_mask(void *d, const void *a, int64_t n, void *stream) {
    if (!d || !a) return omb::set_error(OMB_ERR_INVALID, "NULL buffer passed to omb_unet_relu_mask");
    return omb::unet_relu_mask(d, a, n, (cudaStream_t)stream);
}

int omb_unet_make_input(const float *osem, int64_t osem_stride, const float *sens, const float *scale,
                        float sens_scale, void *out, int32_t X, int32_t Y, int32_t Z, int32_t Zs, int32_t B,
                        void *stream) {
    if (!osem || !sens || !scale || !out) return omb::set_error(OMB_ERR_INVALID, "NULL buffer passed to omb_unet_make_input");
    return omb::unet_make_input(osem, osem_stride, sens, scale, sens_scale, out, X, Y, Z, Zs, B, (cudaStream_t)stream);
}

int omb_unet_head_fwd(const void *a, const void *inp, const float *w, const float *bias, float *pred, int64_t nvox,
                      void *stream) {
    if (!a || !inp || !w || !bias || !pred) return omb::set_error(OMB_ERR_INVALID, "NULL buffer passed to omb_unet_head_fwd");
    return omb::unet_head_fwd(a, inp, w, bias, pred, nvox, (cudaStream_t)stream);
}

int omb_unet_head_bwd(const void *a, const float *pred, const float *target, int64_t target_stride,
                      const float *tscale, const float *w, void *da, float *dw, float *db, float *loss, int32_t X,
                      int32_t Y, int32_t Z, int32_t Zs, int32_t B, void *stream) {
    if (!a || !pred || !target || !tscale || !w || !da || !dw || !db || !loss)
        return omb::set_error(OMB_ERR_INVALID, "NULL buffer passed to omb_unet_head_bwd");
    return omb::unet_head_bwd(a, pred, target, target_stride, tscale, w, da, dw, db, loss, X, Y, Z, Zs, B,
                              (cudaStream_t)stream);
}

int omb_unet_head_out(const float *pred, const float *scale, float *out, int64_t out_stride, float floor_v, int32_t X,
                      int32_t Y, int32_t Z, int32_t Zs, int32_t B, void *stream) {
    if (!pred || !scale || !out) return omb::set_error(OMB_ERR_INVALID, "NULL buffer passed to omb_unet_head_out");
    return omb::unet_head_out(pred, scale, out, out_stride, floor_v, X, Y, Z, Zs, B, (cudaStream_t)stream);
}

int omb_unet_adam(float *p, float *m, float *v, const float *g, void *p_bf16, int64_t n, float lr, float beta1,
                  float beta2, int32_t step, float eps, void *stream) {
    if (!p || !m || !v || !g) return omb::set_error(OMB_ERR_INVALID, "NULL buffer passed to omb_unet_adam");
    if (step < 1) return omb::set_error(OMB_ERR_INVALID, "Adam step must be >= 1");
    return omb::unet_adam(p, m, v, g, p_bf16, n, lr, beta1, beta2, step, eps, (cudaStream_t)stream);
}

int omb_unet_to_bf16(const float *a, void *b, int64_t n, void *stream) {
    if (!a || !b) return omb::set_error(OMB_ERR_INVALID, "NULL buffer passed to omb_unet_to_bf16");
    return omb::unet_to_bf16(a, b, n, (cudaStream_t)stream);
}

}  // extern "C"
