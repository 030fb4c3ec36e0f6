// Weight gradient of a 3x3 convolution (stride 1, zero padding 1) of NHWC BF16 tensors on the
// tcgen05 tensor cores:
//   dW[co, tap, ci] = sum_p dz[p, co] x[p + off(tap), ci]
// as D[co, (dx, dy, ci)] = A^T B with the pixels p as the contraction: A = dz and B = x shifted
// by the tap, both as they lie in memory (channels contiguous), which the tensor core reads as
// M- and N-major operands; nothing is transposed or copied.
//
// A CTA takes 32 (or 16) input channels and every output channel, and walks the pixel tiles
// t = blockIdx.x, + gridDim.x, ... of 16 x 8 pixels.  Per tile, TMA brings dz (one box of 128
// pixels per 32 channels) and three boxes of x of 18 x 8 pixels, one per dx, zero-filled outside
// the image.  8 pixels of an image row are one swizzle atom, so 16 pixels of the contraction are
// two atoms, and the three dy are the same box started 0, 1 or 2 atoms further: one MMA of
// N = 3 * 32 covers them (the operand's N blocks lie one atom apart, as its K blocks do).
// The tensor core does not round its running sum to nearest, so a sum left there over many tiles
// drifts in proportion to their number: 1.1e-5 of layer 8's weights for 64 images of 64 x 64,
// 3.6e-4 for 1024, against 2.3e-7 and 3.7e-6 of FP32 sums over 2048 pixels on the CUDA cores.  It
// therefore holds one tile at a time, an accumulator for each dx, and the epilogue warps add it to
// running sums in their registers (4.7e-8 and 3.1e-7).  Tensor memory has room for five such
// accumulators: the next tile waits only for the first of this one to be read.  Each CTA writes one
// partial sum, added over the CTAs by k_sum_parts in a fixed order.
//   warps 0-11: four for each dy, a lane for each output channel, 3 * 32 running sums a lane;
//   warp 12: TMA producer; warp 13: MMA issuer (24 instructions of 128 x 96 x 16 a tile);
//   warps 14-15: the bias gradient from the dz tiles in shared memory (first channel block only).
// Fewer than 128 output channels leave rows of D unused: the instruction reads what lies behind
// the dz boxes for them (other boxes, and kWgBehind bytes kept after the last stage), and they are
// not written.
// Bound: the MMA warp, 24 x 60 cycles of issue and two waits a tile and channel block (the narrow
// N and the unused rows cost up to 4x the useful products at 32 channels).  Four images of 256 x
// 256, all ten layers: CUDA-core sums over 32 x 32 blocks 8.40 ms, 0.32 ms so; with the sums left
// in the tensor core over all tiles 0.29 ms.
#pragma once
#include "unet_conv.cuh"

namespace lica {
namespace unet {

constexpr int kWgThreads = 512;
constexpr int kWgRing = 5;              // accumulators in tensor memory: 5 * 96 columns
constexpr int kWgMaxStages = 6;
constexpr int kWgDzBox = kTileM * 64;   // bytes of a dz box: 128 pixels x 32 channels
constexpr int kWgBehind = 4 * kWgDzBox; // room behind the last stage for the unused rows' reads

struct WgradParams {
    int h, w, tiles;      // image size, pixel tiles of the launch
    int cout, ctot;
    int cblk;             // input channels of a block: 32 or 16
    int c0;               // channels of the first input
    int nstages, stage;   // ring stages and bytes of one
    float* part;          // [gridDim.x][cout][9][ctot]
    float* bpart;         // [gridDim.x][cout]
    int* err;
};

// M- or N-major swizzled operand of rows (one pixel's channels) of 64 or 32 bytes: row blocks of
// that many bytes lie mn bytes apart along M or N, groups of 8 pixels k bytes apart.
__device__ __forceinline__ uint64_t mn_desc(uint32_t addr, uint32_t row_bytes, uint32_t mn, uint32_t k) {
    uint64_t d = 0;
    d |= (uint64_t)((addr & 0x3FFFFu) >> 4);
    d |= (uint64_t)(mn >> 4) << 16;
    d |= (uint64_t)(k >> 4) << 32;
    d |= 1ull << 46;
    d |= (row_bytes == 64 ? 4ull : 6ull) << 61;
    return d;
}

// tc::mbar_wait_warp without the suspend-time hint.  The MMA warp waits twice a tile on barriers that
// are mostly ready, and a try_wait with the hint takes 700 to 900 cycles even then, 130 without it.
__device__ __forceinline__ bool wait_warp(uint64_t* bar, uint32_t parity, int lane) {
    int ok = 1;
    if (lane == 0) {
        auto ready = [&] {
            uint32_t r;
            asm volatile(
                "{\n\t.reg .pred p;\n\t"
                "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
                "selp.u32 %0, 1, 0, p;\n\t}"
                : "=r"(r)
                : "r"(tc::smem_u32(bar)), "r"(parity)
                : "memory");
            return r != 0;
        };
        if (!ready()) {
            const uint64_t t0 = tc::global_ns();
            while (ok && !ready()) ok = tc::global_ns() - t0 <= tc::kWaitNs;
        }
    }
    return __shfl_sync(0xffffffffu, ok, 0) != 0;
}

__global__ void __launch_bounds__(kWgThreads, 1)
    k_wgrad3x3(const __grid_constant__ CUtensorMap tm_dz, const __grid_constant__ CUtensorMap tm_x0,
               const __grid_constant__ CUtensorMap tm_x1, const WgradParams P) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    unsigned char* base = reinterpret_cast<unsigned char*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    __shared__ uint64_t full[kWgMaxStages], empty[kWgMaxStages], sums_full[2], drained, done;
    __shared__ uint32_t tmem_slot;
    __shared__ float sbias[128];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int NS = P.nstages, nco = P.cout / 32;
    const bool bias = blockIdx.y == 0;
    if (threadIdx.x == 0) {
        for (int s = 0; s < NS; ++s) {
            tc::mbar_init(&full[s], 1);
            tc::mbar_init(&empty[s], bias ? 3 : 1);   // the MMAs, and the two warps that sum dz
        }
        for (int b = 0; b < 2; ++b) tc::mbar_init(&sums_full[b], 1);
        tc::mbar_init(&drained, 3 * nco);             // the warps that have output channels
        tc::mbar_init(&done, 1);
        tc::fence_barrier_init();
    }
    after_previous();  // before the tensor memory is taken
    if (warp == 0) tc::tmem_alloc(&tmem_slot, 512);
    tc::tc_fence_before();
    __syncthreads();
    tc::tc_fence_after();
    const uint32_t tmem = tmem_slot;
    const int ci0 = (int)blockIdx.y * P.cblk;
    const int row = 2 * P.cblk;                        // bytes of a pixel of x
    const int dz_bytes = nco * kWgDzBox, xbox = kHaloRows * row;
    const int ncol = 3 * P.cblk;                       // columns of one dx

    if (warp == 12) {
        int s = 0;
        uint32_t ph = 0;
        const void* tmx = ci0 < P.c0 ? (const void*)&tm_x0 : (const void*)&tm_x1;
        const int cx = ci0 < P.c0 ? ci0 : ci0 - P.c0;
        int g = 0;
        for (int t = blockIdx.x; t < P.tiles; t += gridDim.x, ++g) {
            if (g >= NS && !wait_warp(&empty[s], ph ^ 1u, lane)) {
                if (lane == 0) atomicExch(P.err, 1);
                break;
            }
            const int tiles_x = P.w / kTileW, tiles_y = P.h / kTileH;
            const int x0 = (t % tiles_x) * kTileW, y0 = (t / tiles_x) % tiles_y * kTileH, img = t / (tiles_x * tiles_y);
            if (tc::elect_one()) {
                unsigned char* st = base + s * P.stage;
                tc::mbar_expect_tx(&full[s], (uint32_t)(dz_bytes + 3 * xbox));
                for (int b = 0; b < nco; ++b) tc::tma_load_4d(st + b * kWgDzBox, &tm_dz, &full[s], 32 * b, x0, y0, img);
                for (int dx = 0; dx < 3; ++dx)
                    tc::tma_load_4d(st + dz_bytes + dx * xbox, tmx, &full[s], cx, x0 + dx - 1, y0 - 1, img);
            }
            __syncwarp();
            if (++s == NS) {
                s = 0;
                ph ^= 1u;
            }
        }
    } else if (warp == 13) {
        // both operands M-/N-major: bits 15 and 16
        const uint32_t idesc = tc::idesc_bf16_f32(128, (uint32_t)ncol) | (1u << 15) | (1u << 16);
        const uint32_t atom = 8u * (uint32_t)row;
        int s = 0;
        uint32_t ph = 0;
        bool ok = true;
        int slot = 0;     // the tile's first accumulator
        for (int t = blockIdx.x, i = 0; t < P.tiles; t += gridDim.x, ++i) {
            // the third accumulator was the first of the tile before; the others' last contents were
            // read by the same warps before that
            ok = wait_warp(&full[s], ph, lane) && (i == 0 || wait_warp(&drained, (unsigned)(i - 1) & 1u, lane));
            if (!ok) break;
            tc::tc_fence_after();
            const uint32_t st = tc::smem_u32(base + s * P.stage);
            const uint64_t a0 = mn_desc(st, 64, (uint32_t)kWgDzBox, 512);
            const uint64_t b0 = mn_desc(st + (uint32_t)dz_bytes, (uint32_t)row, atom, atom);
            uint32_t acc[3];
#pragma unroll
            for (int dx = 0; dx < 3; ++dx) {
                acc[dx] = tmem + (uint32_t)(slot * ncol);
                slot = slot + 1 == kWgRing ? 0 : slot + 1;
            }
            if (tc::elect_one()) {
#pragma unroll 1
                for (int k = 0; k < kTileM / 16; ++k)
#pragma unroll
                    for (int dx = 0; dx < 3; ++dx)
                        tc::mma_bf16(acc[dx], a0 + (uint32_t)(k * 1024 / 16),
                                     b0 + (uint32_t)(dx * xbox) / 16u + (uint32_t)k * (2u * atom / 16u), idesc, k != 0);
                tc::mma_commit(&sums_full[i & 1]);
                tc::mma_commit(&empty[s]);
            }
            __syncwarp();
            if (++s == NS) {
                s = 0;
                ph ^= 1u;
            }
        }
        if (tc::elect_one()) tc::mma_commit(&done);
        __syncwarp();
        if (!wait_warp(&done, 0, lane) || !ok)
            if (lane == 0) atomicExch(P.err, 1);
    } else if (warp >= 14) {
        if (bias) {
            // lane = 8 channels (one 16-byte chunk of 4) of every 32-channel box, pixels p, p + 8, ... of the
            // warp's half of the tile, whose sum is formed by itself, then added
            float acc[4][8];
#pragma unroll
            for (int b = 0; b < 4; ++b)
#pragma unroll
                for (int q = 0; q < 8; ++q) acc[b][q] = 0.f;
            const int chunk = lane & 3, p0 = (warp - 14) * (kTileM / 2) + (lane >> 2);
            int s = 0;
            uint32_t ph = 0;
            for (int t = blockIdx.x; t < P.tiles; t += gridDim.x) {
                if (!wait_warp(&full[s], ph, lane)) {
                    if (lane == 0) atomicExch(P.err, 1);
                    break;
                }
                const unsigned char* st = base + s * P.stage;
#pragma unroll
                for (int b = 0; b < 4; ++b)
                    if (b < nco) {
                        float v[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll 4
                        for (int p = p0; p < p0 + kTileM / 2; p += 8) {
                            // the 64-byte swizzle: address bits 4-5 exclusive-or bits 7-8
                            const uint4 w = *reinterpret_cast<const uint4*>(st + b * kWgDzBox + p * 64 +
                                                                            ((chunk ^ ((p >> 1) & 3)) << 4));
                            const uint32_t u[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
                            for (int q = 0; q < 4; ++q) {
                                v[2 * q] += __uint_as_float(u[q] << 16);
                                v[2 * q + 1] += __uint_as_float(u[q] & 0xffff0000u);
                            }
                        }
#pragma unroll
                        for (int q = 0; q < 8; ++q) acc[b][q] += v[q];
                    }
                __syncwarp();
                if (lane == 0) tc::mbar_arrive(&empty[s]);
                if (++s == NS) {
                    s = 0;
                    ph ^= 1u;
                }
            }
            // over the 8 pixel groups (lanes of one chunk are 4 apart), then the two halves
#pragma unroll
            for (int b = 0; b < 4; ++b)
                if (b < nco)
#pragma unroll
                    for (int q = 0; q < 8; ++q)
                        for (int o = 16; o >= 4; o >>= 1) acc[b][q] += __shfl_xor_sync(0xffffffffu, acc[b][q], o);
            if (warp == 15 && lane < 4)
#pragma unroll
                for (int b = 0; b < 4; ++b)
#pragma unroll
                    for (int q = 0; q < 8; ++q) sbias[32 * b + 8 * chunk + q] = acc[b][q];
            asm volatile("bar.sync 1, 64;" ::: "memory");
            if (warp == 14 && lane < 4)
#pragma unroll
                for (int b = 0; b < 4; ++b)
                    if (b < nco)
#pragma unroll
                        for (int q = 0; q < 8; ++q) {
                            const int c = 32 * b + 8 * chunk + q;
                            P.bpart[(size_t)blockIdx.x * P.cout + c] = acc[b][q] + sbias[c];
                        }
        }
    } else if (32 * (warp & 3) < P.cout) {
        const int dy = warp >> 2;
        const uint32_t taddr = tmem + ((uint32_t)(32 * (warp & 3)) << 16) + (uint32_t)(dy * P.cblk);
        float acc[3][32];
#pragma unroll
        for (int dx = 0; dx < 3; ++dx)
#pragma unroll
            for (int q = 0; q < 32; ++q) acc[dx][q] = 0.f;
        int slot = 0;
        bool ok = true;
        for (int t = blockIdx.x, i = 0; t < P.tiles; t += gridDim.x, ++i) {
            if (!(ok = wait_warp(&sums_full[i & 1], (unsigned)(i >> 1) & 1u, lane))) {
                if (lane == 0) atomicExch(P.err, 1);
                break;
            }
            tc::tc_fence_after();
#pragma unroll
            for (int dx = 0; dx < 3; ++dx) {
                const uint32_t at = taddr + (uint32_t)(slot * ncol);
                slot = slot + 1 == kWgRing ? 0 : slot + 1;
#pragma unroll
                for (int c = 0; c < 32; c += 16)
                    if (c < P.cblk) {
                        float v[16];
                        tc::tmem_ld16(at + (uint32_t)c, v);
#pragma unroll
                        for (int q = 0; q < 16; ++q) acc[dx][c + q] += v[q];
                    }
                if (dx == 0) {
                    tc::tc_fence_before();
                    __syncwarp();
                    if (lane == 0) tc::mbar_arrive(&drained);
                }
            }
        }
        if (ok) {
            const int co = 32 * (warp & 3) + lane;
            float* dst = P.part + ((size_t)blockIdx.x * P.cout + co) * 9 * P.ctot + ci0;
#pragma unroll
            for (int dx = 0; dx < 3; ++dx)
#pragma unroll
                for (int q = 0; q < 32; q += 4)
                    if (q < P.cblk)
                        *reinterpret_cast<float4*>(dst + (3 * dy + dx) * P.ctot + q) =
                            make_float4(acc[dx][q], acc[dx][q + 1], acc[dx][q + 2], acc[dx][q + 3]);
        }
    }
    __syncwarp();
    tc::tc_fence_before();
    __syncthreads();
    if (warp == 0) {
        tc::tc_fence_after();
        tc::tmem_dealloc(tmem, 512);
    }
}

}  // namespace unet
}  // namespace lica
